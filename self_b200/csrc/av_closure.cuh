// Artificial-viscosity closure of the CompressibleIdealGas2D tendency.
//
// Not a reference routine: the shock closure built from the reference's own
// operators -- BassiRebaySides + GradientBR (src/SELF_MappedData.f90:919-1078),
// VectorBoundaryInterp (src/SELF_Lagrange.f90:2284-2316), SideExchange of a
// vector (src/SELF_MappedData.f90:1870-1958) and the Advection2D diffusive flux
// templates (src/models/hip/SELF_Advection2D.cpp:66-95, :140-175) -- with one
// viscosity per element instead of one diffusivity.
//
// With the closure on, each RK stage runs, before the stage kernel:
//   k_av_nu     (the first stage of an RK step, and a tendency evaluation;
//               the step's other two stages keep its viscosity and list) the
//               element viscosity nu (modal-decay indicator of the density,
//               or the closure MLP with the indicator as fallback and screen),
//               and the list of elements with nu > 0: one lane per element for
//               the indicator, warp-wide for the few elements that need the
//               MLP or the wave speed;
//   k_av_grad   the listed elements only: the BR1 gradient of the four
//               conservative variables from the averaged traces of the stage's
//               trace cache, the contravariant viscous volume flux
//               -(dsdx^T nu grad q) and the face traces of nu grad q;
//   the stage   kernel adds the viscous volume flux to its contravariant flux
//               and, on exchanged sides, -1/2 (nu grad q_in + nu grad q_ex) . n
//               nScale to its face flux, the exterior value coming from the
//               neighbour's traces; physical sides carry no viscous flux.
// Only elements with nu > 0 form the gradient and write viscous terms; the
// stage kernel reads them only where nu > 0 (the rest add exact zeros).
//
// Modal decay indicator (Persson & Peraire, AIAA 2006-112): c_kl are the
// orthonormal Legendre modes of the density, S = sum_{max(k,l)=N} c^2 /
// sum c^2, s = log10 S, activation a = 0 below s0 - kappa, 1 above s0 + kappa,
// (1 + sin(pi (s - s0) / (2 kappa))) / 2 between; nu = a c_av h / N lambda with
// lambda = max over nodes of |u| + c and h = sqrt(element area).
//
// Closure MLP: 36 features (per variable, density then total energy, the
// energy fractions of the six highest shells max(k,l), xi-degrees and
// eta-degrees, log-scaled) -> 32 -> 32 -> 1, ReLU, bfloat16 weights, float32
// accumulation, output clamp(z, 0, 1) replaces a.
#pragma once

#include <cuda_bf16.h>

#include <atomic>

#include "fused_stage.cuh"

namespace selfgpu {

constexpr int kMlpIn = 36, kMlpHidden = 32;
// row strides of the weight matrices in shared memory: odd, so that the lanes'
// (one unit each) reads of a column fall into distinct banks
constexpr int kW1Stride = kMlpIn + 1, kW2Stride = kMlpHidden + 1;
constexpr int kMlpWeights = kMlpHidden * kMlpIn + kMlpHidden * kMlpHidden + kMlpHidden;  // bf16 values
constexpr int kMlpFloats = kMlpHidden + kMlpHidden + 1 + 2 * kMlpIn;                    // b1 b2 b3 fmin fmax
constexpr double kAvPi = 3.141592653589793;                                             // 4 atan(1)
constexpr float kMlpRangeMargin = 0.05f;
// Screening: an element whose modal decay lies more than kMlpGate decades
// below the start of the activation ramp (s < s0 - kappa - kMlpGate) is smooth
// by a wide margin and gets a = 0 without evaluating the MLP.
constexpr double kMlpGate = 1.0;

enum AvMode { AV_OFF = 0, AV_INDICATOR = 1, AV_MLP = 2 };

struct AvArgs {
  int nEl;
  int mode;  // AV_INDICATOR or AV_MLP
  const double* q;
  const double* dsdx;
  const double* J;
  const double* nHat;
  const double* nScale;
  const int* sideInfo;
  const void* trIn;     // trace cache of this stage (bulk type); conservative traces are fields 0..3
  const double* presc;  // prescribed solution boundary (P,4,4,nEl) or null
  const double* hEl;    // element size sqrt(area), (nEl)
  double gamma, avC, s0, kappa;
  double* nu;          // element viscosity (nEl)
  float* act;          // activation applied (nEl)
  float* actInd;       // indicator activation (nEl), written in AV_MLP mode
  int* fallbacks;      // AV_MLP counters: [0] features outside the training range, [1] MLP evaluations
  int* activeCount;    // elements with nu > 0, written by the viscosity kernel's last block
  int* nuState;        // its running count and the blocks that have finished, zero between launches
  int* activeList;     // their ids (nEl capacity)
  void* visc;          // contravariant viscous volume flux (P*P, 2, 4, nEl), bulk type
  void* vtr;           // per (element, side): nu grad q traces at [i + P (d + 2 v)], bulk type
  const __nv_bfloat16* mlpW;  // W1 (32 x 36, row-major), W2 (32 x 32), w3 (32)
  const float* mlpB;          // b1 (32), b2 (32), b3, fmin (36), fmax (36)
  double T[kMaxP * kMaxP];    // modal matrix T(k,i) = w_i Lt_k(x_i) at [k + P i]
  double dgM[kMaxP * kMaxP];
  double bM[2 * kMaxP];
  double qw[kMaxP];
};

template <typename R>
__device__ __forceinline__ R av_log10(R x) {
  if constexpr (sizeof(R) == 8) return log10(x);
  else return log10f(x);
}
template <typename R>
__device__ __forceinline__ R av_sin(R x) {
  if constexpr (sizeof(R) == 8) return sin(x);
  else return sinf(x);
}
template <typename R>
__device__ __forceinline__ R av_sqrt(R x) {
  if constexpr (sizeof(R) == 8) return sqrt(x);
  else return sqrtf(x);
}

// Modal decay activation from the energies of the top shell and of all modes.
template <typename R>
__device__ R activation_of(R top, R total, double s0, double kappa) {
  if (!(top > (R)0) || !(total > (R)0)) return (R)0;
  const R sv = av_log10<R>(top / total);
  if (sv < (R)s0 - (R)kappa) return (R)0;
  if (sv > (R)s0 + (R)kappa) return (R)1;
  return (R)0.5 * ((R)1 + av_sin<R>((R)kAvPi * (sv - (R)s0) / ((R)2 * (R)kappa)));
}

// ------------------------------------------------------ viscosity kernel
// Density modes, activation and screening by a group of lanes per element;
// then, warp wide (warp-level synchronisation only) and only for the warp's
// elements that need them, the MLP where the indicator does not screen the
// element out, and the wave speed where the activation is not zero; the
// viscosity and an entry in the list of active elements.
template <int P, typename R>
struct NuWarpSmem {
  static constexpr int PP = P * P;
  R q[2][PP];  // density, total energy
  R tt[PP];
  R c[2][PP];  // modal energies c^2
  R part[3][P];
  R act[32], lam[32];  // per element of the warp
  float feat[kMlpIn];
  float h1[kMlpHidden];
};

// Orthonormal modal energies of one P x P field of this warp's element:
// c(k,l) = sum_j T(l,j) sum_i T(k,i) q(i,j), then c^2 in place.
template <int P, typename R>
__device__ __forceinline__ void warp_modal_energy(const R* sT, const R* q, R* tt, R* c, int lane) {
  constexpr int PP = P * P;
  for (int o = lane; o < PP; o += 32) {
    const int k = o % P, jj = o / P;
    R acc = (R)0;
#pragma unroll
    for (int m = 0; m < P; ++m) acc = acc + sT[k + P * m] * q[m + P * jj];
    tt[k + P * jj] = acc;
  }
  __syncwarp();
  for (int o = lane; o < PP; o += 32) {
    const int k = o % P, l = o / P;
    R acc = (R)0;
#pragma unroll
    for (int m = 0; m < P; ++m) acc = acc + sT[l + P * m] * tt[k + P * m];
    c[k + P * l] = acc * acc;
  }
  __syncwarp();
}

constexpr int kNuWarps = 4;

// The closure MLP's activation for element e (warp-wide): the density and
// total-energy modes, the 36 features, the two hidden layers and the clamped
// output; the indicator activation actInd stays when a feature lies outside
// the training range (counted).  Lane 0's result is returned on every lane.
template <int P, typename R>
__device__ R warp_mlp_act(const AvArgs& a, const R* sT, NuWarpSmem<P, R>& s, const float* sW1, const float* sW2,
                          const float* sw3, const float* sB, long long e, int lane, R actInd) {
  constexpr int PP = P * P, N = P - 1;
  R act = actInd;
  for (int k = lane; k < PP; k += 32) {
    s.q[0][k] = (R)a.q[k + (long long)PP * (2 + 4 * e)];
    s.q[1][k] = (R)a.q[k + (long long)PP * (3 + 4 * e)];
  }
  __syncwarp();
  warp_modal_energy<P, R>(sT, s.q[0], s.tt, s.c[0], lane);
  warp_modal_energy<P, R>(sT, s.q[1], s.tt, s.c[1], lane);
  if (lane < P) {  // fixed-order sums per eta-degree l, then over l
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      R tot = (R)0;
#pragma unroll
      for (int k = 0; k < P; ++k) tot = tot + s.c[r][k + P * lane];
      s.part[r][lane] = tot;
    }
  }
  __syncwarp();
  if (lane < 2) {
    R total = (R)0;
#pragma unroll
    for (int l = 0; l < P; ++l) total = total + s.part[lane][l];
    s.part[2][lane] = total;
  }
  __syncwarp();
  for (int f = lane; f < kMlpIn; f += 32) {
    const int r = f / 18, grp = (f % 18) / 6, m = N - 5 + f % 6;
    const R* e2 = s.c[r];
    R sum = (R)0;
    if (grp == 0) {
      for (int l = 0; l < m; ++l) sum = sum + e2[m + P * l];
      for (int k = 0; k <= m; ++k) sum = sum + e2[k + P * m];
    } else if (grp == 1) {
      for (int l = 0; l < P; ++l) sum = sum + e2[m + P * l];
    } else {
      for (int k = 0; k < P; ++k) sum = sum + e2[k + P * m];
    }
    const R total = s.part[2][r];
    R qf = total > (R)0 ? sum / total : (R)0;
    if (qf < (R)1e-16) qf = (R)1e-16;
    s.feat[f] = (float)((av_log10<R>(qf) + (R)8) / (R)8);
  }
  __syncwarp();
  {
    float acc = 0.f;  // lane = hidden unit
#pragma unroll 12
    for (int k = 0; k < kMlpIn; ++k) acc = fmaf(sW1[lane * kW1Stride + k], s.feat[k], acc);
    acc = acc + sB[lane];
    s.h1[lane] = acc > 0.f ? acc : 0.f;
  }
  __syncwarp();
  float h2;
  {
    float acc = 0.f;
#pragma unroll 16
    for (int k = 0; k < kMlpHidden; ++k) acc = fmaf(sW2[lane * kW2Stride + k], s.h1[k], acc);
    acc = acc + sB[kMlpHidden + lane];
    h2 = acc > 0.f ? acc : 0.f;
  }
  __syncwarp();
  s.h1[lane] = h2;  // the second hidden layer reuses the first's array
  __syncwarp();
  const float *fmin = sB + 2 * kMlpHidden + 1, *fmax = fmin + kMlpIn;
  bool mine = true;  // this lane's features lie in the training range
  for (int k = lane; k < kMlpIn; k += 32)
    mine = mine && s.feat[k] >= fmin[k] - kMlpRangeMargin && s.feat[k] <= fmax[k] + kMlpRangeMargin;
  const bool inRange = __all_sync(0xffffffffu, mine);
  if (lane == 0) {
    if (a.fallbacks) atomicAdd(a.fallbacks + 1, 1);
    if (inRange) {
      float z = 0.f;
#pragma unroll
      for (int k = 0; k < kMlpHidden; ++k) z = fmaf(sw3[k], s.h1[k], z);
      z = z + sB[2 * kMlpHidden];
      act = (R)(z < 0.f ? 0.f : (z > 1.f ? 1.f : z));
    } else if (a.fallbacks) {
      atomicAdd(a.fallbacks, 1);
    }
  }
  act = __shfl_sync(0xffffffffu, act, 0);
  __syncwarp();
  return act;
}

// Wave speed |u| + c of element e, max over its nodes (warp-wide;
// src/models/SELF_CompressibleIdealGas2D.f90:1090-1110).
template <int P, typename R>
__device__ R warp_wave_speed(const AvArgs& a, long long e, int lane) {
  constexpr int PP = P * P;
  const R gam = (R)a.gamma;
  R lam = (R)0;
  for (int k = lane; k < PP; k += 32) {
    const long long b = k + (long long)PP * 4 * e;
    const R ru = (R)a.q[b], rv = (R)a.q[b + PP], rho = (R)a.q[b + 2 * PP], rE = (R)a.q[b + 3 * PP];
    const R u = ru / rho, v = rv / rho;
    const R ke = (R)0.5 * (ru * u + rv * v);
    const R p = (gam - (R)1) * (rE - ke);
    const R c = av_sqrt<R>(gam * p / rho);
    const R wv = av_sqrt<R>(u * u + v * v) + c;
    if (wv > lam) lam = wv;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const R other = __shfl_xor_sync(0xffffffffu, lam, o);
    if (other > lam) lam = other;
  }
  return lam;
}

// Indicator activation from the totals of all modal energies and of the top
// shell, and whether the MLP must be evaluated (not screened out).
template <typename R>
__device__ __forceinline__ void indicator_act(const AvArgs& a, R total, R top, bool mlp, R& actInd, int& need) {
  actInd = (R)0;
  need = 0;
  if (top > (R)0 && total > (R)0) {
    const R sv = av_log10<R>(top / total);
    if (sv > (R)a.s0 + (R)a.kappa) actInd = (R)1;
    else if (!(sv < (R)a.s0 - (R)a.kappa))
      actInd = (R)0.5 * ((R)1 + av_sin<R>((R)kAvPi * (sv - (R)a.s0) / ((R)2 * (R)a.kappa)));
    need = mlp && !(sv < (R)(a.s0 - a.kappa - kMlpGate));
  }
}

// One group of kNuLanes lanes per element, lane j holding row j of the density:
// the xi transform is the lane's own, the eta transform reads the group's rows
// from shared memory, and lane l sums eta-degree l -- the operations and
// summation orders of one thread that does it all.  (One lane per element held
// 64 densities, left 4 of 5 resident warps idle on a mesh of 10 560 elements
// and took 15 us there in FP64 at P = 8, each lane's chain of 1 024
// multiply-adds and 64 uncoalesced loads being the time.)
template <int P>
constexpr int nu_lanes() {
  return P <= 2 ? 2 : (P <= 4 ? 4 : 8);
}

template <int P, typename R>
__global__ void __launch_bounds__(32 * kNuWarps) k_av_nu(const AvArgs a) {
  constexpr int PP = P * P, N = P - 1, GL = nu_lanes<P>(), GE = 32 / GL;  // elements per warp
  __shared__ NuWarpSmem<P, R> ws[kNuWarps];
  __shared__ R sTt[kNuWarps][GE][PP + 1];  // xi transforms (k, jj) at [jj + P k]
  __shared__ R sT[PP];
  __shared__ float sW1[kMlpHidden * kW1Stride], sW2[kMlpHidden * kW2Stride], sw3[kMlpHidden], sB[kMlpFloats];
  // (see k_av_grad)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const bool mlp = (a.mode == AV_MLP) && (P >= 6);
  for (int k = threadIdx.x; k < PP; k += blockDim.x) sT[k] = (R)a.T[k];
  if (mlp) {
    for (int k = threadIdx.x; k < kMlpHidden * kMlpIn; k += blockDim.x)
      sW1[k / kMlpIn * kW1Stride + k % kMlpIn] = __bfloat162float(a.mlpW[k]);
    for (int k = threadIdx.x; k < kMlpHidden * kMlpHidden; k += blockDim.x)
      sW2[k / kMlpHidden * kW2Stride + k % kMlpHidden] = __bfloat162float(a.mlpW[kMlpHidden * kMlpIn + k]);
    for (int k = threadIdx.x; k < kMlpHidden; k += blockDim.x)
      sw3[k] = __bfloat162float(a.mlpW[kMlpHidden * kMlpIn + kMlpHidden * kMlpHidden + k]);
    for (int k = threadIdx.x; k < kMlpFloats; k += blockDim.x) sB[k] = a.mlpB[k];
  }
  __syncthreads();
  const int w = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int grp = lane / GL, r = lane % GL;  // the lane's element of the warp's GE, and its row / eta-degree
  const int leader = grp * GL;
  NuWarpSmem<P, R>& s = ws[w];
  R* tt = sTt[w][grp];
  // a warp's elements are spread over the mesh, so that the few that need the
  // MLP or the wave speed, done warp-wide, are spread over the warps too
  const long long nW = (long long)gridDim.x * kNuWarps;
  for (long long base = (long long)blockIdx.x * kNuWarps + w; base < a.nEl; base += GE * nW) {
    const long long e = base + (long long)grp * nW;
    const bool live = e < a.nEl;
    if (live && r < P) {
      R q[P];
      const double* qg = a.q + (long long)PP * (2 + 4 * e) + P * r;
#pragma unroll
      for (int m = 0; m < P; ++m) q[m] = (R)qg[m];
#pragma unroll
      for (int k = 0; k < P; ++k) {
        R acc = (R)0;
#pragma unroll
        for (int m = 0; m < P; ++m) acc = acc + sT[k + P * m] * q[m];
        tt[r + P * k] = acc;
      }
    }
    __syncwarp();
    R tot = (R)0, topL = (R)0;  // eta-degree r: all xi-degrees, and xi-degree N
    if (live && r < P) {
#pragma unroll
      for (int k = 0; k < P; ++k) {
        R acc = (R)0;
#pragma unroll
        for (int m = 0; m < P; ++m) acc = acc + sT[r + P * m] * tt[m + P * k];
        const R c = acc * acc;
        tot = tot + c;
        if (k == N) topL = c;
      }
      if (r == N) topL = tot;
    }
    R total = (R)0, topS = (R)0;
#pragma unroll
    for (int l = 0; l < P; ++l) {
      total = total + __shfl_sync(0xffffffffu, tot, leader + l);
      topS = topS + __shfl_sync(0xffffffffu, topL, leader + l);
    }
    R actInd = (R)0;
    int need = 0;
    if (live && r == 0) {
      indicator_act<R>(a, total, topS, mlp, actInd, need);
      s.act[grp] = actInd;
    }
    const unsigned needMask = __ballot_sync(0xffffffffu, need);
    __syncwarp();
    for (unsigned mk = needMask; mk; mk &= mk - 1) {
      const int ln = __ffs(mk) - 1, b = ln / GL;
      const R act = warp_mlp_act<P, R>(a, sT, s, sW1, sW2, sw3, sB, base + (long long)b * nW, lane,
                                       __shfl_sync(0xffffffffu, actInd, ln));
      if (lane == 0) s.act[b] = act;
      __syncwarp();
    }
    const bool mine = live && r == 0;  // the element's lane
    const R act = mine ? s.act[grp] : (R)0;
    const unsigned actMask = __ballot_sync(0xffffffffu, act != (R)0);
    for (unsigned mk = actMask; mk; mk &= mk - 1) {
      const int b = (__ffs(mk) - 1) / GL;
      const R lam = warp_wave_speed<P, R>(a, base + (long long)b * nW, lane);
      if (lane == 0) s.lam[b] = lam;
    }
    __syncwarp();
    double nu = 0.0;
    if (mine) {
      if (act != (R)0) nu = (double)act * a.avC * a.hEl[e] / (double)N * (double)s.lam[grp];
      a.nu[e] = nu;
      a.act[e] = (float)act;
      if (mlp && a.actInd) a.actInd[e] = (float)actInd;
    }
    const unsigned nzMask = __ballot_sync(0xffffffffu, nu != 0.0);
    if (nzMask) {
      int b0 = 0;
      if (lane == 0) b0 = atomicAdd(&a.nuState[0], __popc(nzMask));
      b0 = __shfl_sync(0xffffffffu, b0, 0);
      if (nu != 0.0) a.activeList[b0 + __popc(nzMask & ((1u << lane) - 1u))] = (int)e;
    }
    __syncwarp();
  }
  // the last block publishes the count and leaves the state zero for the next
  // launch (a memset before each launch cost a gap of its own)
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&a.nuState[1], 1) == (int)gridDim.x - 1) {
      __threadfence();
      *a.activeCount = atomicExch(&a.nuState[0], 0);
      a.nuState[1] = 0;
    }
  }
}

// ------------------------------------------------------ viscous-term kernel
// The active elements only (the list the viscosity kernel filled): BR1
// gradient scaled by nu, contravariant viscous flux and face traces of nu grad q.
template <int P, typename R>
struct GradSmem {
  static constexpr int PP = P * P;
  R q[4][PP];
  R dsdx[4][PP];  // (dsdx11, dsdx21, dsdx12, dsdx22) per node
  R avg[4][4][P];
  R nh[4][P][2], ns[4][P];
  R g[2][4][PP];  // nu grad q
};

// elements per block: one thread per node and variable
template <int P, typename R>
constexpr int av_elems_per_block() {
  int e = 256 / (4 * P * P);
  if (e < 1) e = 1;
  while (e > 1 && (size_t)e * sizeof(GradSmem<P, R>) > 44 * 1024) --e;
  return e;
}

// A shocked region is a few hundred elements, so the kernel's time is the
// latency of one element's chain (loads, sums, ten divisions per node and
// variable, traces): a thread per (node, variable) and the face metrics in
// shared memory.  (One thread per node doing its four variables in turn, the
// metrics read from global memory for each: 12 us for the 5 % of 10 560
// elements at P = 8 in FP64 that a shock band activates.  Each value stored to
// shared memory as it came, so that the loads waited for one another: 9.1 us on
// the 256x256 Riemann problem at P = 6 in FP32, now 8.1.)
template <int P, typename R, int EPB>
__global__ void __launch_bounds__(EPB * 4 * P * P) k_av_grad(const AvArgs a) {
  constexpr int PP = P * P, N = P - 1, VS = visc_side_stride<P>(), TPE = 4 * PP;
  constexpr int TS = trace_side_stride<P, 9, R>();
  __shared__ GradSmem<P, R> sm_all[EPB];
  __shared__ double sdg[PP], sb[2 * P], sw[P];
  const int tid = threadIdx.x;
  const int slot = tid / TPE;
  const int u = tid - slot * TPE;  // thread of the element
  const int v = u / PP;            // variable (and metric component)
  const int t = u - v * PP;        // node
  const int i = t % P, j = t / P;
  GradSmem<P, R>& sm = sm_all[slot];
  for (int k = tid; k < PP; k += blockDim.x) sdg[k] = a.dgM[k];
  for (int k = tid; k < 2 * P; k += blockDim.x) sb[k] = a.bM[k];
  for (int k = tid; k < P; k += blockDim.x) sw[k] = a.qw[k];
  __syncthreads();
  // A programmatic dependent launch, as the stage kernel's: what precedes the
  // wait reads kernel parameters only, and the next kernel of the stage may
  // start while this one runs.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const R* trIn = reinterpret_cast<const R*>(a.trIn);
  // this thread's entry of the list, read along with the count
  long long base = (long long)blockIdx.x * EPB;
  int first = base + slot < a.nEl ? a.activeList[base + slot] : 0;
  const int count = *a.activeCount;
  // every block runs the same number of rounds (block-uniform barriers)
  for (; base < count; base += (long long)gridDim.x * EPB) {
    const bool live = base + slot < count;
    const long long e = live ? first : 0;
    first = base + slot + (long long)gridDim.x * EPB < a.nEl ? a.activeList[base + slot + (long long)gridDim.x * EPB] : 0;
    R nu = (R)0, Jij = (R)1;
    if (live) {
      // averaged conservative traces (BassiRebaySides) with the stage's
      // exterior states; the first task's connectivity, then all the element's
      // values, are requested before any is used
      auto trace_average = [&](int k, int si2, int si3, int bcid, R L) {
        const int w = k / (4 * P), c = k - w * 4 * P, s1 = c / P, ii = c % P;
        const R* own = trIn + (long long)TS * (s1 + 4 * e) + ii;
        R X = (R)0;
        if (bcid == 0) {
          const long long e2 = si2 - 1;
          const int s2 = si3 / 10 - 1, flip = si3 % 10;
          X = trIn[(long long)TS * (s2 + 4 * e2) + (flip ? N - ii : ii) + P * w];
        } else if (si2 == 0) {  // physical side: the boundary condition's exterior state
          if (bcid == SG_BC_NONORMALFLOW) {
            if (w < 2) {
              const double* nh = a.nHat + 2 * (ii + (long long)P * (s1 + 4 * e));
              R x0, x1;
              reflect<R>(own[0], own[P], nh[0], nh[1], x0, x1);
              X = w == 0 ? x0 : x1;
            } else {
              X = L;
            }
          } else if ((bcid == SG_BC_PRESCRIBED || bcid == SG_BC_RADIATION) && a.presc) {
            X = (R)a.presc[ii + (long long)P * (w + 4 * (s1 + 4 * e))];
          }
        }
        return (R)0.5 * (L + X);
      };
      int si2 = 0, si3 = 0, si4 = 1;
      R L = (R)0, X = (R)0;
      const int tw = u / (4 * P), tc = u - tw * 4 * P, ts = tc / P, ti = tc % P;
      if (u < 16 * P) {
        const int* si = a.sideInfo + 5 * (ts + 4 * e);
        si2 = si[2], si3 = si[3], si4 = si[4];
        L = trIn[(long long)TS * (ts + 4 * e) + ti + P * tw];
      }
      const double qv = a.q[t + (long long)PP * (v + 4 * e)], dv = a.dsdx[v + 4 * (t + (long long)PP * e)];
      const double nuE = a.nu[e], Jv = a.J[t + (long long)PP * e];
      double n1 = 0.0, n2 = 0.0, ns = 0.0;
      if (u < 4 * P) {
        n1 = a.nHat[2 * (u + (long long)P * 4 * e)];
        n2 = a.nHat[2 * (u + (long long)P * 4 * e) + 1];
        ns = a.nScale[u + (long long)P * 4 * e];
      }
      if (u < 16 * P) X = trace_average(u, si2, si3, si4, L);
      nu = (R)nuE;
      Jij = (R)Jv;
      sm.q[v][t] = (R)qv;
      sm.dsdx[v][t] = (R)dv;
      if (u < 4 * P) {
        sm.nh[u / P][u % P][0] = (R)n1;
        sm.nh[u / P][u % P][1] = (R)n2;
        sm.ns[u / P][u % P] = (R)ns;
      }
      if (u < 16 * P) sm.avg[ts][tw][ti] = X;
      for (int k = u + TPE; k < 16 * P; k += TPE) {  // (P = 2 and 3)
        const int w = k / (4 * P), c = k - w * 4 * P, s1 = c / P, ii = c % P;
        const int* si = a.sideInfo + 5 * (s1 + 4 * e);
        const R Lk = trIn[(long long)TS * (s1 + 4 * e) + ii + P * w];
        sm.avg[s1][w][ii] = trace_average(k, si[2], si[3], si[4], Lk);
      }
    }
    __syncthreads();
    // BR1 gradient (GradientBR_MappedScalar2D, src/SELF_MappedData.f90:990-1074) scaled by nu,
    // and the contravariant viscous flux (src/models/hip/SELF_Advection2D.cpp:66-95)
    if (live) {
      R* visc = reinterpret_cast<R*>(a.visc);
      R gx = (R)0, gy = (R)0;
#pragma unroll
      for (int ii = 0; ii < P; ++ii) {
        const R qa = sm.q[v][ii + P * j], qb = sm.q[v][i + P * ii];
        R f1 = qa * sm.dsdx[0][ii + P * j];
        R f2 = qb * sm.dsdx[2][i + P * ii];
        gx = gx + (R)sdg[ii + P * i] * f1 + (R)sdg[ii + P * j] * f2;
        f1 = qa * sm.dsdx[1][ii + P * j];
        f2 = qb * sm.dsdx[3][i + P * ii];
        gy = gy + (R)sdg[ii + P * i] * f1 + (R)sdg[ii + P * j] * f2;
      }
      R f1 = sm.avg[1][v][j] * sm.nh[1][j][0] * sm.ns[1][j];
      R f2 = sm.avg[3][v][j] * sm.nh[3][j][0] * sm.ns[3][j];
      gx = gx + (f1 * (R)sb[i + P] + f2 * (R)sb[i]) / (R)sw[i];
      f1 = sm.avg[2][v][i] * sm.nh[2][i][0] * sm.ns[2][i];
      f2 = sm.avg[0][v][i] * sm.nh[0][i][0] * sm.ns[0][i];
      gx = gx + (f1 * (R)sb[j + P] + f2 * (R)sb[j]) / (R)sw[j];
      f1 = sm.avg[1][v][j] * sm.nh[1][j][1] * sm.ns[1][j];
      f2 = sm.avg[3][v][j] * sm.nh[3][j][1] * sm.ns[3][j];
      gy = gy + (f1 * (R)sb[i + P] + f2 * (R)sb[i]) / (R)sw[i];
      f1 = sm.avg[2][v][i] * sm.nh[2][i][1] * sm.ns[2][i];
      f2 = sm.avg[0][v][i] * sm.nh[0][i][1] * sm.ns[0][i];
      gy = gy + (f1 * (R)sb[j + P] + f2 * (R)sb[j]) / (R)sw[j];
      gx = gx / Jij;
      gy = gy / Jij;
      gx = gx * nu;
      gy = gy * nu;
      sm.g[0][v][t] = gx;
      sm.g[1][v][t] = gy;
      const R c1 = -(sm.dsdx[0][t] * gx + sm.dsdx[1][t] * gy);
      const R c2 = -(sm.dsdx[2][t] * gx + sm.dsdx[3][t] * gy);
      visc[t + (long long)PP * (0 + 2 * (v + 4 * e))] = c1;
      visc[t + (long long)PP * (1 + 2 * (v + 4 * e))] = c2;
    }
    __syncthreads();
    // face traces of nu grad q (VectorBoundaryInterp_2D, src/SELF_Lagrange.f90:2284-2316)
    if (live) {
      R* vo = reinterpret_cast<R*>(a.vtr) + (long long)4 * VS * e;
      for (int k = u; k < 4 * 8 * P; k += TPE) {
        const int ii = k % P, d = (k / P) % 2, vv = (k / (2 * P)) % 4, s1 = k / (8 * P);
        vo[s1 * VS + ii + P * (d + 2 * vv)] = face_trace<P, R>(sm.g[d][vv], sb, s1, ii);
      }
    }
    __syncthreads();  // the slot's arrays are reused by the next round
  }
}

// Closure features of a stored FP64 state (training-data harvest): per element
// the indicator activation and the 36 features, one warp per element.  Both
// modal transforms are FP64 tensor-core products (m8n8k4, a P x P field padded
// with zeros), the matrix held in registers as both products' operand, the
// first product's result moved into the second's operand layout by shuffles;
// then one lane per feature.  (A block per element whose first two threads
// summed and took the logarithms alone: 115 us for 16 384 elements at P = 8.)
template <int P>
__global__ void __launch_bounds__(32 * kNuWarps) k_closure_features(const double* __restrict__ q, int nEl,
                                                                    const AvArgs a, float* __restrict__ act,
                                                                    float* __restrict__ feat) {
  constexpr int PP = P * P, N = P - 1, KK = (P + 3) / 4;
  __shared__ double cc[kNuWarps][2][PP];
  const int w = threadIdx.x / 32, lane = threadIdx.x % 32, row = lane >> 2, col = lane & 3;
  // T(row, col + 4 kk): rows of T as the first product's A, columns of T^T as the second's B
  double T[KK];
#pragma unroll
  for (int kk = 0; kk < KK; ++kk) T[kk] = row < P && col + 4 * kk < P ? a.T[row + P * (col + 4 * kk)] : 0.0;
  auto mma = [](double& c0, double& c1, double x, double y) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c0), "+d"(c1)
                 : "d"(x), "d"(y));
  };
  for (long long e = (long long)blockIdx.x * kNuWarps + w; e < nEl; e += (long long)gridDim.x * kNuWarps) {
    double total[2] = {0.0, 0.0};
#pragma unroll
    for (int r = 0; r < 2; ++r) {  // density, total energy
      if (r == 1 && (P < 6 || !feat)) break;
      const double* qe = q + (long long)PP * (2 + r + 4 * e);
      double t0 = 0.0, t1 = 0.0;  // sum_m T(k, m) q(m, jj) at k = row, jj = 2 col, 2 col + 1
#pragma unroll
      for (int kk = 0; kk < KK; ++kk) {
        const int m = col + 4 * kk;
        mma(t0, t1, T[kk], row < P && m < P ? qe[m + P * row] : 0.0);
      }
      double c0 = 0.0, c1 = 0.0;  // sum_m (..)(k, m) T(l, m) at k = row, l = 2 col, 2 col + 1
#pragma unroll
      for (int kk = 0; kk < KK; ++kk) {
        const int src = (lane & 28) + ((col + 4 * kk) >> 1);
        const double x0 = __shfl_sync(0xffffffffu, t0, src), x1 = __shfl_sync(0xffffffffu, t1, src);
        mma(c0, c1, (col & 1) ? x1 : x0, T[kk]);
      }
      c0 = c0 * c0;
      c1 = c1 * c1;
      if (row < P && 2 * col < P) cc[w][r][row + P * 2 * col] = c0;
      if (row < P && 2 * col + 1 < P) cc[w][r][row + P * (2 * col + 1)] = c1;
      double s = c0 + c1;  // (the padding's are zero)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      total[r] = s;
    }
    __syncwarp();
    // lane tasks: the features, then (task kMlpIn) the activation
    const int f0 = (P >= 6 && feat) ? lane : (lane == 0 ? kMlpIn : kMlpIn + 1);
    for (int f = f0; f <= kMlpIn; f += 32) {
      const bool top = f == kMlpIn;
      const int r = top ? 0 : f / 18, grp = top ? 0 : (f % 18) / 6, m = top ? N : N - 5 + f % 6;
      const double* e2 = cc[w][r];
      double sum = 0.0;
      if (grp == 0) {
        for (int l = 0; l < m; ++l) sum = sum + e2[m + P * l];
        for (int k = 0; k <= m; ++k) sum = sum + e2[k + P * m];
      } else if (grp == 1) {
        for (int l = 0; l < P; ++l) sum = sum + e2[m + P * l];
      } else {
        for (int k = 0; k < P; ++k) sum = sum + e2[k + P * m];
      }
      const double t = r ? total[1] : total[0];
      if (top) {
        if (act) act[e] = (float)activation_of<double>(sum, t, a.s0, a.kappa);
      } else {
        double x = t > 0.0 ? sum / t : 0.0;
        if (x < 1e-16) x = 1e-16;
        feat[kMlpIn * e + f] = (float)((log10(x) + 8.0) / 8.0);
      }
    }
    __syncwarp();
  }
}

struct QwArr {
  double w[kMaxP];
};

// formNu: form the element viscosity and the active list (the first stage of
// an RK step, or a tendency evaluation); otherwise the viscous terms are
// formed with the viscosity the step's first stage found.
template <int P, typename R>
cudaError_t launch_av_pair(const AvArgs& a, cudaStream_t st, int numSMs, bool formNu) {
  constexpr int EPB = av_elems_per_block<P, R>();
  auto grad = [&]() { return launch_dependent(k_av_grad<P, R, EPB>, 4 * numSMs, EPB * 4 * P * P, st, a); };
  if (!formNu) return grad();
  // one wave of resident blocks, each warp striding over its share of the
  // elements (a partial second wave would run at low occupancy)
  static std::atomic<int> nuPerSM{0};  // resident blocks per SM, one instantiation per (P, R)
  if (nuPerSM.load() == 0) {
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_av_nu<P, R>, 32 * kNuWarps, 0) != cudaSuccess || nb < 1)
      nb = 4;
    nuPerSM.store(nb);
  }
  const int perBlock = kNuWarps * 32 / nu_lanes<P>();  // elements
  const long long nuBlocks = ((long long)a.nEl + perBlock - 1) / perBlock;
  const long long cap = (long long)nuPerSM.load() * numSMs;
  const int g1 = (int)(nuBlocks < cap ? nuBlocks : cap);
  cudaError_t e = launch_dependent(k_av_nu<P, R>, g1, 32 * kNuWarps, st, a);
  return e == cudaSuccess ? grad() : e;
}

template <typename R>
cudaError_t launch_av_prep_impl(int P, const AvArgs& a, cudaStream_t st, int numSMs, bool formNu) {
  switch (P) {
    case 2: return launch_av_pair<2, R>(a, st, numSMs, formNu);
    case 3: return launch_av_pair<3, R>(a, st, numSMs, formNu);
    case 4: return launch_av_pair<4, R>(a, st, numSMs, formNu);
    case 5: return launch_av_pair<5, R>(a, st, numSMs, formNu);
    case 6: return launch_av_pair<6, R>(a, st, numSMs, formNu);
    case 7: return launch_av_pair<7, R>(a, st, numSMs, formNu);
    case 8: return launch_av_pair<8, R>(a, st, numSMs, formNu);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace selfgpu
