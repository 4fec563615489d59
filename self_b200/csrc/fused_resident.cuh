// All RK stages of an rk3 call in one launch with the state held on chip, for
// meshes whose tiles of elements all fit resident CTAs at once.
//
// A CTA works on tiles of TmaTraits::EPG elements (one thread per node, as a
// group of k_fused_stage_tma).  With one tile per CTA the solution, the RK
// register, the metric terms and the model fields live in registers from the
// first stage to the last; with several (kMany; the CTA takes them in turn in
// every stage) the solution and the register live in shared memory and the
// metric terms and fields are read from L2.  Otherwise a stage's only global
// traffic is the face traces: each CTA publishes its elements' traces and reads
// its neighbours'.  There is no grid barrier and no
// fence: every published value travels with the number of the trace set it
// belongs to in one 16-byte (FP32 bulk: 8-byte) store, which is a single
// relaxed access, and the reader polls the value itself until its number is
// the expected one.  A stage of a small mesh is bound by that exchange's round
// trip and the latency of one element's phases, so the volume sums run on the
// warps the face threads leave free while those poll.
//
// The trace sets alternate between two buffers.  A CTA publishes set s + 2 only
// after its neighbours' set s + 1 has arrived, and a neighbour publishes set
// s + 1 only after it has read set s, so no unread value is overwritten.  Set
// numbers grow from launch to launch (a counter in device memory that the last
// CTA of a launch advances), so a value of an earlier launch, or of an earlier
// replay of a graph that holds this launch, never matches.
//
// Per stage, three CTA barriers:
//   traces of the current solution (published, and kept for the tile's own
//   faces), contravariant flux | volume sums and, on the face threads,
//   neighbour traces and Riemann flux | lift, 1/J, source, RK update
// The phases evaluate k_fused_stage_tma's expressions, so the results are
// those of the stage launches bit for bit.
//
// Waits are bounded (StageArgs::waitCycles): on timeout the CTA sets the error
// word and returns without writing the solution.  The launch is cooperative
// (all CTAs resident).
#pragma once

#include "fused_stage_tma.cuh"

namespace selfgpu {

// Counter of the exchange sets used so far and the CTAs that have finished the
// current launch.
struct ResidentEpoch {
  unsigned long long sets;
  unsigned done;
};

// Most tiles per CTA: four, three with the reference's roundings, fewer where
// the smallest meshes of that many tiles were slower than their stage launches.
// us per stage in calls of 20 steps on nx x nx meshes, stage launches -> this
// launch, for CompressibleIdealGas2D FP64 at P = 8 (1 184 elements per tile of
// the CTAs): one tile 6.5 -> 2.7 (34x34), two 9.6 -> 6.2 (48x48), three 10.3 ->
// 8.9 (52x52), four 13.0 -> 11.7 (60x60).  Over all P, models and forms on 21
// meshes each, the ratio is at worst 0.65 for one tile, 0.91 for two (0.99 for
// CompressibleIdealGas2D FP32 at P = 3), 1.01 for three and 0.93 for four, but
// for those excepted here:
//   CompressibleIdealGas2D at P = 3: three 1.04 FP64, 1.06 reference roundings,
//     1.12 FP32;
//   CompressibleIdealGas2D FP64 at P = 4: three 1.02, four 1.22; at P = 6: four
//     1.07;
//   ShallowWater with the reference's roundings at P = 6: three 1.06.
// Least steps of a call.  A call pays some 6 us to load and store the state and
// to start all CTAs at once.  With one tile a single step wins that back (ratio
// 0.91 at worst); with several it takes as many steps as the stages' gain needs
// on the smallest meshes of the tile count.  us per call, stage launches -> this
// launch, with the reference's roundings at P = 8: ShallowWater two tiles one
// step 22.6 -> 26.8, two 45.2 -> 45.5; CompressibleIdealGas2D three tiles three
// steps 123 -> 129, four 164 -> 169, 20 819 -> 816.  In the other forms one step
// of three or four tiles: at P = 8 CompressibleIdealGas2D FP64 40.8 -> 41.3,
// ShallowWater 35.0 -> 37.1, FP32 28.8 -> 31.1; at P = 6 LinearShallowWater FP64
// 24.7 -> 26.8, CompressibleIdealGas2D FP32 30.8 -> 34.5, two steps 59.5 -> 61.7.
// LinearShallowWater elsewhere and P = 5 and 7 gain with one step too (P = 5
// FP64 four tiles, ratio 0.81 to 0.96).
inline namespace SELFGPU_FORM_NS {
template <int P, class Phys, typename R>
__host__ __device__ constexpr int resident_tiles() {
  constexpr bool cig = Phys::NV == 4, prod = sizeof(R) == 8 && !ref_rounding<R>();
  if (cig && (P == 3 || (P == 4 && prod))) return 2;
  if (ref_rounding<R>()) return P == 6 && Phys::kLaggedVelocity ? 2 : 3;
  return cig && P == 6 && prod ? 3 : 4;
}
template <int P, class Phys, typename R>
__host__ __device__ constexpr int resident_min_steps(int tiles) {
  constexpr bool cig = Phys::NV == 4, lsw = !cig && !Phys::kLaggedVelocity;
  if (tiles <= 1) return 1;
  if (ref_rounding<R>()) {
    if (P == 6 || P == 8) return tiles == 2 ? 2 : 4;
    return tiles == 2 && (P == 5 || (P < 6 && lsw)) ? 1 : 2;
  }
  if (P == 5 || P == 7 || (lsw && !(P == 6 && sizeof(R) == 8))) return 1;
  return tiles > 2 || (cig && P == 3 && sizeof(R) == 4) ? 2 : 1;
}
}  // namespace SELFGPU_FORM_NS

struct ResidentArgs {
  int nStages;      // 3 per RK step
  int fresh;        // 1: the trace caches are stale, form the traces of q first
  double dt;
  double rkA[3], rkG[3];
  const void* trIn;   // trace and velocity caches of the solution (fresh = 0)
  const void* velIn;
  void* trOut;        // caches of the final solution
  void* velOut;
  void* xch[2];       // published traces: per (element, side) NT x P (value, set number) pairs
  int tiles;          // tiles per CTA (the launch's grid takes tile b, b + grid, ...)
  ResidentEpoch* epoch;
};

// One published value.
struct __align__(16) Pub64 {
  double v;
  unsigned long long set;
};
struct __align__(8) Pub32 {
  float v;
  unsigned set;
};
__device__ __forceinline__ void publish(Pub64* p, double v, unsigned long long set) {
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p),
               "l"(__double_as_longlong(v)), "l"(set)
               : "memory");
}
__device__ __forceinline__ void publish(Pub32* p, float v, unsigned long long set) {
  const unsigned long long u = ((set & 0xffffffffull) << 32) | __float_as_uint(v);
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(u) : "memory");
}
// The value and whether it belongs to the set.
__device__ __forceinline__ bool peek(const Pub64* p, unsigned long long set, double& v) {
  unsigned long long a, s;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
               : "=l"(a), "=l"(s)
               : "l"(p)
               : "memory");
  v = __longlong_as_double(a);
  return s == set;
}
__device__ __forceinline__ bool peek(const Pub32* p, unsigned long long set, float& v) {
  unsigned long long u;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(u) : "l"(p) : "memory");
  v = __uint_as_float((unsigned)u);
  return (unsigned)(u >> 32) == (unsigned)set;
}

template <int P, class Phys, typename R>
struct ResTraits {
  using T = TmaTraits<P, Phys, R>;
  using Pub = typename std::conditional<sizeof(R) == 8, Pub64, Pub32>::type;
  // node fields apart from the fluxes (a thread writes its next flux while
  // others still form traces; within the element's arrays where TmaTraits keeps
  // them apart already), then (one tile per CTA) the tile's own traces
  static constexpr int arrays = T::EPG * (T::EB + T::kDiv);
  static constexpr int oFields = T::kSep ? T::oN : arrays;
  static constexpr int FB = T::kSep ? T::EB : T::NT * T::FS, OB = 4 * T::NT * P;  // per element
  static constexpr int oOwn = arrays + (T::kSep ? 0 : T::EPG * FB);
  static constexpr int values(bool many) { return oOwn + (many ? 0 : T::EPG * OB); }
  // 128 registers per thread: the node state of a tile is about 50
  static constexpr int kMinCtas = 65536 / (128 * T::TPE) > 1 ? 65536 / (128 * T::TPE) : 1;
  // a tile's state in shared memory (kMany): solution and register, the lagged
  // velocities of its face nodes
  static constexpr int nodes = T::EPG * T::PP, faces = T::EPG * 4 * P;
  static constexpr int tileBytes =
      (nodes * T::NV * (8 + (int)sizeof(R)) + (Phys::kLaggedVelocity ? 4 * faces * (int)sizeof(R) : 0) + 15) / 16 * 16;
};

template <int P, class Phys, typename R, bool kMany>
__global__ void __launch_bounds__(TmaTraits<P, Phys, R>::TPE, ResTraits<P, Phys, R>::kMinCtas)
    k_fused_resident(const StageArgs a, const ResidentArgs ra) {
  using T = TmaTraits<P, Phys, R>;
  using X = ResTraits<P, Phys, R>;
  using Pub = typename X::Pub;
  constexpr int NV = T::NV, NT = T::NT, NF = T::NF, PP = T::PP, TS = T::TS, TPE = T::TPE, N = P - 1;
  constexpr int FS = T::FS, SS = T::SS, EPG = T::EPG, EB = T::EB;
  constexpr bool kLSW = (NV == 3 && !Phys::kLaggedVelocity);
  constexpr bool kSW = Phys::kLaggedVelocity;
  // an orientation per warp (tile_traces), us per stage, tasks in common -> per
  // warp: LinearShallowWater FP64 34x34 1.63 -> 1.54, 64x64 7.70 -> 7.43,
  // CompressibleIdealGas2D FP64 64x64 12.5 -> 11.9, FP32 34x34 2.43 -> 2.35 but
  // 64x64 9.39 -> 9.85; reference roundings 3.34 -> 3.46
  constexpr bool kWarpTraces = T::kSwz && !ref_rounding<R>() && !(kMany && NV == 4 && sizeof(R) == 4);
  constexpr int kGeo = geo_kind<P, R>();
  constexpr GeoRec kRec = geo_rec(P, kGeo);
  constexpr int kWm = kRec.wm, rBytes = kRec.bytes, rNhat = kRec.oNhat, rNs = kRec.oNs, rJ = kRec.oJ, rSi = kRec.oSi;
  __shared__ __align__(16) R sm[X::values(kMany)];
  __shared__ __align__(16) double sdg[PP];
  __shared__ R sdgR[T::kRegDiv ? PP : 1];
  // bMatrix, and the quadrature weights (reference roundings) or their
  // reciprocals, in the bulk type
  __shared__ R sb[2 * P], sw[P];
  __shared__ unsigned long long sSet;
  __shared__ int sOk;
  extern __shared__ __align__(16) unsigned char state[];  // kMany: the tiles' state
  const int t = threadIdx.x;
  for (int k = t; k < PP; k += TPE) {
    const double d = a.dgM[k / P + P * (k % P)];
    sdg[T::dgat(k / P, k % P)] = d;
    if constexpr (T::kRegDiv) sdgR[T::dgat(k / P, k % P)] = (R)d;
  }
  for (int k = t; k < 2 * P; k += TPE) sb[k] = k < P ? bm_left<R>(a, k) : bm_right<R, P>(a, k - P);
  for (int k = t; k < P; k += TPE) sw[k] = ref_rounding<R>() ? (R)a.qw[k] : (R)(1.0 / a.qw[k]);
  if (t == 0) {
    sSet = *reinterpret_cast<volatile unsigned long long*>(&ra.epoch->sets);
    sOk = 1;
  }

  // the tile at hand
  long long e0 = 0;
  int nLive = 0;
  auto set_tile = [&](int k) {
    e0 = ((long long)blockIdx.x + (long long)k * gridDim.x) * EPG;
    nLive = (a.nEl - e0) < EPG ? (int)(a.nEl - e0) : EPG;
    return nLive > 0;
  };

  // node role: node n of element ee
  const int ee = t / PP, n = t - ee * PP, i = n % P, j = n / P;
  const bool nodeOn = t < EPG * PP;
  bool active = false;
  R* gBase = sm;
  R* gU = gBase + ee * EB;
  R* gF1 = gU + NV * PP;
  R* gfb = gU + T::kU;
  R* gD = T::kDiv ? gBase + EPG * EB + ee * NV * PP : gU;
  R* gN = sm + X::oFields + ee * X::FB;
  double q[NV], G[NV], na[3] = {0.0, 0.0, 0.0}, Jij = 1.0, gdtE = 0.0;
  R m11 = (R)0, m21 = (R)0, m12 = (R)0, m22 = (R)0;
  auto load_state = [&]() {  // solution and register from global memory
    if (!active) return;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const size_t gi = n + (size_t)PP * (v + NV * (size_t)(e0 + ee));
      q[v] = a.q[gi];
      G[v] = sizeof(R) == 4 ? (double)a.Gf[gi] : a.G[gi];
    }
  };
  auto load_node = [&]() {  // metric terms, model fields, time step
    if (!active) return;
    const long long e = e0 + ee;
    const unsigned char* rec = reinterpret_cast<const unsigned char*>(a.geo) + (size_t)e * rBytes;
    node_aux_global<Phys>(a, n, e, PP, na);
    if constexpr (kWm == 4) {
      const float2* gp = reinterpret_cast<const float2*>(rec);
      const float2 c1 = gp[n], c2 = gp[PP + n];
      m11 = c1.x, m21 = c1.y, m12 = c2.x, m22 = c2.y;
    } else {
      const double2* gp = reinterpret_cast<const double2*>(rec);
      const double2 c1 = gp[n], c2 = gp[PP + n];
      m11 = (R)c1.x, m21 = (R)c1.y, m12 = (R)c2.x, m22 = (R)c2.y;
      if constexpr (kGeo == GEO_NOJ) Jij = 1.0 / (c1.x * c2.y - c2.x * c1.y);
    }
    if constexpr (kGeo != GEO_NOJ) Jij = reinterpret_cast<const double*>(rec + rJ)[n];
    if (a.dtElem) gdtE = a.dtElem[e];
  };

  // face role: node ii of side s1 of element eC
  const int faceWarp = 0;
  const int c0 = TPE - EPG * 4 * P;
  const int cf = (EPG == 1) ? (t & 31) : t - c0;
  const bool faceRole = (EPG == 1) ? ((t >> 5) == faceWarp && (t & 31) < 4 * P) : (t >= c0);
  const int eC = cf / (4 * P);
  bool faceOn = false;
  const int cc = cf - eC * 4 * P;
  const int s1 = cc / P, ii = cc % P;
  long long eF = 0;
  int bcid = 0;
  bool physical = false;
  long long nbBlk = -1;  // the neighbour's (element, side) block
  int i2 = 0;
  double2 nh = make_double2(0.0, 0.0);
  double ns = 0.0;
  typename Phys::template FaceK<R> faceK{};
  R velL[2] = {(R)0, (R)0}, velR[2] = {(R)0, (R)0};
  auto load_face = [&]() {
    eF = e0 + eC;
    if (!faceOn) return;
    const unsigned char* rec = reinterpret_cast<const unsigned char*>(a.geo) + (size_t)eF * rBytes;
    const int* si = reinterpret_cast<const int*>(rec + rSi) + 5 * s1;
    bcid = si[4];
    physical = (bcid != 0) && (si[2] == 0);
    nbBlk = bcid == 0 ? si[3] / 10 - 1 + 4 * (long long)(si[2] - 1) : -1;
    i2 = (si[3] % 10) ? N - ii : ii;
    if constexpr (kWm == 4) {
      const float2 f2 = reinterpret_cast<const float2*>(rec + rNhat)[ii + P * s1];
      nh = make_double2(f2.x, f2.y);
      ns = reinterpret_cast<const float*>(rec + rNs)[ii + P * s1];
    } else {
      nh = reinterpret_cast<const double2*>(rec + rNhat)[ii + P * s1];
      ns = reinterpret_cast<const double*>(rec + rNs)[ii + P * s1];
    }
    if constexpr (kLSW) {
      const double hb = a.fld[1][ii + (size_t)P * (s1 + 4 * eF)];
      faceK = Phys::template face_constants<R>(&hb, a);
    }
  };
  auto load_velocity = [&]() {  // the lagged velocity traces from their cache
    if constexpr (kSW)
      if (faceOn && !ra.fresh) {
        const R* vi = reinterpret_cast<const R*>(ra.velIn);
        velL[0] = vi[ii + P * (0 + 2 * (s1 + 4 * eF))];
        velL[1] = vi[ii + P * (1 + 2 * (s1 + 4 * eF))];
        if (nbBlk >= 0) {
          velR[0] = vi[i2 + P * (0 + 2 * nbBlk)];
          velR[1] = vi[i2 + P * (1 + 2 * nbBlk)];
        }
      }
  };
  // a tile's state in shared memory (kMany)
  auto tile_q = [&](int k) { return reinterpret_cast<double*>(state + (size_t)k * X::tileBytes) + t; };
  auto tile_G = [&](int k) {
    return reinterpret_cast<R*>(state + (size_t)k * X::tileBytes + X::nodes * NV * 8) + t;
  };
  auto tile_vel = [&](int k) {
    return reinterpret_cast<R*>(state + (size_t)k * X::tileBytes + X::nodes * NV * (8 + sizeof(R))) + cf;
  };

  // node fields of the solution q -> shared memory (first: of a solution set
  // from outside, rounded as k_traces does)
  auto put_fields = [&](bool first) {
    R f[NT];
#pragma unroll
    for (int v = 0; v < NV; ++v) f[v] = (R)q[v];
    if constexpr (NV == 4 && sizeof(R) == 4) {
      if (first) cig_fields_rounded(f, (float)a.gamma);
      else T::trace_fields(f, a);
    } else {
      T::trace_fields(f, a);
    }
#pragma unroll
    for (int v = 0; v < NT; ++v) gN[v * FS + T::nf(v, i, j)] = f[v];
  };
  // traces of the node fields: published as `set` (and, one tile per CTA, kept
  // for the tile's own faces), or (last) written to the trace cache
  auto put_traces = [&](unsigned long long set, bool last) {
    Pub* out = reinterpret_cast<Pub*>(ra.xch[set & 1]);
    const bool stall = a.debugStarve == 2 && blockIdx.x == 0;  // (test hook: CTA 0 publishes nothing)
    tile_traces<P, Phys, R, kWarpTraces>(sm + X::oFields, X::FB, EPG, nLive, t, TPE, a,
                                         [&](int eE, int fi, int l, bool row, R lo, R hi) {
      const int sl = row ? 3 : 0, sh = row ? 1 : 2;
      if (last) {
        R* o = reinterpret_cast<R*>(ra.trOut) + (size_t)4 * TS * (e0 + eE);
        o[l + P * fi + TS * sl] = lo;
        o[l + P * fi + TS * sh] = hi;
        return;
      }
      Pub* o = out + (size_t)4 * NT * P * (e0 + eE) + l + P * fi;
      if (!stall) {
        publish(o + NT * P * sl, lo, set);
        publish(o + NT * P * sh, hi, set);
      }
      if constexpr (!kMany) {
        R* own = sm + X::oOwn + eE * X::OB + l + P * fi;
        own[NT * P * sl] = lo;
        own[NT * P * sh] = hi;
      }
    });
  };

  const int tiles = kMany ? ra.tiles : 1;
  __syncthreads();  // the operator matrix and the set number
  const unsigned long long set0 = sSet + 1;  // the first stage's traces are set0, stage s's are set0 + s
  for (int k = 0; k < tiles; ++k) {
    if (!set_tile(k)) break;
    active = nodeOn && ee < nLive;
    faceOn = faceRole && eC < nLive;
    load_state();
    if constexpr (!kMany) load_node();
    if (!kMany || kSW) load_face();
    load_velocity();
    if constexpr (kMany) {
      if (active)
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          tile_q(k)[v * X::nodes] = q[v];
          tile_G(k)[v * X::nodes] = (R)G[v];
        }
      if constexpr (kSW)
        if (faceOn) {
          R* sv = tile_vel(k);
          sv[0] = velL[0], sv[X::faces] = velL[1], sv[2 * X::faces] = velR[0], sv[3 * X::faces] = velR[1];
          velR[0] = velR[1] = (R)0;  // (a wall's stay zero)
        }
    }
    if (ra.fresh) {
      if (active) put_fields(true);
      __syncthreads();
      put_traces(set0, false);
      if constexpr (kMany) __syncthreads();  // the fields are rewritten by the next tile
    }
  }

  for (int s = 0; s < ra.nStages && sOk; ++s) {
    const bool last = s + 1 == ra.nStages;
    const int m3 = s % 3;
    const double rkA = m3 == 0 ? ra.rkA[0] : (m3 == 1 ? ra.rkA[1] : ra.rkA[2]);
    const double rkG = m3 == 0 ? ra.rkG[0] : (m3 == 1 ? ra.rkG[1] : ra.rkG[2]);
    const double rkGdt = rkG * ra.dt;
    const bool cached = s == 0 && !ra.fresh;  // this stage's traces are in the caches
    for (int k = 0; k < tiles; ++k) {
      if constexpr (kMany) {
        if (!set_tile(k)) break;
        active = nodeOn && ee < nLive;
        faceOn = faceRole && eC < nLive;
        load_node();
        load_face();
        if (active)
#pragma unroll
          for (int v = 0; v < NV; ++v) q[v] = tile_q(k)[v * X::nodes];
        if constexpr (kSW)
          if (faceOn) {
            const R* sv = tile_vel(k);
            velL[0] = sv[0], velL[1] = sv[X::faces], velR[0] = sv[2 * X::faces], velR[1] = sv[3 * X::faces];
          }
      }

      // contravariant flux of the node
      if (active) {
        R f[NF];
#pragma unroll
        for (int v = 0; v < NV; ++v) f[v] = (R)q[v];
        T::flux_fields(f, a);
        R Fx[NV], Fy[NV];
        Phys::template flux<R>(f, na, a, Fx, Fy);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          gU[v * PP + T::f0at(i, j)] = m11 * Fx[v] + m21 * Fy[v];
          gF1[v * PP + T::f1at(i, j)] = m12 * Fx[v] + m22 * Fy[v];
        }
      }
      __syncthreads();  // fluxes and own traces

      // volume sums, alongside the face threads' exchange and Riemann flux
      tile_volume_sums<P, Phys, R>(gBase, sdg, t, faceWarp, nLive, a);
      R dreg[NV];
      if constexpr (T::kRegDiv) {
        if (active) {
#pragma unroll
          for (int v = 0; v < NV; ++v) dreg[v] = (R)0;
#pragma unroll
          for (int m = 0; m < P; ++m) {
            const R gi = sdgR[T::dgat(m, i)], gj = sdgR[T::dgat(m, j)];
#pragma unroll
            for (int v = 0; v < NV; ++v)
              dreg[v] = dreg[v] + gi * gU[v * PP + T::f0at(m, j)] + gj * gF1[v * PP + T::f1at(i, m)];
          }
        }
      }
      // ShallowWater: the next stage's lagged velocities are those of this stage's
      // traces (and, after SetSolution, the first stage's too); walls keep velR =
      // 0.  With kAhead the side's own is formed before the neighbour's traces are
      // waited for and the neighbour's after the barrier: at P = 8 with one tile
      // per CTA a stage on 10x10 / 34x34 takes 1.59 / 2.09 us instead of 1.72 /
      // 2.28 in FP64, 2.39 / 3.50 instead of 2.68 / 3.89 with the reference's
      // roundings, 1.39 / 1.72 instead of 1.48 / 1.79 in FP32; with several tiles
      // 2-10 % slower, at P = 4 to 6 between 8 % faster and 7 % slower.
      constexpr bool kAhead = kSW && !kMany && P == 8;
      constexpr bool kDivide = ref_rounding<R>() || (T::kOdd && sizeof(R) == 4);  // as the stage launches
      auto velocity = [&](const R* tr, R v[2], bool divide) {
        if (divide) {
          v[0] = tr[0] / tr[2];
          v[1] = tr[1] / tr[2];
        } else {
          const R rH = (R)1 / tr[2];
          v[0] = tr[0] * rH;
          v[1] = tr[1] * rH;
        }
      };
      R L[NT], Xn[NT], nextL[2] = {(R)0, (R)0};
      if (faceOn) {
        if (cached) {
          const R* tr = reinterpret_cast<const R*>(ra.trIn);
#pragma unroll
          for (int f = 0; f < NT; ++f) {
            L[f] = tr[(size_t)TS * (s1 + 4 * eF) + ii + P * f];
            Xn[f] = nbBlk >= 0 ? tr[(size_t)TS * nbBlk + i2 + P * f] : (R)0;
          }
        } else {
          const unsigned long long set = set0 + s;
          const Pub* pub = reinterpret_cast<const Pub*>(ra.xch[set & 1]);
          if constexpr (kMany) {  // the CTA's own, published a stage ago
            const Pub* own = pub + (size_t)NT * P * (s1 + 4 * eF) + ii;
#pragma unroll
            for (int f = 0; f < NT; ++f) peek(own + P * f, set, L[f]);
          } else {
            const R* own = sm + X::oOwn + eC * X::OB + NT * P * s1 + ii;
#pragma unroll
            for (int f = 0; f < NT; ++f) L[f] = own[P * f];
          }
          if constexpr (kAhead) velocity(L, nextL, kDivide);
#pragma unroll
          for (int f = 0; f < NT; ++f) Xn[f] = (R)0;
          if (nbBlk >= 0) {
            const Pub* nb = pub + (size_t)NT * P * nbBlk + i2;
            const long long c = clock64();
            while (true) {
              bool ok = true;
#pragma unroll
              for (int f = 0; f < NT; ++f) ok &= peek(nb + P * f, set, Xn[f]);
              if (ok) break;
              if (clock64() - c > a.waitCycles) {
                sOk = 0;
                break;
              }
            }
          }
        }
        double fx[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        if constexpr (!kLSW)
          if (physical) face_aux_global<Phys>(a, s1, ii, eF, P, fx);
        R vL[2] = {velL[0], velL[1]}, vR[2] = {velR[0], velR[1]};  // this stage's lagged velocities
        if constexpr (kSW) {
          if (cached || !kAhead) velocity(L, nextL, kDivide);
          if constexpr (!kAhead) {
            velL[0] = nextL[0], velL[1] = nextL[1];
            if (nbBlk >= 0) velocity(Xn, velR, kDivide);
          }
          if constexpr (kMany) {
            R* sv = tile_vel(k);
            sv[0] = velL[0], sv[X::faces] = velL[1], sv[2 * X::faces] = velR[0], sv[3 * X::faces] = velR[1];
          }
          if (s == 0 && ra.fresh) {
            velocity(L, vL, true);
            if (nbBlk >= 0) velocity(Xn, vR, true);
          }
          if (last) {
            R* vo = reinterpret_cast<R*>(ra.velOut);
            vo[ii + P * (0 + 2 * (s1 + 4 * eF))] = nextL[0];
            vo[ii + P * (1 + 2 * (s1 + 4 * eF))] = nextL[1];
          }
        }
        R out[NV];
        Phys::template face<R>(bcid, physical, L, Xn, vL, vR, nh.x, nh.y, ns, fx, faceK, a, out);
#pragma unroll
        for (int v = 0; v < NV; ++v) (gBase + eC * EB + T::kU)[s1 * SS + v * P + ii] = out[v];
      }
      __syncthreads();  // volume sums and face fluxes
      if (!sOk) break;

      if constexpr (kAhead)
        if (faceOn) {
          velL[0] = nextL[0], velL[1] = nextL[1];
          if (nbBlk >= 0) velocity(Xn, velR, kDivide);
        }
      if (active) {
        double Src[NV];
        Phys::template source<double>(q, na, a, Src);
        R d[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) d[v] = T::kRegDiv ? dreg[v] : T::kLines ? gU[v * PP + n] + gF1[v * PP + T::f1at(i, j)] : gD[v * PP + n];
        const double gdt = a.dtElem ? rkG * gdtE : rkGdt;
        const R bi0 = sb[i], bi1 = sb[i + P], bj0 = sb[j], bj1 = sb[j + P], wi = sw[i], wj = sw[j];
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          double dsdt;
          if constexpr (ref_rounding<R>()) {
            const R dv = d[v] + (bi1 * gfb[1 * SS + v * P + j] + bi0 * gfb[3 * SS + v * P + j]) / wi +
                         (bj1 * gfb[2 * SS + v * P + i] + bj0 * gfb[0 * SS + v * P + i]) / wj;
            dsdt = Src[v] - (double)dv / Jij;
          } else {
            const R dv = d[v] + (bi1 * gfb[1 * SS + v * P + j] + bi0 * gfb[3 * SS + v * P + j]) * wi +
                         (bj1 * gfb[2 * SS + v * P + i] + bj0 * gfb[0 * SS + v * P + i]) * wj;
            dsdt = fma(-(double)dv, Jij, Src[v]);
          }
          if constexpr (kMany) G[v] = (double)tile_G(k)[v * X::nodes];
          const double Gn = rkA * G[v] + dsdt;
          q[v] = q[v] + gdt * Gn;
          if constexpr (kMany) {
            tile_G(k)[v * X::nodes] = (R)Gn;
            tile_q(k)[v * X::nodes] = q[v];
          } else {
            G[v] = sizeof(R) == 4 ? (double)(float)Gn : Gn;  // the FP32-bulk register is FP32
          }
        }
        put_fields(false);
      }
      __syncthreads();  // node fields
      put_traces(set0 + s + 1, last);
    }
  }

  if (sOk) {
    for (int k = 0; k < tiles; ++k) {
      if (!set_tile(k)) break;
      if (!nodeOn || ee >= nLive) continue;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const size_t gi = n + (size_t)PP * (v + NV * (size_t)(e0 + ee));
        a.q[gi] = kMany ? tile_q(k)[v * X::nodes] : q[v];
        if constexpr (sizeof(R) == 4) a.Gf[gi] = kMany ? (float)tile_G(k)[v * X::nodes] : (float)G[v];
        else a.G[gi] = kMany ? (double)tile_G(k)[v * X::nodes] : G[v];
      }
    }
  } else if (t == 0 && a.err) {
    atomicExch(a.err, 1);
  }
  // The last CTA to finish moves the set counter on (every CTA has read it).
  if (t == 0 && atomicAdd(&ra.epoch->done, 1u) == gridDim.x - 1) {
    ra.epoch->done = 0;
    ra.epoch->sets = set0 + ra.nStages + 1;
  }
}

}  // namespace selfgpu
