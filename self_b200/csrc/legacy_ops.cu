// Drop-in replacements for SELF's per-operator HIP wrappers (FP64).
//
// Same symbol names and arguments as the reference (see include/selfgpu.h for
// the file:line each replaces); each wrapper dereferences the real** it gets,
// launches on the legacy default stream and returns without synchronising, as
// the reference does.  Unlike the reference kernels (one block per
// (var, element), one thread per node, strided uncoalesced traces), the
// pointwise ones are grid-stride kernels over contiguous outputs, so that every
// warp reads and writes consecutive addresses, and for degrees 1-7 the
// interpolation and derivative operators take whole planes or elements per
// block, each input read once from memory; the arithmetic of each output
// follows the CPU branch of the reference term by term.  The whole-stage
// kernels (fused_stage_tma.cuh, fused_resident.cuh) are the fast path; these
// exist so an unmodified SELF caller can use the library operator by operator.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <type_traits>

#include "physics.cuh"
#include "selfgpu_internal.h"

namespace selfgpu {
namespace {

constexpr int kThreads = 256;

inline int blocks_for(long long n) {
  long long b = (n + kThreads - 1) / kThreads;
  if (b < 1) b = 1;
  if (b > 148LL * 64) b = 148LL * 64;  // grid-stride beyond 64 CTAs per SM
  return (int)b;
}

inline void check_launch(const char* name) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) set_error(SELFGPU_ERR_CUDA, std::string(name) + ": " + cudaGetErrorString(e));
}

// Every kernel here is launched as a programmatic dependent of the previous one
// on the stream (a right-hand side is some twenty short kernels): its launch
// and its first blocks' start overlap that kernel's last wave.  The first thing
// each does is to let its own successor start and to wait for the previous
// kernel's completion, before it touches any data.  (64x64 elements, N = 7, the
// operators of one right-hand side: 152 us without, 113 with.)  No pointer is
// __restrict__: the previous kernel may write what this one reads while this
// one is already running, and the qualifier would let the compiler read it
// through the non-coherent path or ahead of the wait.
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

#define GRID_STRIDE(k, n) for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < (n); \
                               k += (long long)gridDim.x * blockDim.x)

// The kernels below take the number of nodes per direction as a template
// argument PC (2..8; 0 = any other, read at run time): index arithmetic by a
// run-time P in 64 bits took more instructions than the operators themselves.
// P-independent totals stay 64-bit.
template <int PC>
__device__ __forceinline__ int nodes(int N) {
  return PC ? PC : N + 1;
}
// quotient and remainder of a 64-bit index by a small divisor, in 32 bits
// where the index fits
__device__ __forceinline__ long long divide(long long k, int d, int& rem) {
  if (k < (1LL << 32)) {
    const unsigned q = (unsigned)k / (unsigned)d;
    rem = (int)((unsigned)k - q * (unsigned)d);
    return q;
  }
  const long long q = k / d;
  rem = (int)(k - q * d);
  return q;
}

// Run-time degrees (N > 7) and target grids too large for a block's shared
// memory: one thread per output, operands from global memory.
// src/SELF_Lagrange.f90:741-789; iM(ii,m) at iM[ii + P*m]
__global__ void k_scalar_grid_interp(const double* iM, const double* f,
                                     double* fo, int N, int M, long long n) {
  after_previous();
  const int P = N + 1, Q = M + 1;
  GRID_STRIDE(k, n) {
    const int i = k % Q, j = (k / Q) % Q;
    const long long ve = k / ((long long)Q * Q);
    const double* fe = f + ve * P * P;
    double fij = 0.0;
    for (int jj = 0; jj < P; ++jj) {
      double fi = 0.0;
      for (int ii = 0; ii < P; ++ii) fi = fi + fe[ii + P * jj] * iM[ii + P * i];
      fij = fij + fi * iM[jj + P * j];
    }
    fo[k] = fij;
  }
}

// src/SELF_Lagrange.f90:824-875
__global__ void k_vector_grid_interp(const double* iM, const double* f,
                                     double* fo, int N, int M, long long n) {
  after_previous();
  const int P = N + 1, Q = M + 1;
  GRID_STRIDE(k, n) {  // k enumerates (dir, i, j, var*el)
    const int d = k & 1;
    const long long kn = k >> 1;
    const int i = kn % Q, j = (kn / Q) % Q;
    const long long ve = kn / ((long long)Q * Q);
    const double* fe = f + ve * 2 * P * P;
    double o = 0.0;
    for (int jj = 0; jj < P; ++jj) {
      double fi = 0.0;
      for (int ii = 0; ii < P; ++ii) fi = fi + fe[d + 2 * (ii + P * jj)] * iM[ii + P * i];
      o = o + fi * iM[jj + P * j];
    }
    fo[k] = o;
  }
}

// src/SELF_Lagrange.f90:2241-2270; one thread per (i, var, el) writes 4 sides
__global__ void k_scalar_boundary_interp(const double* bM, const double* f,
                                         double* fb, int N, int nVar, long long n) {
  after_previous();
  const int P = N + 1;
  GRID_STRIDE(k, n) {
    const int i = k % P;
    const long long ve = k / P;
    const int v = ve % nVar;
    const long long e = ve / nVar;
    const double* fe = f + ve * P * P;
    double b1 = 0, b2 = 0, b3 = 0, b4 = 0;
    for (int ii = 0; ii < P; ++ii) {
      b1 = b1 + bM[ii] * fe[i + P * ii];
      b2 = b2 + bM[ii + P] * fe[ii + P * i];
      b3 = b3 + bM[ii + P] * fe[i + P * ii];
      b4 = b4 + bM[ii] * fe[ii + P * i];
    }
    double* o = fb + i + (long long)P * (v + (long long)nVar * 4 * e);
    const long long ss = (long long)P * nVar;
    o[0] = b1;
    o[ss] = b2;
    o[2 * ss] = b3;
    o[3 * ss] = b4;
  }
}

// src/SELF_Lagrange.f90:2284-2316 (C = 2) and 2330-2366 (C = 4): components fastest
template <int C>
__global__ void k_multi_boundary_interp(const double* bM, const double* f,
                                        double* fb, int N, int nVar, long long n) {
  after_previous();
  const int P = N + 1;
  GRID_STRIDE(k, n) {  // k enumerates (comp, i, var, el)
    const int c = k % C;
    const int i = (k / C) % P;
    const long long ve = k / ((long long)C * P);
    const int v = ve % nVar;
    const long long e = ve / nVar;
    const double* fe = f + ve * C * P * P;
    double b1 = 0, b2 = 0, b3 = 0, b4 = 0;
    for (int ii = 0; ii < P; ++ii) {
      b1 = b1 + bM[ii] * fe[c + C * (i + P * ii)];
      b2 = b2 + bM[ii + P] * fe[c + C * (ii + P * i)];
      b3 = b3 + bM[ii + P] * fe[c + C * (i + P * ii)];
      b4 = b4 + bM[ii] * fe[c + C * (ii + P * i)];
    }
    double* o = fb + c + C * (i + (long long)P * (v + (long long)nVar * 4 * e));
    const long long ss = (long long)C * P * nVar;
    o[0] = b1;
    o[ss] = b2;
    o[2 * ss] = b3;
    o[3 * ss] = b4;
  }
}

// src/SELF_Lagrange.f90:1424-1463
__global__ void k_vector_gradient_any(const double* dM, const double* f,
                                      double* gf, int N, long long n) {
  after_previous();
  const int P = N + 1;
  GRID_STRIDE(k, n) {  // k enumerates (i, j, var*el)
    const int i = k % P, j = (k / P) % P;
    const long long ve = k / ((long long)P * P);
    const double* fe = f + ve * 2 * P * P;
    double g11 = 0, g21 = 0, g12 = 0, g22 = 0;
    for (int ii = 0; ii < P; ++ii) {
      g11 = g11 + dM[ii + P * i] * fe[0 + 2 * (ii + P * j)];
      g21 = g21 + dM[ii + P * i] * fe[1 + 2 * (ii + P * j)];
      g12 = g12 + dM[ii + P * j] * fe[0 + 2 * (i + P * ii)];
      g22 = g22 + dM[ii + P * j] * fe[1 + 2 * (i + P * ii)];
    }
    double* o = gf + 4 * k;
    o[0] = g11;
    o[1] = g21;
    o[2] = g12;
    o[3] = g22;
  }
}

// src/SELF_Lagrange.f90:1589-1625
__global__ void k_vector_dg_divergence_any(const double* dgM, const double* bM,
                                       const double* qw, const double* f,
                                       const double* bf, double* df, int N, int nVar,
                                       long long n) {
  after_previous();
  const int P = N + 1;
  GRID_STRIDE(k, n) {
    const int i = k % P, j = (k / P) % P;
    const long long ve = k / ((long long)P * P);
    const int v = ve % nVar;
    const long long e = ve / nVar;
    const double* fe = f + ve * 2 * P * P;
    double d = 0.0;
    for (int ii = 0; ii < P; ++ii)
      d = d + dgM[ii + P * i] * fe[0 + 2 * (ii + P * j)] + dgM[ii + P * j] * fe[1 + 2 * (i + P * ii)];
    const double* b = bf + (long long)P * (v + (long long)nVar * 4 * e);
    const long long ss = (long long)P * nVar;
    d = d + (bM[i + P] * b[j + ss] + bM[i] * b[j + 3 * ss]) / qw[i] +
        (bM[j + P] * b[i + 2 * ss] + bM[j] * b[i]) / qw[j];
    df[k] = d;
  }
}

// Stencil operators work on planes (one variable of one element, C components
// of P x P nodes, contiguous).  A block takes `planes` consecutive ones: their
// values go to shared memory with coalesced loads, once, and the row and column
// sums read them there.  Rows are padded to an odd stride.
__host__ __device__ constexpr int row_stride(int P) { return P | 1; }

// ------------------------------------------------------------------ Lagrange
// src/SELF_Lagrange.f90:741-789 (C = 1) and 824-875 (C = 2); iM(ii,m) at
// iM[ii + P*m].  The xi sums of a row are formed once for all eta targets (the
// reference's order per value).
template <int P, int C>
__global__ void __launch_bounds__(kThreads) k_grid_interp(const double* iM,
                                                          const double* f, double* fo, int M,
                                                          int planes, long long nPlanes) {
  after_previous();
  extern __shared__ double sm[];
  const int Q = M + 1;
  // quotients of indices below 2^16 by C Q and Q (Q >= 2): multiply-high by the rounded-up reciprocal
  const unsigned rCQ = 0xffffffffu / (unsigned)(C * Q) + 1u, rQ = 0xffffffffu / (unsigned)Q + 1u;
  double* sM = sm;                 // iM (P x Q)
  double* sf = sM + P * Q;         // planes x C x P x P
  double* sg = sf + planes * C * P * P;  // planes x C x P (jj) x Q (i): xi sums
  for (int k = threadIdx.x; k < P * Q; k += kThreads) sM[k] = iM[k];
  for (long long p0 = (long long)blockIdx.x * planes; p0 < nPlanes; p0 += (long long)gridDim.x * planes) {
    const int live = (int)(nPlanes - p0 < planes ? nPlanes - p0 : planes);
    __syncthreads();
    for (int k = threadIdx.x; k < live * C * P * P; k += kThreads) sf[k] = f[p0 * C * P * P + k];
    __syncthreads();
    for (int k = threadIdx.x; k < live * C * P * Q; k += kThreads) {  // (c, i, r = jj + P plane)
      const int r = __umulhi(k, rCQ), ci = k - r * C * Q, c = ci % C, i = ci / C;
      const double *row = sf + C * P * r + c, *m = sM + P * i;
      double fi = 0.0;
#pragma unroll
      for (int ii = 0; ii < P; ++ii) fi = fi + row[C * ii] * m[ii];
      sg[k] = fi;
    }
    __syncthreads();
    double* o = fo + p0 * C * Q * Q;
    for (int k = threadIdx.x; k < live * C * Q * Q; k += kThreads) {  // (c, i, r = j + Q plane)
      const int r = __umulhi(k, rCQ), ci = k - r * C * Q, pl = __umulhi(r, rQ), j = r - pl * Q;
      const double *g = sg + C * Q * P * pl + ci, *m = sM + P * j;
      double fij = 0.0;
#pragma unroll
      for (int jj = 0; jj < P; ++jj) fij = fij + g[C * Q * jj] * m[jj];
      o[k] = fij;
    }
  }
}

// src/SELF_Lagrange.f90:2241-2270 (C = 1), 2284-2316 (C = 2) and 2330-2366
// (C = 4): components fastest; one task per (component, node, side, plane)
template <int P, int C>
__global__ void __launch_bounds__(kThreads) k_boundary_interp(const double* bM,
                                                              const double* f, double* fb,
                                                              int nVar, int planes, long long nPlanes) {
  after_previous();
  extern __shared__ double sm[];
  constexpr int RS = row_stride(P);
  double* sb = sm;           // bMatrix
  double* sf = sm + 2 * P;   // planes x P rows of RS nodes x C
  for (int k = threadIdx.x; k < 2 * P; k += kThreads) sb[k] = bM[k];
  for (long long p0 = (long long)blockIdx.x * planes; p0 < nPlanes; p0 += (long long)gridDim.x * planes) {
    const int live = (int)(nPlanes - p0 < planes ? nPlanes - p0 : planes);
    __syncthreads();
    for (int k = threadIdx.x; k < live * C * P * P; k += kThreads) {
      const int r = k / (C * P);
      sf[k - r * C * P + r * C * RS] = f[p0 * C * P * P + k];
    }
    __syncthreads();
    for (int k = threadIdx.x; k < live * 4 * C * P; k += kThreads) {
      const int ci = k % (C * P), s = (k / (C * P)) % 4, pl = k / (4 * C * P);
      const int c = ci % C, i = ci / C;
      int v;
      const long long e = divide(p0 + pl, nVar, v);
      // south and north sum along eta at fixed i, east and west along xi
      const bool eta = (s == 0 || s == 2);
      const double* x = sf + C * RS * P * pl + c + (eta ? C * i : C * RS * i);
      const int step = eta ? C * RS : C;
      const double* b = sb + ((s == 1 || s == 2) ? P : 0);
      double acc = 0.0;
#pragma unroll
      for (int ii = 0; ii < P; ++ii) acc = acc + b[ii] * x[step * ii];
      fb[ci + (long long)C * P * (v + (long long)nVar * (s + 4 * e))] = acc;
    }
  }
}

// The derivative kernels give each thread one node of a plane slot, the same
// for every plane it takes, so the node's matrix columns and lift weights stay
// in registers over a block's sweep; the planes' values pass through shared
// memory, the next ones loaded while the present ones are summed.  (Reading
// the matrix from shared memory for every product, with a block per few
// planes, held the divergence at its shared-memory rate: 22 us for 16 384
// planes at P = 8, cold.)
template <int P>
struct NodeBlock {
  static constexpr int PP = P * P, RS = row_stride(P), FS = RS * P;
  static constexpr int slots = kThreads / PP > 0 ? kThreads / PP : 1, threads = slots * PP;
};

// column i of a P x P matrix at m[ii + P i]
template <int P>
__device__ __forceinline__ void load_column(const double* m, int i, double c[P]) {
#pragma unroll
  for (int ii = 0; ii < P; ++ii) c[ii] = m[ii + P * i];
}

// src/SELF_Lagrange.f90:1424-1463
template <int P>
__global__ void __launch_bounds__(NodeBlock<P>::threads, 3) k_vector_gradient(const double* dM,
                                                                           const double* f,
                                                                           double* gf,
                                                                           long long nPlanes) {
  after_previous();
  using B = NodeBlock<P>;
  constexpr int PP = B::PP, RS = B::RS, FS = B::FS;
  __shared__ double sf[B::slots][2][FS];
  const int slot = threadIdx.x / PP, n = threadIdx.x - slot * PP, j = n / P, i = n - j * P;
  double di[P], dj[P];
  load_column<P>(dM, i, di);
  load_column<P>(dM, j, dj);
  const long long step = (long long)gridDim.x * B::slots;
  long long p = (long long)blockIdx.x * B::slots + slot;
  double x = 0.0, y = 0.0;
  auto load = [&](long long k) {
    if (k < nPlanes) {
      x = f[2 * (k * PP + n)];
      y = f[2 * (k * PP + n) + 1];
    }
  };
  load(p);
  for (; p - slot < nPlanes; p += step) {
    __syncthreads();
    sf[slot][0][RS * j + i] = x;
    sf[slot][1][RS * j + i] = y;
    __syncthreads();
    load(p + step);
    if (p >= nPlanes) continue;
    const double *f0 = sf[slot][0], *f1 = sf[slot][1];
    double g11 = 0, g21 = 0, g12 = 0, g22 = 0;
#pragma unroll
    for (int ii = 0; ii < P; ++ii) {
      g11 = g11 + di[ii] * f0[ii + RS * j];
      g21 = g21 + di[ii] * f1[ii + RS * j];
      g12 = g12 + dj[ii] * f0[i + RS * ii];
      g22 = g22 + dj[ii] * f1[i + RS * ii];
    }
    double* o = gf + 4 * (p * PP + n);
    o[0] = g11;
    o[1] = g21;
    o[2] = g12;
    o[3] = g22;
  }
}

// src/SELF_Lagrange.f90:1589-1625
template <int P>
__global__ void __launch_bounds__(NodeBlock<P>::threads, 3) k_vector_dg_divergence(
    const double* dgM, const double* bM, const double* qw,
    const double* f, const double* bf, double* df, int nVar,
    long long nPlanes) {
  after_previous();
  using B = NodeBlock<P>;
  constexpr int PP = B::PP, RS = B::RS, FS = B::FS;
  __shared__ double sf[B::slots][2][FS];
  const int slot = threadIdx.x / PP, n = threadIdx.x - slot * PP, j = n / P, i = n - j * P;
  double di[P], dj[P];
  load_column<P>(dgM, i, di);
  load_column<P>(dgM, j, dj);
  const double bi0 = bM[i], bi1 = bM[i + P], bj0 = bM[j], bj1 = bM[j + P], wi = qw[i], wj = qw[j];
  const long long step = (long long)gridDim.x * B::slots, ss = (long long)P * nVar;
  long long p = (long long)blockIdx.x * B::slots + slot;
  double x = 0.0, y = 0.0, bS = 0.0, bE = 0.0, bN = 0.0, bW = 0.0;
  auto load = [&](long long k) {
    if (k < nPlanes) {
      x = f[2 * (k * PP + n)];
      y = f[2 * (k * PP + n) + 1];
      int v;
      const long long e = divide(k, nVar, v);
      const double* b = bf + (long long)P * (v + (long long)nVar * 4 * e);
      bS = b[i], bE = b[j + ss], bN = b[i + 2 * ss], bW = b[j + 3 * ss];
    }
  };
  load(p);
  for (; p - slot < nPlanes; p += step) {
    __syncthreads();
    sf[slot][0][RS * j + i] = x;
    sf[slot][1][RS * j + i] = y;
    const double cS = bS, cE = bE, cN = bN, cW = bW;
    __syncthreads();
    load(p + step);
    if (p >= nPlanes) continue;
    const double *f0 = sf[slot][0], *f1 = sf[slot][1];
    double d = 0.0;
#pragma unroll
    for (int ii = 0; ii < P; ++ii) d = d + di[ii] * f0[ii + RS * j] + dj[ii] * f1[i + RS * ii];
    d = d + (bi1 * cE + bi0 * cW) / wi + (bj1 * cN + bj0 * cS) / wj;
    df[p * PP + n] = d;
  }
}

// src/SELF_Data.f90:1570-1607
__global__ void k_determinant(const double* t, double* det, long long n) {
  after_previous();
  GRID_STRIDE(k, n) {
    const double* a = t + 4 * k;
    det[k] = a[0] * a[3] - a[2] * a[1];
  }
}

// src/SELF_Geometry.f90:448-457 (dsdx(:,1) = (dy/ds2, -dx/ds2), dsdx(:,2) = (-dy/ds1, dx/ds1))
__global__ void k_contravariant_basis(const double* dxds, double* dsdx, long long n) {
  after_previous();
  GRID_STRIDE(k, n) {
    const double* a = dxds + 4 * k;
    double* o = dsdx + 4 * k;
    o[0] = a[3];
    o[1] = -a[2];
    o[2] = -a[1];
    o[3] = a[0];
  }
}

// Sign adjustment of dsdx on the faces: outward on East/North for J > 0,
// src/SELF_Geometry.f90:462-520 (fac), applied to all four components.
__global__ void k_adjust_boundary_basis(double* dsdxB, const double* JB, int N,
                                        long long n) {
  after_previous();
  const int P = N + 1;
  GRID_STRIDE(k, n) {  // k enumerates (i, side, el) of the scalar face layout
    const int s = (k / P) % 4;
    const double j = JB[k];
    const double fac = (s == 1 || s == 2) ? copysign(1.0, j) : -copysign(1.0, j);
    double* o = dsdxB + 4 * k;
    for (int q = 0; q < 4; ++q) o[q] = o[q] * fac;
  }
}

// nHat and nScale from the (unsigned) face contravariant basis, then the sign
// adjustment, as CalculateContravariantBasis_SEMQuad does on the host
// (src/SELF_Geometry.f90:458-522).
__global__ void k_face_normals(double* dsdxB, const double* JB, double* nHat,
                               double* nScale, int N, long long n) {
  after_previous();
  const int P = N + 1;
  GRID_STRIDE(k, n) {
    const int s = (k / P) % 4;
    const double j = JB[k];
    const double fac = (s == 1 || s == 2) ? copysign(1.0, j) : -copysign(1.0, j);
    double* t = dsdxB + 4 * k;
    const int col = (s == 0 || s == 2) ? 1 : 0;
    const double a0 = t[2 * col], a1 = t[2 * col + 1];
    const double mag = sqrt(a0 * a0 + a1 * a1);
    nScale[k] = mag;
    nHat[2 * k] = fac * a0 / mag;
    nHat[2 * k + 1] = fac * a1 / mag;
    for (int q = 0; q < 4; ++q) t[q] = t[q] * fac;
  }
}

// ---------------------------------------------------------------- MappedData
// src/SELF_MappedData.f90:955-1078 (BR1 gradient, weak form), N > 7
__global__ void k_gradient_br(const double* f, const double* avgB,
                              const double* dsdx, const double* J,
                              const double* nHat, const double* nScale,
                              double* gradF, const double* dgM,
                              const double* bM, const double* qw, int N, int nVar,
                              long long n) {
  after_previous();
  const int P = N + 1;
  GRID_STRIDE(k, n) {
    const int i = k % P, j = (k / P) % P;
    const long long ve = k / ((long long)P * P);
    const int v = ve % nVar;
    const long long e = ve / nVar;
    const double* fe = f + ve * P * P;
    const double* ge = dsdx + e * 4 * P * P;
    double gx = 0.0, gy = 0.0;
    for (int ii = 0; ii < P; ++ii) {
      const double* a = ge + 4 * (ii + P * j);
      const double* b = ge + 4 * (i + P * ii);
      double f1 = fe[ii + P * j] * a[0];
      double f2 = fe[i + P * ii] * b[2];
      gx = gx + dgM[ii + P * i] * f1 + dgM[ii + P * j] * f2;
      f1 = fe[ii + P * j] * a[1];
      f2 = fe[i + P * ii] * b[3];
      gy = gy + dgM[ii + P * i] * f1 + dgM[ii + P * j] * f2;
    }
    const double* av = avgB + (long long)P * (v + (long long)nVar * 4 * e);
    const long long ss = (long long)P * nVar;
    const double* nh = nHat + 2 * P * 4 * e;
    const double* ns = nScale + P * 4 * e;
    auto NH = [&](int d, int q, int s) { return nh[d + 2 * (q + P * s)]; };
    auto NS = [&](int q, int s) { return ns[q + P * s]; };
    double f1 = av[j + ss] * NH(0, j, 1) * NS(j, 1);
    double f2 = av[j + 3 * ss] * NH(0, j, 3) * NS(j, 3);
    gx = gx + (f1 * bM[i + P] + f2 * bM[i]) / qw[i];
    f1 = av[i + 2 * ss] * NH(0, i, 2) * NS(i, 2);
    f2 = av[i] * NH(0, i, 0) * NS(i, 0);
    gx = gx + (f1 * bM[j + P] + f2 * bM[j]) / qw[j];
    f1 = av[j + ss] * NH(1, j, 1) * NS(j, 1);
    f2 = av[j + 3 * ss] * NH(1, j, 3) * NS(j, 3);
    gy = gy + (f1 * bM[i + P] + f2 * bM[i]) / qw[i];
    f1 = av[i + 2 * ss] * NH(1, i, 2) * NS(i, 2);
    f2 = av[i] * NH(1, i, 0) * NS(i, 0);
    gy = gy + (f1 * bM[j + P] + f2 * bM[j]) / qw[j];
    const double Jij = J[i + P * (j + P * e)];
    gradF[2 * k] = gx / Jij;
    gradF[2 * k + 1] = gy / Jij;
  }
}

// src/SELF_MappedData.f90:1080-1149 (strong form), N > 7
__global__ void k_gradient_sf(const double* f, const double* dsdx,
                              const double* J, double* gradF, const double* dM,
                              int N, int nVar, long long n) {
  after_previous();
  const int P = N + 1;
  GRID_STRIDE(k, n) {
    const int i = k % P, j = (k / P) % P;
    const long long ve = k / ((long long)P * P);
    const long long e = ve / nVar;
    const double* fe = f + ve * P * P;
    const double* ge = dsdx + e * 4 * P * P;
    double gx = 0.0, gy = 0.0;
    for (int ii = 0; ii < P; ++ii) {
      const double* a = ge + 4 * (ii + P * j);
      const double* b = ge + 4 * (i + P * ii);
      double f1 = fe[ii + P * j] * a[0];
      double f2 = fe[i + P * ii] * b[2];
      gx = gx + dM[ii + P * i] * f1 + dM[ii + P * j] * f2;
      f1 = fe[ii + P * j] * a[1];
      f2 = fe[i + P * ii] * b[3];
      gy = gy + dM[ii + P * i] * f1 + dM[ii + P * j] * f2;
    }
    const double Jij = J[i + P * (j + P * e)];
    gradF[2 * k] = gx / Jij;
    gradF[2 * k + 1] = gy / Jij;
  }
}

// src/SELF_MappedData.f90:955-1078 (kWeak: BR1 gradient, weak form, D = dgMatrix)
// and 1080-1149 (strong form, D = dMatrix).  A node's four products with the
// metric terms are formed once and shared by the sums of its row and column,
// a face node's products with the normal by the nodes of its line.
template <int P, bool kWeak>
__global__ void __launch_bounds__(NodeBlock<P>::threads, 3) k_gradient(
    const double* f, const double* avgB, const double* dsdx,
    const double* J, const double* nHat, const double* nScale,
    double* gradF, const double* D, const double* bM,
    const double* qw, int nVar, long long nPlanes) {
  after_previous();
  using B = NodeBlock<P>;
  constexpr int PP = B::PP, RS = B::RS, FS = B::FS;
  __shared__ double sf[B::slots][4][FS];
  __shared__ double sF[kWeak ? B::slots : 1][2][4 * P];  // face products, x and y
  const int slot = threadIdx.x / PP, n = threadIdx.x - slot * PP, j = n / P, i = n - j * P;
  double di[P], dj[P], bi0 = 0, bi1 = 0, bj0 = 0, bj1 = 0, wi = 1, wj = 1;
  load_column<P>(D, i, di);
  load_column<P>(D, j, dj);
  if (kWeak) bi0 = bM[i], bi1 = bM[i + P], bj0 = bM[j], bj1 = bM[j + P], wi = qw[i], wj = qw[j];
  const long long step = (long long)gridDim.x * B::slots, ss = (long long)P * nVar;
  long long p = (long long)blockIdx.x * B::slots + slot;
  double x = 0.0, g0 = 0.0, g1 = 0.0, g2 = 0.0, g3 = 0.0, nextJ = 1.0;
  auto load = [&](long long k) {
    if (k < nPlanes) {
      int v;
      const long long e = divide(k, nVar, v);
      const double* g = dsdx + 4 * (n + (long long)PP * e);
      x = f[k * PP + n];
      g0 = g[0], g1 = g[1], g2 = g[2], g3 = g[3];
      nextJ = J[n + (long long)PP * e];
    }
  };
  load(p);
  for (; p - slot < nPlanes; p += step) {
    __syncthreads();
    double* h = sf[slot][0] + RS * j + i;
    h[0] = x * g0;
    h[FS] = x * g1;
    h[2 * FS] = x * g2;
    h[3 * FS] = x * g3;
    const double Jij = nextJ;
    if (kWeak && p < nPlanes) {
      int v;
      const long long e = divide(p, nVar, v);
      const double* av = avgB + (long long)P * (v + (long long)nVar * 4 * e);
      for (int k = n; k < 4 * P; k += PP) {  // face node k = q + P side
        const long long kf = k + 4LL * P * e;
        const double a = av[k % P + ss * (k / P)], sc = nScale[kf];
        sF[slot][0][k] = a * nHat[2 * kf] * sc;
        sF[slot][1][k] = a * nHat[2 * kf + 1] * sc;
      }
    }
    __syncthreads();
    load(p + step);
    if (p >= nPlanes) continue;
    h = sf[slot][0];
    double gx = 0.0, gy = 0.0;
#pragma unroll
    for (int ii = 0; ii < P; ++ii) {
      const int a = ii + RS * j, b = i + RS * ii;
      gx = gx + di[ii] * h[a] + dj[ii] * h[b + 2 * FS];
      gy = gy + di[ii] * h[a + FS] + dj[ii] * h[b + 3 * FS];
    }
    if (kWeak) {
      const double *X = sF[slot][0], *Y = sF[slot][1];
      const int qE = j + P, qW = j + 3 * P, qN = i + 2 * P, qS = i;
      gx = gx + (X[qE] * bi1 + X[qW] * bi0) / wi;
      gx = gx + (X[qN] * bj1 + X[qS] * bj0) / wj;
      gy = gy + (Y[qE] * bi1 + Y[qW] * bi0) / wi;
      gy = gy + (Y[qN] * bj1 + Y[qS] * bj0) / wj;
    }
    double* o = gradF + 2 * (p * PP + n);
    o[0] = gx / Jij;
    o[1] = gy / Jij;
  }
}

// src/SELF_MappedData.f90:1235-1268 (C = 1) and the vector analogue (C = 2)
template <int PC, int C>
__global__ void k_jacobian_weight(double* f, const double* J, int N, int nVar,
                                  long long n) {
  after_previous();
  const int P = nodes<PC>(N);
  GRID_STRIDE(k, n) {
    const long long node = k / C;
    const int ij = node % (P * P);
    int v;
    const long long e = divide(node / (P * P), nVar, v);
    f[k] = f[k] / J[ij + (long long)P * P * e];
  }
}

// src/SELF_MappedData.f90:2220-2269
template <int PC>
__global__ void k_contravariant_projection(double* f, const double* dsdx, int N, int nVar,
                                           long long n) {
  after_previous();
  const int P = nodes<PC>(N);
  GRID_STRIDE(k, n) {
    const int ij = k % (P * P);
    int v;
    const long long e = divide(k / (P * P), nVar, v);
    const double* g = dsdx + 4 * (ij + (long long)P * P * e);
    const double Fx = f[2 * k], Fy = f[2 * k + 1];
    f[2 * k] = g[0] * Fx + g[1] * Fy;
    f[2 * k + 1] = g[2] * Fx + g[3] * Fy;
  }
}

// src/SELF_MappedData.f90:834-917 (C = 1) and 1870-1958 (C = 2): one thread per
// (component, node, var, side, element) output of extBoundary.
template <int PC, int C>
__global__ void k_side_exchange(double* ext, const double* bnd,
                                const int* sideInfo, const int* elemToRank, int rankId,
                                int offset, int N, int nVar, long long n) {
  after_previous();
  const int P = nodes<PC>(N);
  GRID_STRIDE(k, n) {
    const int c = k % C;
    const int i1 = (k / C) % P;
    const long long r = k / ((long long)C * P);  // (var, side, el)
    int v;
    const long long se = divide(r, nVar, v);
    const int s1 = se & 3;
    const long long e1 = se >> 2;
    const int* si = sideInfo + 5 * (s1 + 4 * e1);
    const int bcid = si[4];
    if (bcid != 0) continue;
    const int e2g = si[2];
    if (elemToRank != nullptr && elemToRank[e2g - 1] != rankId) continue;
    const int s2 = si[3] / 10, flip = si[3] - s2 * 10;
    const long long e2 = (long long)e2g - 1 - offset;
    const long long nEl = n / (4LL * C * P * nVar);
    if (e2 < 0 || e2 >= nEl || s2 < 1 || s2 > 4) continue;  // malformed record: leave ext untouched
    int i2;
    if (flip == 0) i2 = i1;
    else if (flip == 1) i2 = N - i1;
    else continue;
    ext[k] = bnd[c + C * (i2 + (long long)P * (v + (long long)nVar * ((s2 - 1) + 4 * e2)))];
  }
}

// src/SELF_MappedData.f90:919-953
__global__ void k_bassi_rebay(double* avg, const double* bnd,
                              const double* ext, long long n) {
  after_previous();
  GRID_STRIDE(k, n) avg[k] = 0.5 * (bnd[k] + ext[k]);
}

// ------------------------------------------------------------------- Model2D
// src/SELF_Model2D.f90:734-748 (workSol may have nWork != nVar variables)
template <int PC>
__global__ void k_update_grk(double* grk, double* sol, const double* dSdt,
                             double a, double g, double dt, int nWork, int N, int nVar, long long n) {
  after_previous();
  const int P2 = nodes<PC>(N) * nodes<PC>(N);
  GRID_STRIDE(k, n) {
    const int ij = k % P2;
    const long long ve = k / P2;
    int v;
    const long long e = divide(ve, nVar, v);
    const long long kw = ij + (long long)P2 * (v + (long long)nWork * e);
    const double G = a * grk[kw] + dSdt[k];
    grk[kw] = G;
    sol[k] = sol[k] + g * dt * G;
  }
}

__global__ void k_update_solution(double* sol, const double* dSdt, double dt, long long n) {
  after_previous();
  GRID_STRIDE(k, n) sol[k] = sol[k] + dt * dSdt[k];
}

// src/SELF_Model2D.f90:845-857
__global__ void k_dsdt(const double* div, const double* src, double* dSdt,
                       long long n) {
  after_previous();
  GRID_STRIDE(k, n) dSdt[k] = src[k] - div[k];
}

// -------------------------------------------------------- LinearShallowWater
// src/models/SELF_LinearShallowWater.f90:298-355; thread per (i, side, el)
template <int PC>
__global__ void k_lsw_bc(const double* sol, double* ext, const double* nHat,
                         const int* sideInfo, int N, int nVar, long long n) {
  after_previous();
  const int P = nodes<PC>(N);
  GRID_STRIDE(k, n) {
    const int i = k % P, s = (k / P) % 4;
    const long long e = k / (4LL * P);
    const int* si = sideInfo + 5 * (s + 4 * e);
    if (si[2] != 0) continue;
    const long long ss = P;  // stride between variables in the face layout
    const long long base = i + (long long)P * nVar * (s + 4 * e);
    if (si[4] == SG_BC_NONORMALFLOW) {
      double ue, ve;
      reflect<double>(sol[base], sol[base + ss], nHat[2 * k], nHat[2 * k + 1], ue, ve);
      ext[base] = ue;
      ext[base + ss] = ve;
      ext[base + 2 * ss] = sol[base + 2 * ss];
    } else {
      ext[base] = 0.0;
      ext[base + ss] = 0.0;
      ext[base + 2 * ss] = 0.0;
    }
  }
}

template <int PC>
__global__ void k_lsw_source(double* src, const double* sol, const double* f,
                             int N, int nVar, long long n) {
  after_previous();
  const int P2 = nodes<PC>(N) * nodes<PC>(N);
  GRID_STRIDE(k, n) {  // (ij, el)
    const int ij = k % P2;
    const long long e = k / P2;
    const long long b = ij + (long long)P2 * nVar * e;
    const double fc = f[k];
    src[b] = fc * sol[b + P2];
    src[b + P2] = -fc * sol[b];
    src[b + 2 * P2] = 0.0;
  }
}

template <int PC>
__global__ void k_lsw_flux(double* flux, const double* sol, const double* H,
                           double g, int N, int nVar, long long n) {
  after_previous();
  const int P2 = nodes<PC>(N) * nodes<PC>(N);
  GRID_STRIDE(k, n) {
    const int ij = k % P2;
    const long long e = k / P2;
    const long long b = ij + (long long)P2 * nVar * e;
    const double Hh = H[k];
    flux[2 * b] = g * sol[b + 2 * P2];
    flux[2 * b + 1] = 0.0;
    flux[2 * (b + P2)] = 0.0;
    flux[2 * (b + P2) + 1] = g * sol[b + 2 * P2];
    flux[2 * (b + 2 * P2)] = Hh * sol[b];
    flux[2 * (b + 2 * P2) + 1] = Hh * sol[b + P2];
  }
}

template <int PC>
__global__ void k_lsw_riemann(double* flux, const double* sol,
                              const double* ext, const double* H,
                              const double* nHat, const double* nScale, double g, int N,
                              int nVar, long long n) {
  after_previous();
  const int P = nodes<PC>(N);
  GRID_STRIDE(k, n) {  // (i, side, el)
    const int i = k % P;
    const long long se = k / P;
    const long long base = i + (long long)P * nVar * se;
    double out[3];
    lsw_riemann<double>(sol[base], sol[base + P], sol[base + 2 * P], ext[base], ext[base + P], ext[base + 2 * P],
                        lsw_face<double>(H[k], g), g, nHat[2 * k], nHat[2 * k + 1], nScale[k], out);
    flux[base] = out[0];
    flux[base + P] = out[1];
    flux[base + 2 * P] = out[2];
  }
}

// -------------------------------------------------------------- ShallowWater
template <int PC>
__global__ void k_sw_bc(const double* sol, double* ext, const double* topoB,
                        const double* nHat, const int* sideInfo, int N, int nVar,
                        long long n) {
  after_previous();
  const int P = nodes<PC>(N);
  GRID_STRIDE(k, n) {
    const int i = k % P, s = (k / P) % 4;
    const long long e = k / (4LL * P);
    const int* si = sideInfo + 5 * (s + 4 * e);
    if (si[2] != 0) continue;
    const long long base = i + (long long)P * nVar * (s + 4 * e);
    if (si[4] == SG_BC_NONORMALFLOW) {
      double ue, ve;
      reflect<double>(sol[base], sol[base + P], nHat[2 * k], nHat[2 * k + 1], ue, ve);
      ext[base] = ue;
      ext[base + P] = ve;
      ext[base + 2 * P] = sol[base + 2 * P];
    } else {
      ext[base] = 0.0;
      ext[base + P] = 0.0;
      ext[base + 2 * P] = topoB[k];
    }
  }
}

template <int PC>
__global__ void k_sw_source(double* src, const double* sol, const double* gH,
                            double fC, double g, int N, int nVar, long long n) {
  after_previous();
  const int P2 = nodes<PC>(N) * nodes<PC>(N);
  GRID_STRIDE(k, n) {
    const int ij = k % P2;
    const long long e = k / P2;
    const long long b = ij + (long long)P2 * nVar * e;
    src[b] = -fC * sol[b + P2] + g * sol[b + 2 * P2] * gH[2 * k];
    src[b + P2] = fC * sol[b] + g * sol[b + 2 * P2] * gH[2 * k + 1];
    src[b + 2 * P2] = 0.0;
  }
}

template <int PC>
__global__ void k_sw_flux(double* flux, const double* sol, const double* vel,
                          double g, int N, int nVar, long long n) {
  after_previous();
  const int P2 = nodes<PC>(N) * nodes<PC>(N);
  GRID_STRIDE(k, n) {
    const int ij = k % P2;
    const long long e = k / P2;
    const long long b = ij + (long long)P2 * nVar * e;
    double Fx[3], Fy[3];
    sw_flux<double>(sol[b], sol[b + P2], sol[b + 2 * P2], vel[2 * k], vel[2 * k + 1], g, Fx, Fy);
    for (int v = 0; v < 3; ++v) {
      flux[2 * (b + v * P2)] = Fx[v];
      flux[2 * (b + v * P2) + 1] = Fy[v];
    }
  }
}

template <int PC>
__global__ void k_sw_riemann(double* flux, const double* sol, const double* ext,
                             const double* vel, const double* velExt,
                             const double* nHat, const double* nScale, double g, int N,
                             int nVar, long long n) {
  after_previous();
  const int P = nodes<PC>(N);
  GRID_STRIDE(k, n) {
    const int i = k % P;
    const long long se = k / P;
    const long long base = i + (long long)P * nVar * se;
    double out[3];
    sw_riemann<double>(sol[base], sol[base + P], sol[base + 2 * P], ext[base], ext[base + P], ext[base + 2 * P],
                       vel[2 * k], vel[2 * k + 1], velExt[2 * k], velExt[2 * k + 1], g, nHat[2 * k],
                       nHat[2 * k + 1], nScale[k], out);
    flux[base] = out[0];
    flux[base + P] = out[1];
    flux[base + 2 * P] = out[2];
  }
}

// velocity = (Hu, Hv)/H on interior nodes (first kernel) and on face nodes
// (second), src/models/SELF_ShallowWater.f90:205-236
template <int PC, bool kFace>
__global__ void k_sw_velocity(const double* sol, double* vel, int N, int nVar,
                              long long n) {
  after_previous();
  const int stride = kFace ? nodes<PC>(N) : nodes<PC>(N) * nodes<PC>(N);
  GRID_STRIDE(k, n) {  // k enumerates (node-or-face-node, block)
    const int q = k % stride;
    const long long blk = k / stride;
    const long long b = q + (long long)stride * nVar * blk;
    const double H = sol[b + 2 * stride];
    vel[2 * k] = sol[b] / H;
    vel[2 * k + 1] = sol[b + stride] / H;
  }
}

// ---------------------------------------------------- CompressibleIdealGas2D
template <int PC>
__global__ void k_cig_source(double* src, const double* sol,
                             const double* envGrad, int N, int nVar, long long n) {
  after_previous();
  const int P2 = nodes<PC>(N) * nodes<PC>(N);
  GRID_STRIDE(k, n) {
    const int ij = k % P2;
    const long long e = k / P2;
    const long long b = ij + (long long)P2 * nVar * e;
    const double* gg = envGrad + 2 * (ij + (long long)P2 * 2 * e);  // variable 1 of 2
    const double gx = gg[0], gy = gg[1];
    const double rhou = sol[b], rhov = sol[b + P2], rho = sol[b + 2 * P2];
    src[b] = -rho * gx;
    src[b + P2] = -rho * gy;
    src[b + 2 * P2] = 0.0;
    src[b + 3 * P2] = -rhou * gx - rhou * gy;
    (void)rhov;
  }
}

template <int PC>
__global__ void k_cig_flux(double* flux, const double* sol, const double* prim,
                           const double* diag, int N, int nVar, long long n) {
  after_previous();
  const int P2 = nodes<PC>(N) * nodes<PC>(N);
  GRID_STRIDE(k, n) {
    const int ij = k % P2;
    const long long e = k / P2;
    const long long b = ij + (long long)P2 * nVar * e;
    double Fx[4], Fy[4];
    // rhoH = rhoE + p, the CPU diagnostic (SELF_CompressibleIdealGas2D.f90:1110)
    const double rhoH = diag ? diag[b + P2] : sol[b + 3 * P2] + prim[b + 3 * P2];
    cig_flux<double>(sol[b], sol[b + P2], prim[b], prim[b + P2], prim[b + 3 * P2], rhoH, Fx, Fy);
    for (int v = 0; v < 4; ++v) {
      flux[2 * (b + v * P2)] = Fx[v];
      flux[2 * (b + v * P2) + 1] = Fy[v];
    }
  }
}

template <int PC>
__global__ void k_cig_llf(double* flux, const double* sol, const double* solE,
                          const double* prim, const double* primE,
                          const double* diag, const double* diagE,
                          const double* nHat, const double* nScale, int N, int nVar,
                          int nDiag, long long n) {
  after_previous();
  const int P = nodes<PC>(N);
  GRID_STRIDE(k, n) {
    const int i = k % P;
    const long long se = k / P;
    const long long b = i + (long long)P * nVar * se;
    const long long bd = i + (long long)P * nDiag * se;
    double L[9], R[9], out[4];
    for (int v = 0; v < 4; ++v) {
      L[v] = sol[b + v * P];
      R[v] = solE[b + v * P];
    }
    L[4] = prim[b];
    L[5] = prim[b + P];
    L[6] = prim[b + 3 * P];
    R[4] = primE[b];
    R[5] = primE[b + P];
    R[6] = primE[b + 3 * P];
    L[7] = diag[bd + P];
    L[8] = diag[bd + 2 * P];
    R[7] = diagE[bd + P];
    R[8] = diagE[bd + 2 * P];
    cig_llf<double>(L, R, nHat[2 * k], nHat[2 * k + 1], nScale[k], out);
    for (int v = 0; v < 4; ++v) flux[b + v * P] = out[v];
  }
}

template <int PC>
__global__ void k_cig_bc(const double* in, double* ext, const double* presc,
                         const double* nHat, const int* sideInfo, int N, int nv,
                         int reflectPair, long long n) {
  after_previous();
  const int P = nodes<PC>(N);
  GRID_STRIDE(k, n) {
    const int i = k % P, s = (k / P) % 4;
    const long long e = k / (4LL * P);
    const int* si = sideInfo + 5 * (s + 4 * e);
    if (si[2] != 0) continue;
    const bool wall = si[4] == SG_BC_NONORMALFLOW;
    if (!wall && si[4] != SG_BC_PRESCRIBED && si[4] != SG_BC_RADIATION) continue;
    // four variables' loads in flight together, ahead of the stores (a store may
    // write what a later load reads, so the compiler keeps their order; a load
    // and a store in turn: 4.0 us on the walls of 64x64 elements at N = 7, now 3.3)
    const long long base = i + (long long)P * nv * (s + 4 * e);
    const double* from = (wall ? in : presc) + base;
    const bool pair = wall && reflectPair;
    const double n1 = pair ? nHat[2 * k] : 0.0, n2 = pair ? nHat[2 * k + 1] : 0.0;
    for (int v = 0; v < nv; v += 4) {
      double x[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) x[q] = v + q < nv ? from[(v + q) * P] : 0.0;
      if (pair && v == 0) {
        const double u0 = x[0], v0 = x[1];
        reflect<double>(u0, v0, n1, n2, x[0], x[1]);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (v + q < nv) ext[base + (v + q) * P] = x[q];
    }
  }
}

// CalculateDiagnostics (mode 0), ConservativeToPrimitive (mode 1),
// ConservativeToEntropy (mode 2); src/models/SELF_CompressibleIdealGas2D.f90:1076-1215
template <int PC>
__global__ void k_cig_pointwise(const double* sol, double* out, double gamma, double Rg,
                                int mode, int N, int nVar, int nOut, long long n) {
  after_previous();
  const int P2 = nodes<PC>(N) * nodes<PC>(N);
  GRID_STRIDE(k, n) {
    const int ij = k % P2;
    const long long e = k / P2;
    const long long b = ij + (long long)P2 * nVar * e;
    const long long o = ij + (long long)P2 * nOut * e;
    const double rhoU = sol[b], rhoV = sol[b + P2], rho = sol[b + 2 * P2], rhoE = sol[b + 3 * P2];
    double u, v, p, rhoKE, rhoH, c;
    cig_state<double>(rhoU, rhoV, rho, rhoE, gamma, u, v, p, rhoKE, rhoH, c);
    if (mode == 0) {
      out[o] = rhoKE;
      out[o + P2] = rhoH;
      out[o + 2 * P2] = c;
      out[o + 3 * P2] = (2.0 / 3.0) * ((rhoE - rhoKE) / rho) / Rg;
    } else if (mode == 1) {
      out[o] = u;
      out[o + P2] = v;
      out[o + 2 * P2] = rho;
      out[o + 3 * P2] = p;
    } else {
      const double s = log(p) - gamma * log(rho);
      out[o] = u * rho / p;
      out[o + P2] = v * rho / p;
      out[o + 2 * P2] = (gamma - s) / (gamma - 1.0) - rhoKE / p;
      out[o + 3 * P2] = -rho / p;
    }
  }
}

}  // namespace
}  // namespace selfgpu

using namespace selfgpu;

#define LAUNCH(kernel, n, ...)                                   \
  do {                                                           \
    long long n_ = (n);                                          \
    if (n_ > 0) launch_dependent_smem(kernel, blocks_for(n_), kThreads, 0, 0, __VA_ARGS__, n_); \
    check_launch(#kernel);                                       \
  } while (0)
// kernel<PC, ...>: the node count of degree N, then the extra template arguments
#define UNPAREN(...) __VA_ARGS__
#define PCV decltype(pc)::value
#define LAUNCH_N(kernel, targs, n, ...)                                                                       \
  do {                                                                                                        \
    const long long n_ = (n);                                                                                 \
    if (n_ > 0) with_nodes(N, [&](auto pc) { launch_dependent_smem(kernel UNPAREN targs, blocks_for(n_), kThreads, 0, 0, __VA_ARGS__, n_); }); \
    check_launch(#kernel);                                                                                    \
  } while (0)

namespace {

// f(integral_constant<int, P>) for the compiled node counts, f(0) for others
template <class F>
void with_nodes(int N, F f) {
  using std::integral_constant;
  switch (N + 1) {
    case 2: f(integral_constant<int, 2>{}); break;
    case 3: f(integral_constant<int, 3>{}); break;
    case 4: f(integral_constant<int, 4>{}); break;
    case 5: f(integral_constant<int, 5>{}); break;
    case 6: f(integral_constant<int, 6>{}); break;
    case 7: f(integral_constant<int, 7>{}); break;
    case 8: f(integral_constant<int, 8>{}); break;
    default: f(integral_constant<int, 0>{}); break;
  }
}

// Launch of a stencil kernel: blocks of `planes` planes with `values` doubles
// of shared memory per plane and `fixed` beside them; false (nothing launched)
// for a degree that is not compiled or arrays beyond the 48 KB of a block.
template <class F>
bool launch_planes(int N, int tasks, long long nPlanes, long long values, long long fixed, F launch) {
  int planes = kThreads / tasks;  // about one task per thread
  planes = (int)std::min<long long>(std::max(planes, 1), nPlanes);
  const size_t smem = (size_t)(fixed + values * planes) * sizeof(double);
  if (N < 1 || N > 7 || smem > 48 * 1024) return false;
  const int blocks = (int)std::min<long long>((nPlanes + planes - 1) / planes, 148LL * 64);
  with_nodes(N, [&](auto pc) {
    if constexpr (decltype(pc)::value > 0) launch(pc, blocks, smem, planes);
  });
  return true;
}

template <int C>
void launch_grid_interp(const double* iM, const double* f, double* fo, int N, int M, long long nPlanes,
                        cudaStream_t st = 0) {
  const int P = N + 1, Q = M + 1;
  const long long n = nPlanes * C * Q * Q;
  const bool small = Q > 1 && (long long)C * Q * Q < 30000;  // k_grid_interp's index range
  if (n > 0 && !(small && launch_planes(N, C * P * Q, nPlanes, (long long)C * P * (P + Q), (long long)P * Q,
                              [&](auto pc, int blocks, size_t smem, int planes) {
                                launch_dependent_smem(k_grid_interp<PCV, C>, blocks, kThreads, smem, st, iM, f, fo, M, planes, nPlanes);
                              }))) {
    if (C == 1) launch_dependent_smem(k_scalar_grid_interp, blocks_for(n), kThreads, 0, st, iM, f, fo, N, M, n);
    else launch_dependent_smem(k_vector_grid_interp, blocks_for(n), kThreads, 0, st, iM, f, fo, N, M, n);
  }
  check_launch("k_grid_interp");
}
template <int C>
void launch_boundary_interp(const double* bM, const double* f, double* fb, int N, int nVar, long long nPlanes,
                            cudaStream_t st = 0) {
  const int P = N + 1;
  const long long n = nPlanes * C * P;
  if (n > 0 && !launch_planes(N, 4 * C * P, nPlanes, (long long)C * P * row_stride(P), 2LL * P,
                              [&](auto pc, int blocks, size_t smem, int planes) {
                                launch_dependent_smem(k_boundary_interp<PCV, C>, blocks, kThreads, smem, st, bM, f, fb, nVar, planes, nPlanes);
                              })) {
    if constexpr (C == 1) launch_dependent_smem(k_scalar_boundary_interp, blocks_for(n), kThreads, 0, st, bM, f, fb, N, nVar, n);
    else launch_dependent_smem(k_multi_boundary_interp<C>, blocks_for(n), kThreads, 0, st, bM, f, fb, N, nVar, n);
  }
  check_launch("k_boundary_interp");
}
// Launch of a derivative kernel: launch(P, blocks) with as many blocks as stay
// resident, each sweeping over the planes; false for a degree that is not compiled.
template <class F>
bool launch_nodes(int N, long long nPlanes, F launch) {
  if (N < 1 || N > 7) return false;
  with_nodes(N, [&](auto pc) {
    if constexpr (PCV > 0) {
      using B = NodeBlock<PCV>;
      launch(pc, (int)std::min<long long>((nPlanes + B::slots - 1) / B::slots, 148LL * 3));
    }
  });
  return true;
}
#define NODE_THREADS NodeBlock<PCV>::threads

void launch_vector_gradient(const double* dM, const double* f, double* df, int N, long long nPlanes,
                            cudaStream_t st = 0) {
  const long long n = nPlanes * (N + 1) * (N + 1);
  if (n > 0 && !launch_nodes(N, nPlanes, [&](auto pc, int blocks) {
        launch_dependent_smem(k_vector_gradient<PCV>, blocks, NODE_THREADS, 0, st, dM, f, df, nPlanes);
      }))
    launch_dependent_smem(k_vector_gradient_any, blocks_for(n), kThreads, 0, st, dM, f, df, N, n);
  check_launch("k_vector_gradient");
}

}  // namespace

extern "C" {

void ScalarGridInterp_2D_gpu_wrapper(double** iMatrix, double** f, double** fInterp, int N, int M, int nVar, int nEl) {
  launch_grid_interp<1>(*iMatrix, *f, *fInterp, N, M, (long long)nVar * nEl);
}
void VectorGridInterp_2D_gpu_wrapper(double** iMatrix, double** f, double** fInterp, int N, int M, int nVar, int nEl) {
  launch_grid_interp<2>(*iMatrix, *f, *fInterp, N, M, (long long)nVar * nEl);
}
void ScalarBoundaryInterp_2D_gpu_wrapper(double** bMatrix, double** f, double** fBound, int N, int nVar, int nEl) {
  launch_boundary_interp<1>(*bMatrix, *f, *fBound, N, nVar, (long long)nVar * nEl);
}
void VectorBoundaryInterp_2D_gpu_wrapper(double** bMatrix, double** f, double** fBound, int N, int nVar, int nEl) {
  launch_boundary_interp<2>(*bMatrix, *f, *fBound, N, nVar, (long long)nVar * nEl);
}
void TensorBoundaryInterp_2D_gpu_wrapper(double** bMatrix, double** f, double** fBound, int N, int nVar, int nEl) {
  launch_boundary_interp<4>(*bMatrix, *f, *fBound, N, nVar, (long long)nVar * nEl);
}
void VectorGradient_2D_gpu_wrapper(double** dMatrix, double** f, double** df, int N, int nVar, int nEl) {
  launch_vector_gradient(*dMatrix, *f, *df, N, (long long)nVar * nEl);
}
void VectorDGDivergence_2D_gpu_wrapper(double** dgMatrix, double** bMatrix, double** qWeights, double** f, double** bf,
                                       double** df, int N, int nVar, int nEl) {
  const long long nPlanes = (long long)nVar * nEl, n = nPlanes * (N + 1) * (N + 1);
  if (n > 0 && !launch_nodes(N, nPlanes, [&](auto pc, int blocks) {
        launch_dependent_smem(k_vector_dg_divergence<PCV>, blocks, NODE_THREADS, 0, 0, *dgMatrix, *bMatrix, *qWeights, *f, *bf, *df, nVar, nPlanes);
      }))
    launch_dependent_smem(k_vector_dg_divergence_any, blocks_for(n), kThreads, 0, 0, *dgMatrix, *bMatrix, *qWeights, *f, *bf, *df, N, nVar, n);
  check_launch("k_vector_dg_divergence");
}
void Determinant_Tensor2D_gpu_wrapper(double** tensor, double** detTensor, int N, int nVar, int nEl) {
  LAUNCH(k_determinant, (long long)(N + 1) * (N + 1) * nVar * nEl, *tensor, *detTensor);
}
void CalculateContravariantBasis_SEMQuad_gpu_wrapper(double** dxds, double** dsdx, int N, int nEl) {
  LAUNCH(k_contravariant_basis, (long long)(N + 1) * (N + 1) * nEl, *dxds, *dsdx);
}
void AdjustBoundaryContravariantBasis_SEMQuad_gpu_wrapper(double** dsdx, double** J, int N, int nEl) {
  LAUNCH(k_adjust_boundary_basis, (long long)(N + 1) * 4 * nEl, *dsdx, *J, N);
}
void GradientBR_MappedScalar2D_gpu_wrapper(double** scalar, double** avgBoundary, double** dsdx, double** jacobian,
                                           double** nHat, double** nScale, double** gradF, double** dgMatrix,
                                           double** bMatrix, double** qWeights, int N, int nVar, int nEl) {
  const long long nPlanes = (long long)nVar * nEl, n = nPlanes * (N + 1) * (N + 1);
  if (n > 0 && !launch_nodes(N, nPlanes, [&](auto pc, int blocks) {
        launch_dependent_smem(k_gradient<PCV, true>, blocks, NODE_THREADS, 0, 0, *scalar, *avgBoundary, *dsdx, *jacobian, *nHat, *nScale, *gradF,
                                                        *dgMatrix, *bMatrix, *qWeights, nVar, nPlanes);
      }))
    launch_dependent_smem(k_gradient_br, blocks_for(n), kThreads, 0, 0, *scalar, *avgBoundary, *dsdx, *jacobian, *nHat, *nScale, *gradF,
                                               *dgMatrix, *bMatrix, *qWeights, N, nVar, n);
  check_launch("k_gradient_br");
}
void GradientSF_MappedScalar2D_gpu_wrapper(double** scalar, double** dsdx, double** jacobian, double** gradF,
                                           double** dMatrix, int N, int nVar, int nEl) {
  const long long nPlanes = (long long)nVar * nEl, n = nPlanes * (N + 1) * (N + 1);
  if (n > 0 && !launch_nodes(N, nPlanes, [&](auto pc, int blocks) {
        launch_dependent_smem(k_gradient<PCV, false>, blocks, NODE_THREADS, 0, 0, *scalar, nullptr, *dsdx, *jacobian, nullptr, nullptr, *gradF,
                                                         *dMatrix, nullptr, nullptr, nVar, nPlanes);
      }))
    launch_dependent_smem(k_gradient_sf, blocks_for(n), kThreads, 0, 0, *scalar, *dsdx, *jacobian, *gradF, *dMatrix, N, nVar, n);
  check_launch("k_gradient_sf");
}
void JacobianWeight_MappedScalar2D_gpu_wrapper(double** scalar, double** jacobian, int N, int nVar, int nEl) {
  LAUNCH_N(k_jacobian_weight, (<PCV, 1>), (long long)(N + 1) * (N + 1) * nVar * nEl, *scalar, *jacobian, N, nVar);
}
void JacobianWeight_MappedVector2D_gpu_wrapper(double** vector, double** jacobian, int N, int nVar, int nEl) {
  LAUNCH_N(k_jacobian_weight, (<PCV, 2>), 2LL * (N + 1) * (N + 1) * nVar * nEl, *vector, *jacobian, N, nVar);
}
void ContravariantProjection_MappedVector2D_gpu_wrapper(double** vector, double** dsdx, int N, int nVar, int nEl) {
  LAUNCH_N(k_contravariant_projection, (<PCV>), (long long)(N + 1) * (N + 1) * nVar * nEl, *vector, *dsdx, N, nVar);
}
void SideExchange_MappedScalar2D_gpu_wrapper(double** extBoundary, double** boundary, int** sideInfo,
                                             int** elemToRank, int rankId, int offset, int N, int nVar, int nEl) {
  LAUNCH_N(k_side_exchange, (<PCV, 1>), (long long)(N + 1) * nVar * 4 * nEl, *extBoundary, *boundary, *sideInfo,
         elemToRank ? *elemToRank : nullptr, rankId, offset, N, nVar);
}
void SideExchange_MappedVector2D_gpu_wrapper(double** extBoundary, double** boundary, int** sideInfo,
                                             int** elemToRank, int rankId, int offset, int N, int nVar, int nEl) {
  LAUNCH_N(k_side_exchange, (<PCV, 2>), 2LL * (N + 1) * nVar * 4 * nEl, *extBoundary, *boundary, *sideInfo,
         elemToRank ? *elemToRank : nullptr, rankId, offset, N, nVar);
}
void BassiRebaySides_MappedScalar2D_gpu_wrapper(double** avgBoundary, double** boundary, double** extBoundary, int N,
                                                int nVar, int nEl) {
  LAUNCH(k_bassi_rebay, (long long)(N + 1) * nVar * 4 * nEl, *avgBoundary, *boundary, *extBoundary);
}
void UpdateGRK_Model2D_gpu_wrapper(double** grk, double** solution, double** dSdt, double rk_a, double rk_g, double dt,
                                   int nWork, int N, int nVar, int nEl) {
  LAUNCH_N(k_update_grk, (<PCV>), (long long)(N + 1) * (N + 1) * nVar * nEl, *grk, *solution, *dSdt, rk_a, rk_g, dt, nWork, N,
         nVar);
}
void UpdateSolution_Model2D_gpu_wrapper(double** solution, double** dSdt, double dt, int N, int nVar, int nEl) {
  LAUNCH(k_update_solution, (long long)(N + 1) * (N + 1) * nVar * nEl, *solution, *dSdt, dt);
}
void CalculateDSDt_Model2D_gpu_wrapper(double** fluxDivergence, double** source, double** dSdt, int N, int nVar,
                                       int nEl) {
  LAUNCH(k_dsdt, (long long)(N + 1) * (N + 1) * nVar * nEl, *fluxDivergence, *source, *dSdt);
}
void SetBoundaryCondition_LinearShallowWater_gpu_wrapper(double** solution, double** extBoundary, double** nHat,
                                                         int** sideInfo, int N, int nVar, int nEl) {
  LAUNCH_N(k_lsw_bc, (<PCV>), (long long)(N + 1) * 4 * nEl, *solution, *extBoundary, *nHat, *sideInfo, N, nVar);
}
void Source_LinearShallowWater_gpu_wrapper(double** source, double** solution, double** f, int N, int nVar, int nEl) {
  LAUNCH_N(k_lsw_source, (<PCV>), (long long)(N + 1) * (N + 1) * nEl, *source, *solution, *f, N, nVar);
}
void Flux_LinearShallowWater_gpu_wrapper(double** flux, double** solution, double** H, double g, int N, int nVar,
                                         int nEl) {
  LAUNCH_N(k_lsw_flux, (<PCV>), (long long)(N + 1) * (N + 1) * nEl, *flux, *solution, *H, g, N, nVar);
}
void RiemannSolver_LinearShallowWater_gpu_wrapper(double** flux, double** solution, double** extBoundary, double** H,
                                                  double** nHat, double** nScale, double g, int N, int nVar,
                                                  int nEl) {
  LAUNCH_N(k_lsw_riemann, (<PCV>), (long long)(N + 1) * 4 * nEl, *flux, *solution, *extBoundary, *H, *nHat, *nScale, g, N, nVar);
}
void SetBoundaryCondition_ShallowWater_gpu_wrapper(double** solution, double** extBoundary, double** topoBoundary,
                                                   double** nHat, int** sideInfo, int N, int nVar, int nEl) {
  LAUNCH_N(k_sw_bc, (<PCV>), (long long)(N + 1) * 4 * nEl, *solution, *extBoundary, *topoBoundary, *nHat, *sideInfo, N, nVar);
}
void Source_ShallowWater_gpu_wrapper(double** source, double** solution, double** gradH, double fCori, double g, int N,
                                     int nVar, int nEl) {
  LAUNCH_N(k_sw_source, (<PCV>), (long long)(N + 1) * (N + 1) * nEl, *source, *solution, *gradH, fCori, g, N, nVar);
}
void Flux_ShallowWater_gpu_wrapper(double** flux, double** solution, double** velocity, double g, int N, int nVar,
                                   int nEl) {
  LAUNCH_N(k_sw_flux, (<PCV>), (long long)(N + 1) * (N + 1) * nEl, *flux, *solution, *velocity, g, N, nVar);
}
void RiemannSolver_ShallowWater_gpu_wrapper(double** flux, double** solution, double** extBoundary, double** velocity,
                                            double** extVelocity, double** nHat, double** nScale, double g, int N,
                                            int nVar, int nEl) {
  LAUNCH_N(k_sw_riemann, (<PCV>), (long long)(N + 1) * 4 * nEl, *flux, *solution, *extBoundary, *velocity, *extVelocity, *nHat,
         *nScale, g, N, nVar);
}
void PreTendency_ShallowWater_gpu_wrapper(double** solution, double** solutionBoundary, double** velocity,
                                          double** velocityBoundary, int N, int nVar, int nEl) {
  const int P = N + 1;
  LAUNCH_N(k_sw_velocity, (<PCV, false>), (long long)P * P * nEl, *solution, *velocity, N, nVar);
  LAUNCH_N(k_sw_velocity, (<PCV, true>), (long long)P * 4 * nEl, *solutionBoundary, *velocityBoundary, N, nVar);
}
void Source_CompressibleIdealGas2D_gpu_wrapper(double** source, double** solution, double** environmentalsGradient,
                                               int N, int nVar, int nEl) {
  LAUNCH_N(k_cig_source, (<PCV>), (long long)(N + 1) * (N + 1) * nEl, *source, *solution, *environmentalsGradient, N, nVar);
}
void Flux_CompressibleIdealGas2D_gpu_wrapper(double** flux, double** solution, double** primitive, int N, int nVar,
                                             int nEl) {
  // The signature carries no diagnostics array; rhoH = rhoE + p is formed from
  // the solution and the primitive pressure, as the reference device kernel does.
  LAUNCH_N(k_cig_flux, (<PCV>), (long long)(N + 1) * (N + 1) * nEl, *flux, *solution, *primitive, (const double*)nullptr, N, nVar);
}
void NaiveLLF_CompressibleIdealGas2D_gpu_wrapper(double** flux, double** solution, double** extSolution,
                                                 double** primitive, double** extPrimitive, double** diagnostics,
                                                 double** extDiagnostics, double** nHat, double** nScale, int N,
                                                 int nVar, int nDiag, int nEl) {
  LAUNCH_N(k_cig_llf, (<PCV>), (long long)(N + 1) * 4 * nEl, *flux, *solution, *extSolution, *primitive, *extPrimitive,
         *diagnostics, *extDiagnostics, *nHat, *nScale, N, nVar, nDiag);
}
void SetBoundaryCondition_CompressibleIdealGas2D_gpu_wrapper(
    double** solution, double** extSolution, double** prescribedSolution, double** primitive, double** extPrimitive,
    double** prescribedPrimitive, double** diagnostics, double** extDiagnostics, double** prescribedDiagnostics,
    double** nHat, int** sideInfo, int N, int nVar, int nDiag, int nEl) {
  const long long n = (long long)(N + 1) * 4 * nEl;
  LAUNCH_N(k_cig_bc, (<PCV>), n, *solution, *extSolution, *prescribedSolution, *nHat, *sideInfo, N, nVar, 1);
  LAUNCH_N(k_cig_bc, (<PCV>), n, *primitive, *extPrimitive, *prescribedPrimitive, *nHat, *sideInfo, N, nVar, 1);
  LAUNCH_N(k_cig_bc, (<PCV>), n, *diagnostics, *extDiagnostics, *prescribedDiagnostics, *nHat, *sideInfo, N, nDiag, 0);
}
void CalculateDiagnostics_CompressibleIdealGas2D_gpu_wrapper(double** solution, double** diagnostics,
                                                             double expansionFactor, double R, int N, int nVar,
                                                             int nDiag, int nEl) {
  LAUNCH_N(k_cig_pointwise, (<PCV>), (long long)(N + 1) * (N + 1) * nEl, *solution, *diagnostics, expansionFactor, R, 0, N, nVar,
         nDiag);
}
void ConservativeToPrimitive_CompressibleIdealGas2D_gpu_wrapper(double** solution, double** primitive,
                                                                double expansionFactor, int N, int nVar, int nEl) {
  LAUNCH_N(k_cig_pointwise, (<PCV>), (long long)(N + 1) * (N + 1) * nEl, *solution, *primitive, expansionFactor, 1.0, 1, N, nVar,
         nVar);
}
void ConservativeToEntropy_CompressibleIdealGas2D_gpu_wrapper(double** solution, double** entropy,
                                                              double expansionFactor, int N, int nVar, int nEl) {
  LAUNCH_N(k_cig_pointwise, (<PCV>), (long long)(N + 1) * (N + 1) * nEl, *solution, *entropy, expansionFactor, 1.0, 2, N, nVar,
         nVar);
}

}  // extern "C"

// ---------------------------------------------------------- device geometry
extern "C" int selfgpu_semquad_generate(int N, int nEl, const double* nodeCoords_d, const double* m2m_iMatrix,
                                        const double* dMatrix, const double* bMatrix, double* x_d, double* dxds_d,
                                        double* dsdx_d, double* J_d, double* dsdxB_d, double* JB_d, double* nHat_d,
                                        double* nScale_d, void* stream) {
  if (N < 1 || N > 15 || nEl < 1 || !nodeCoords_d || !m2m_iMatrix || !dMatrix || !bMatrix || !x_d || !dxds_d ||
      !dsdx_d || !J_d || !dsdxB_d || !JB_d || !nHat_d || !nScale_d)
    return set_error(SELFGPU_ERR_ARG, "selfgpu_semquad_generate: bad arguments");
  cudaStream_t st = (cudaStream_t)stream;
  const int P = N + 1;
  // Matrices to the device: iM (0:1,0:N), dM (P*P), bM (P*2)
  double* mats = nullptr;
  const size_t nm = 2 * P + P * P + 2 * P;
  if (cudaMalloc(&mats, nm * sizeof(double)) != cudaSuccess)
    return set_error(SELFGPU_ERR_CUDA, "selfgpu_semquad_generate: cudaMalloc failed");
  cudaMemcpyAsync(mats, m2m_iMatrix, 2 * P * sizeof(double), cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(mats + 2 * P, dMatrix, P * P * sizeof(double), cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(mats + 2 * P + P * P, bMatrix, 2 * P * sizeof(double), cudaMemcpyHostToDevice, st);
  const double *iM = mats, *dM = mats + 2 * P, *bM = mats + 2 * P + P * P;
  const long long nNodes = (long long)P * P * nEl, nFace = (long long)P * 4 * nEl;
  // GenerateFromMesh_SEMQuad: x = GridInterp(nodeCoords), src/SELF_Geometry.f90:393-435
  launch_grid_interp<2>(iM, nodeCoords_d, x_d, 1, N, nEl, st);
  // CalculateMetricTerms_SEMQuad, src/SELF_Geometry.f90:528-552
  launch_vector_gradient(dM, x_d, dxds_d, N, nEl, st);
  launch_dependent_smem(k_determinant, blocks_for(nNodes), kThreads, 0, st, dxds_d, J_d, nNodes);
  launch_boundary_interp<1>(bM, J_d, JB_d, N, 1, nEl, st);
  launch_dependent_smem(k_contravariant_basis, blocks_for(nNodes), kThreads, 0, st, dxds_d, dsdx_d, nNodes);
  launch_boundary_interp<4>(bM, dsdx_d, dsdxB_d, N, 1, nEl, st);
  launch_dependent_smem(k_face_normals, blocks_for(nFace), kThreads, 0, st, dsdxB_d, JB_d, nHat_d, nScale_d, N, nFace);
  cudaError_t e = cudaStreamSynchronize(st);
  cudaFree(mats);
  if (e != cudaSuccess) return set_error(SELFGPU_ERR_CUDA, std::string("selfgpu_semquad_generate: ") + cudaGetErrorString(e));
  e = cudaGetLastError();
  if (e != cudaSuccess) return set_error(SELFGPU_ERR_CUDA, std::string("selfgpu_semquad_generate: ") + cudaGetErrorString(e));
  return SELFGPU_OK;
}
