// Training and standalone inference kernels of the closure MLP
// (36 -> 32 -> 32 -> 1, ReLU, output clamped to [0, 1]; see av_closure.cuh).
//
// Training: minibatch Adam on float32 master weights, two kernels per step:
//   k_grad  rounds the weights to bfloat16 for the forward pass (the precision
//           the closure runs in) and takes the batch in tiles of 32 samples; a
//           block keeps its tiles' activations and deltas in shared memory and
//           every thread sums its own few parameters' gradients over the tile's
//           samples in registers (dW = delta^T activation, an outer-product
//           contraction), so the block writes each partial sum once;
//   k_adam  adds the blocks' partial sums in a fixed order and updates.
// Samples are drawn with replacement by a counter-based hash of
// (seed, step, lane) and every sum has a fixed order, so a run is reproducible
// bit for bit for a given seed.
//
// Loss: (clamp(z) - y)^2 with the gradient passed straight through the clamp
// when z lies on the wrong side of it (z < 0 < y or z > 1 > y); a clamped
// output on the target's side of the clamp has zero gradient.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstring>
#include <memory>
#include <new>
#include <string>

#include "av_closure.cuh"
#include "selfgpu_internal.h"

using namespace selfgpu;

namespace {

constexpr int IN = kMlpIn, H = kMlpHidden;
constexpr int oW1 = 0, oB1 = oW1 + H * IN, oW2 = oB1 + H, oB2 = oW2 + H * H, oW3 = oB2 + H, oB3 = oW3 + H;
constexpr int NP = oB3 + 1;  // 2273 master parameters
static_assert(NP == SELFGPU_MLP_MASTER, "master parameter count");
static_assert(kMlpWeights == SELFGPU_MLP_WEIGHTS && kMlpFloats == SELFGPU_MLP_PARAMS, "closure weight layout");

__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

__device__ __forceinline__ bool is_weight(int k) {
  return (k >= oW1 && k < oB1) || (k >= oW2 && k < oB2) || (k >= oW3 && k < oB3);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

constexpr int kTile = 32;            // samples per tile, one per lane
constexpr int kGradThreads = 256;
constexpr int NPP = (NP + 31) / 32 * 32;  // stride of a block's partial sums
constexpr int kMaxGradBlocks = 296;  // two blocks per SM; larger batches loop over tiles

// Sums of eight values by pairs.
__device__ __forceinline__ float pairwise(const float v[8]) {
  return ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
}

// A tile's products D[r][row] A[r][col + k], k < K, summed over its samples and
// added to acc: four chains of eight samples, then by pairs, so that a value
// passes through ten roundings at most (one chain over the tile would be 32, and
// as many more for each further tile of the block).
template <int K, int W>
__device__ __forceinline__ void tile_sums(const float (*D)[H + 1], const float (*A)[W], int row, int col,
                                          float acc[9]) {
  float c[4][K];
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int k = 0; k < K; ++k) c[q][k] = 0.f;
#pragma unroll 2
  for (int r = 0; r < kTile / 4; ++r)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float d = D[r + kTile / 4 * q][row];
#pragma unroll
      for (int k = 0; k < K; ++k) c[q][k] = fmaf(d, A[r + kTile / 4 * q][col + k], c[q][k]);
    }
#pragma unroll
  for (int k = 0; k < K; ++k) acc[k] = acc[k] + ((c[0][k] + c[1][k]) + (c[2][k] + c[3][k]));
}

// Latency bounds a step (a 4096-sample batch is 54 MFLOP): 128 tiles on as
// many SMs.  Adding each sample's gradient to shared memory by warp shuffles
// (2 273 five-step sums per warp, a block per 256 samples) took 390 us for a
// 4096-sample step; this kernel and k_adam together are launch-bound.
__global__ void __launch_bounds__(kGradThreads) k_grad(const float* feat, const float* label, int n,
                                                       const float* master, float* part, float* lossPart,
                                                       unsigned long long seed, long long step, int batch) {
  // activations and deltas [sample][unit]; the odd strides keep the lanes'
  // (one sample each) accesses to one unit in distinct banks
  __shared__ float sw[NP], F[kTile][IN + 1], H1[kTile][H + 1], H2[kTile][H + 1], D1[kTile][H + 1], D2[kTile][H + 1];
  __shared__ float sy[kTile], sg[kTile];
  __shared__ long long sidx[kTile];
  const int t = threadIdx.x, s = t & 31, w = t >> 5;
  auto gather = [&](int tile) {  // the tile's samples
    if (t < kTile) {
      const long long b = (long long)tile * kTile + t;
      const long long idx = b < batch ? (long long)(mix64(seed ^ mix64((unsigned long long)step * 0x100000001ull +
                                                                       (unsigned long long)b)) %
                                                    (unsigned long long)n)
                                      : -1;
      sidx[t] = idx;
      sy[t] = idx >= 0 ? label[idx] : 0.f;
    }
    __syncthreads();
    for (int k = t; k < kTile * IN; k += kGradThreads) {
      const int r = k / IN, c = k - r * IN;
      const long long idx = sidx[r];
      F[r][c] = idx >= 0 ? feat[c + (long long)IN * idx] : 0.f;
    }
  };
  // the first tile's samples, which no step changes, before the wait
  gather(blockIdx.x);
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the previous step's weights
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  for (int k = t; k < NP; k += kGradThreads) {
    const float m = master[k];
    sw[k] = is_weight(k) ? __bfloat162float(__float2bfloat16_rn(m)) : m;
  }
  // this thread's parameters: 9 of W1 (threads 0-127) or 8 of W2 (128-255),
  // one row's consecutive columns; threads 0-96 also one of b1, b2, w3, b3
  const int half = t >> 7, row = (t & 127) >> 2, col = (t & 3) * (half ? 8 : 9);
  float acc[9], accB = 0.f, lsum = 0.f;
#pragma unroll
  for (int k = 0; k < 9; ++k) acc[k] = 0.f;
  const int tiles = (batch + kTile - 1) / kTile;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    __syncthreads();  // the weights and the first tile, or the previous tile's arrays
    if (tile != (int)blockIdx.x) {
      gather(tile);
      __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {  // lane = sample, warp = 4 hidden units
      const int j = 4 * w + u;
      float a = 0.f;
#pragma unroll
      for (int k = 0; k < IN; ++k) a = fmaf(sw[oW1 + j * IN + k], F[s][k], a);
      a = a + sw[oB1 + j];
      H1[s][j] = a > 0.f ? a : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = 4 * w + u;
      float a = 0.f;
#pragma unroll
      for (int k = 0; k < H; ++k) a = fmaf(sw[oW2 + j * H + k], H1[s][k], a);
      a = a + sw[oB2 + j];
      H2[s][j] = a > 0.f ? a : 0.f;
    }
    __syncthreads();
    if (w == 0) {
      float z = 0.f;
#pragma unroll
      for (int k = 0; k < H; ++k) z = fmaf(sw[oW3 + k], H2[s][k], z);
      z = z + sw[oB3];
      const long long idx = sidx[s];
      const float y = sy[s];
      const float a = z < 0.f ? 0.f : (z > 1.f ? 1.f : z);
      float d = a - y;
      if ((z < 0.f && y > 0.f) || (z > 1.f && y < 1.f)) d = z - y;  // straight through the clamp
      sg[s] = idx >= 0 ? 2.f * d / (float)batch : 0.f;  // lanes beyond the batch carry no gradient
      lsum += warp_sum(idx >= 0 ? (a - y) * (a - y) : 0.f);
    }
    __syncthreads();
    const float g = sg[s];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = 4 * w + u;
      D2[s][j] = H2[s][j] > 0.f ? g * sw[oW3 + j] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = 4 * w + u;
      float a = 0.f;
#pragma unroll
      for (int j = 0; j < H; ++j) a = fmaf(sw[oW2 + j * H + k], D2[s][j], a);
      D1[s][k] = H1[s][k] > 0.f ? a : 0.f;
    }
    __syncthreads();
    if (half == 0) tile_sums<9, IN + 1>(D1, F, row, col, acc);
    else tile_sums<8, H + 1>(D2, H1, row, col, acc);
    if (t < 3 * H + 1) {
      float v[kTile / 4];
#pragma unroll
      for (int q = 0; q < kTile / 4; ++q) {
        v[q] = 0.f;
#pragma unroll
        for (int r = 4 * q; r < 4 * q + 4; ++r)
          v[q] = v[q] + (t < H ? D1[r][t] : t < 2 * H ? D2[r][t - H] : t < 3 * H ? sg[r] * H2[r][t - 2 * H] : sg[r]);
      }
      accB = accB + pairwise(v);
    }
  }
  float* o = part + (size_t)NPP * blockIdx.x;
#pragma unroll
  for (int k = 0; k < 9; ++k)
    if (half == 0) o[oW1 + row * IN + col + k] = acc[k];
    else if (k < 8) o[oW2 + row * H + col + k] = acc[k];
  if (t < 3 * H + 1) o[t < H ? oB1 + t : t < 2 * H ? oB2 + t - H : t < 3 * H ? oW3 + t - 2 * H : oB3] = accB;
  if (t == 0) lossPart[blockIdx.x] = lsum;
}

// 32 parameters per block: lane = parameter, warp = every eighth block's
// partial sum in eight chains, then the eight strips by pairs.
__global__ void __launch_bounds__(256) k_adam(float* master, const float* part, const float* lossPart, int blocks,
                                              float* m1, float* m2, float* loss, float lr, float c1, float c2) {
  __shared__ float strip[8][32];
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int k = blockIdx.x * 32 + lane;
  // Only this wait makes earlier grids' writes visible here: this step's partial
  // sums, and the moments and weights of the previous step's k_adam.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  float m1k = 0.f, m2k = 0.f, mk = 0.f;  // in flight during the sums
  if (w == 0 && k < NP) m1k = m1[k], m2k = m2[k], mk = master[k];
  float s[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) s[q] = 0.f;
  if (k < NP)
    for (int r = w; r < blocks; r += 64) {  // (a batch of 4 096 samples: two rounds of loads)
      float x[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) x[q] = r + 8 * q < blocks ? part[(size_t)NPP * (r + 8 * q) + k] : 0.f;
#pragma unroll
      for (int q = 0; q < 8; ++q) s[q] = s[q] + x[q];
    }
  strip[w][lane] = pairwise(s);
  __syncthreads();
  if (w == 0 && k < NP) {
    float v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = strip[r][lane];
    const float gk = pairwise(v);
    m1[k] = m1k = b1 * m1k + (1.f - b1) * gk;
    m2[k] = m2k = b2 * m2k + (1.f - b2) * gk * gk;
    const float mh = m1k / c1, vh = m2k / c2;
    master[k] = mk - lr * mh / (sqrtf(vh) + eps);
  }
  if (blockIdx.x == 0 && w == 1) {
    float l = 0.f;
    for (int r = lane; r < blocks; r += 32) l += lossPart[r];
    l = warp_sum(l);
    if (lane == 0) *loss += l;
  }
}

// Minimum and maximum of each feature over the samples (NaN where one is NaN),
// by the last of the blocks to finish.  Consecutive threads read consecutive
// values; a thread's values all belong to its own feature.  (Two reductions by
// the caller's tensor library with a copy each: 79 us for 16 384 samples; this
// kernel's result comes back with the trained weights.)
constexpr int kRangeBlocks = 148, kRangeRows = 8, kRangeThreads = kRangeRows * IN;
struct RangeScratch {
  float result[2 * IN];  // minima, maxima
  unsigned done;         // zero before the launch
  float part[kRangeBlocks][2 * IN];
};
__device__ __forceinline__ float min_nan(float a, float b) { return a != a ? a : (b < a || b != b ? b : a); }
__device__ __forceinline__ float max_nan(float a, float b) { return a != a ? a : (b > a || b != b ? b : a); }
__global__ void __launch_bounds__(kRangeThreads) k_range(const float* __restrict__ feat, int n, RangeScratch* x) {
  __shared__ float slo[kRangeRows][IN], shi[kRangeRows][IN];
  __shared__ bool last;
  const int t = threadIdx.x, r = t / IN, c = t - r * IN;
  const float first = feat[c];
  float lo = first, hi = first;
  for (long long row = (long long)blockIdx.x * kRangeRows + r; row < n; row += (long long)gridDim.x * kRangeRows) {
    const float v = feat[row * IN + c];
    lo = min_nan(lo, v);
    hi = max_nan(hi, v);
  }
  auto block_range = [&]() {  // over the rows of threads, on the first
    slo[r][c] = lo;
    shi[r][c] = hi;
    __syncthreads();
    if (r == 0)
      for (int k = 1; k < kRangeRows; ++k) {
        lo = min_nan(lo, slo[k][c]);
        hi = max_nan(hi, shi[k][c]);
      }
  };
  block_range();
  if (r == 0) {
    x->part[blockIdx.x][c] = lo;
    x->part[blockIdx.x][IN + c] = hi;
    __threadfence();
  }
  __syncthreads();
  if (t == 0) {
    last = atomicAdd(&x->done, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  lo = hi = first;
  for (int b = r; b < (int)gridDim.x; b += kRangeRows) {
    lo = min_nan(lo, __ldcg(&x->part[b][c]));
    hi = max_nan(hi, __ldcg(&x->part[b][IN + c]));
  }
  block_range();
  if (r == 0) {
    x->result[c] = lo;
    x->result[IN + c] = hi;
  }
}

// Weights (bfloat16 pairs) and parameters, passed by value: no device buffer
// and no copy per call.
struct MlpArgs {
  uint32_t w[kMlpWeights / 2];
  float p[kMlpFloats];
};
static_assert(kMlpWeights % 2 == 0, "weights travel as pairs");

// The arithmetic of the in-stage MLP (av_closure.cuh).  Tiles of 32 samples as
// in k_grad: lane = sample, warp = four hidden units.  (One thread per sample
// evaluated its 2 208 products alone on at most one block per 256 samples:
// 28 us for 16 384 samples.)
__global__ void __launch_bounds__(kGradThreads) k_infer(const float* __restrict__ feat, int n,
                                                        const __grid_constant__ MlpArgs args,
                                                        float* __restrict__ out) {
  __shared__ float sw[kMlpWeights], sB[2 * H + 1], F[kTile][IN + 1], H1[kTile][H + 1], H2[kTile][H + 1];
  const int t = threadIdx.x, s = t & 31, w = t >> 5;
  for (int k = t; k < kMlpWeights / 2; k += kGradThreads) {
    const uint32_t x = args.w[k];
    sw[2 * k] = __uint_as_float(x << 16);
    sw[2 * k + 1] = __uint_as_float(x & 0xffff0000u);
  }
  for (int k = t; k < 2 * H + 1; k += kGradThreads) sB[k] = args.p[k];
  const float *sW1 = sw, *sW2 = sw + H * IN, *sw3 = sW2 + H * H;
  for (long long s0 = (long long)blockIdx.x * kTile; s0 < n; s0 += (long long)gridDim.x * kTile) {
    const int live = n - s0 < kTile ? (int)(n - s0) : kTile;
    __syncthreads();
    for (int k = t; k < kTile * IN; k += kGradThreads) {
      const int r = k / IN;
      F[r][k - r * IN] = r < live ? feat[IN * s0 + k] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = 4 * w + u;
      float acc = 0.f;
#pragma unroll
      for (int k = 0; k < IN; ++k) acc = fmaf(sW1[j * IN + k], F[s][k], acc);
      acc = acc + sB[j];
      H1[s][j] = acc > 0.f ? acc : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = 4 * w + u;
      float acc = 0.f;
#pragma unroll
      for (int k = 0; k < H; ++k) acc = fmaf(sW2[j * H + k], H1[s][k], acc);
      acc = acc + sB[H + j];
      H2[s][j] = acc > 0.f ? acc : 0.f;
    }
    __syncthreads();
    if (w == 0 && s < live) {
      float z = 0.f;
#pragma unroll
      for (int j = 0; j < H; ++j) z = fmaf(sw3[j], H2[s][j], z);
      z = z + sB[2 * H];
      out[s0 + s] = z < 0.f ? 0.f : (z > 1.f ? 1.f : z);
    }
  }
}

int fail(const char* where, cudaError_t e) {
  return set_error(SELFGPU_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(e));
}

}  // namespace

extern "C" {

int selfgpu_mlp_train(const float* features, const float* labels, int n, int epochs, int batch, float lr,
                      unsigned long long seed, float* params, float* lossPerEpoch, void* stream) {
  return selfgpu_mlp_train_range(features, labels, n, epochs, batch, lr, seed, params, lossPerEpoch, nullptr, stream);
}

int selfgpu_mlp_train_range(const float* features, const float* labels, int n, int epochs, int batch, float lr,
                            unsigned long long seed, float* params, float* lossPerEpoch, float* range, void* stream) {
  if (!features || !labels || n < 1 || epochs < 0 || batch < 1 || batch > (1 << 22) || !(lr > 0.f) || !params)
    return set_error(SELFGPU_ERR_ARG, "selfgpu_mlp_train: bad arguments");
  cudaStream_t st = (cudaStream_t)stream;
  const int tiles = (batch + kTile - 1) / kTile;
  const int blocks = tiles < kMaxGradBlocks ? tiles : kMaxGradBlocks;
  // master and the per-epoch losses, which come back in one copy with the
  // features' range, m1 and m2 (all zeroed), and the blocks' partial sums
  const size_t rangeAt = NP + (size_t)epochs, back = rangeAt + (range ? 2 * IN : 0);
  const size_t scratch = range ? sizeof(RangeScratch) / sizeof(float) : 0;
  const size_t fixed = rangeAt + scratch + 2 * (size_t)NP, total = fixed + (size_t)blocks * (NPP + 1);
  float* buf = nullptr;
  cudaError_t e = cudaMalloc(&buf, total * sizeof(float));
  if (e != cudaSuccess) return fail("selfgpu_mlp_train", e);
  const std::unique_ptr<float[]> host(new (std::nothrow) float[back]);
  if (!host) {
    cudaFree(buf);
    return fail("selfgpu_mlp_train", cudaErrorMemoryAllocation);
  }
  float *master = buf, *loss = buf + NP, *m1 = buf + rangeAt + scratch, *m2 = m1 + NP, *part = buf + fixed,
        *lossPart = part + (size_t)blocks * NPP;
  e = cudaMemsetAsync(buf, 0, fixed * sizeof(float), st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(master, params, NP * sizeof(float), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess && range) {
    k_range<<<kRangeBlocks, kRangeThreads, 0, st>>>(features, n, reinterpret_cast<RangeScratch*>(buf + rangeAt));
    e = cudaGetLastError();
  }
  const long long stepsPerEpoch = ((long long)n + batch - 1) / batch;
  long long t = 0;
  float c1 = 1.f, c2 = 1.f;
  for (int ep = 0; ep < epochs && e == cudaSuccess; ++ep) {
    for (long long s = 0; s < stepsPerEpoch && e == cudaSuccess; ++s, ++t) {
      e = launch_dependent(k_grad, blocks, kGradThreads, st, features, labels, n, master, part, lossPart, seed, t, batch);
      c1 *= 0.9f;
      c2 *= 0.999f;
      if (e == cudaSuccess)
        e = launch_dependent(k_adam, (NP + 31) / 32, 256, st, master, part, lossPart, blocks, m1, m2, loss + ep, lr,
                             1.f - c1, 1.f - c2);
    }
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(host.get(), buf, back * sizeof(float), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  cudaFree(buf);
  if (e != cudaSuccess) return fail("selfgpu_mlp_train", e);
  std::memcpy(params, host.get(), NP * sizeof(float));
  if (lossPerEpoch)
    for (int ep = 0; ep < epochs; ++ep) lossPerEpoch[ep] = host[NP + ep] / (float)(stepsPerEpoch * batch);
  if (range) std::memcpy(range, host.get() + rangeAt, 2 * IN * sizeof(float));
  return SELFGPU_OK;
}

int selfgpu_mlp_infer(const float* features, int n, const uint16_t* weights, const float* params, float* out,
                      void* stream) {
  if (!features || n < 1 || !weights || !params || !out)
    return set_error(SELFGPU_ERR_ARG, "selfgpu_mlp_infer: bad arguments");
  cudaStream_t st = (cudaStream_t)stream;
  MlpArgs args;
  std::memcpy(args.w, weights, sizeof(args.w));
  std::memcpy(args.p, params, sizeof(args.p));
  const long long tiles = ((long long)n + kTile - 1) / kTile;
  k_infer<<<(int)(tiles < 4 * kMaxGradBlocks ? tiles : 4 * kMaxGradBlocks), kGradThreads, 0, st>>>(features, n, args,
                                                                                               out);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return fail("selfgpu_mlp_infer", e);
  return SELFGPU_OK;
}

}  // extern "C"
