// Persistent variant of the fused stage kernel.
//
// One CTA per SM, made of C consumer groups of TPE threads (one thread per
// node).  A group works through the CTA's elements g, g + C, g + 2C, ... and
// owns two shared-memory buffers: for every element its thread 0 issues 1-D
// bulk asynchronous copies (cp.async.bulk, the non-tensor TMA path) of the
// element's contiguous blocks -- solution, the engine's packed geometry record
// (dsdx, nHat, nScale, J, sideInfo), its own face traces and the model fields
// -- into a buffer whose mbarrier counts the bytes in, two elements ahead: the
// copies for element jj + 2 go out as soon as element jj has released its
// buffer.  The number of copy requests per element, not their bytes, is what
// costs, so the per-element pieces that live in separate arrays are packed
// into one record at set-up.  The face threads load the neighbours' trace
// values themselves (coalesced plain loads).  With no separate producer warp,
// ten groups of two warps fill the SM's four schedulers with five warps each
// at 96 registers per thread.
//
// Every wait is bounded (StageArgs::waitCycles): on timeout the group records
// an error word, waits (again bounded) for its other copy in flight and
// returns; the host reports SELFGPU_ERR_TIMEOUT.
//
// Requires 16-byte aligned base pointers; the engine falls back to
// k_fused_stage otherwise.  (Tiles of odd P hold an even number of elements,
// so that their pieces are multiples of 16 bytes.)
#pragma once

#include "fused_stage.cuh"

namespace selfgpu {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: true when the phase with this parity has completed.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, long long cycles) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if (clock64() - t0 > cycles) return false;
    __nanosleep(64);
  }
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void named_bar(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// Bounded wait until *p >= v (acquire); false when the budget ran out.
__device__ __forceinline__ bool wait_at_least(const unsigned* p, unsigned v, long long cycles) {
  if (ld_acquire(p) >= v) return true;
  const long long t0 = clock64();
  while (true) {
    if (ld_acquire(p) >= v) return true;
    if (clock64() - t0 > cycles) return false;
    __nanosleep(128);
  }
}

// Runtime layout of one element buffer (byte offsets; -1 = piece absent) and
// of the CTA's shared memory.  Built on the host by make_tma_plan().
struct TmaPlan {
  int groups;      // consumer groups per CTA
  int prefetch;    // fetch each tile's RK register into L2 with its copies
  int slotBytes;   // bytes of one element buffer
  int oQ, oDsdx, oNhat, oNs, oJ, oSi, oOwn;  // oDsdx..oSi lie in the packed geometry record
  int oX[5];       // model fields: LSW (H, Hb, fC), SW (topoB, grad), CIG (envG, drag, presc x3 -> oX[2..4])
  int oVelOwn;
  int oMats, oFlags, oSlots, oGroups, groupBytes, smemBytes;
  int oTasks;
};

// Several RK stages in one launch of k_fused_stage_tma<..., true>: stage s
// (0-based) is RK3 stage s % 3 with the trace and velocity caches of parity
// cur0 + s (vcur0 + s), as selfgpu_model2d's stage-by-stage loop would issue
// them.  Every group runs the same tiles in every stage, so each stage's own
// data (solution, own traces and velocity traces) come from the group itself
// and are copied ahead across the stage boundary.  Only the neighbour traces
// need the other CTAs' stage: a group announces the end of its stage on a
// counter (bar) and, in its next stage, its face warp waits for every
// group's announcement before its first neighbour loads (the copies, the
// flux phase and the divergence sums of that tile go ahead meanwhile).  One
// face warp per tile: P = 8 (one element per group) only.  (Per-tile stage
// flags instead of the one counter, so that no stage waits for the whole
// grid, measured 25-45 % slower: a release fence per tile and an acquire
// load per face thread cost more than the waits they save.)
struct TmaSteps {
  int nStages;
  int nGroups;      // groups of the launch (every one has at least 3 tiles)
  double dt;
  double rkA[3], rkG[3];
  void* tr[2];
  void* vel[2];
  int cur0, vcur0;
  unsigned* bar;    // stage-end counter, zero at launch
};

// Smallest stride >= n values of `bytes` bytes whose byte size is 64 mod 128:
// four consecutive sides then occupy alternate halves of the 32 banks.
__host__ __device__ constexpr int side_stride(int n, int bytes) {
  int k = n;
  while ((k * bytes) % 128 != 64) ++k;
  return k;
}

template <int P, class Phys, typename R>
struct TmaTraits {
  static constexpr int PP = P * P, NV = Phys::NV, NT = Phys::NT, NF = Phys::NF;
  static constexpr int TS = trace_side_stride<P, NT, R>();
  // Elements per group (a tile of consecutive elements).  A P = 4 element
  // (16 nodes) would leave half of its warp's lanes idle: two per one-warp
  // group.  A P = 6 element (36 nodes) on a two-warp group leaves 28 lanes
  // idle: four per five-warp group (144 of 160 lanes), measured 1.14x faster
  // for ShallowWater FP64, 1.12x for CompressibleIdealGas2D FP32 and, with
  // three 128-register groups (below), 1.27x for CompressibleIdealGas2D FP64.
  // Odd P takes an even number of elements, so that every piece of a tile is a
  // multiple of 16 bytes (bulk copies): two at P = 7 and 5 (98 of 128 and 50
  // of 64 lanes live), eight at P = 3 (72 of 96; its 96 face nodes fill the
  // lanes).  On 256x256 meshes, us per stage, against the per-element kernel
  // that ran odd P before: CompressibleIdealGas2D FP64 N = 6 491 -> 195, N = 4
  // 248 -> 123, N = 2 136 -> 65; ShallowWater 364 -> 157, 173 -> 97, 75 -> 46.
  // Four elements at P = 7, four or six at P = 5 and two or four at P = 3
  // measured 1-60 % slower in FP64 CompressibleIdealGas2D.
  static constexpr int EPG = (P == 4) ? 2 : ((P == 6) ? 4 : (P == 3) ? 8 : (P == 5 || P == 7) ? 2 : 1);
  static constexpr int TPE = (EPG * PP + 31) / 32 * 32;  // threads per group
  static_assert(TPE >= EPG * 4 * P, "the face phase gives each of the 4P face nodes its own thread");
  // 640 threads (five warps per scheduler at 96 registers) for P = 6 (ten
  // one-element or four four-element groups) and P = 8; up to 20 single-warp
  // groups for P <= 4 (24 in FP32, at 80 registers: 2-6 % faster than 20),
  // which synchronise with the warp barrier (15 for the
  // FP64 CompressibleIdealGas2D and reference-rounding kernels, whose
  // registers would not fit 20: 16 measured 0.6 % slower, 15 with the warp
  // barrier 0.8 % faster than with named barriers).  Larger groups use
  // named barriers 1..15 (barrier 0 is the CTA-wide one).
  // ShallowWater and CompressibleIdealGas2D FP64 at P = 6 run three
  // four-element groups at 128 registers instead: at 96 they spill (measured
  // 108.5 against 113.5 us per stage for ShallowWater on 256x256;
  // CompressibleIdealGas2D's tiles leave room for three groups only anyway:
  // 144 us, against 183 us with one-element groups).  LinearShallowWater and
  // the FP32 forms are faster with four groups (five, at 72 registers with a
  // few spilled words, measured 12-16 % slower in FP32).  The FP32 forms at P = 8 run
  // fourteen groups (896 threads at 72 registers, no spills): against ten,
  // 7-16 % faster per stage on 256x256 meshes and 6 % on 128x128; fifteen (64
  // registers) measured 1.5-22 % slower than fourteen.  Twelve
  // groups (80 registers) run the production FP64
  // ShallowWater and LinearShallowWater kernels (80 registers without spills;
  // CompressibleIdealGas2D FP64 would spill and its shared memory holds ten
  // groups, the reference-rounding build would spill).
  // Odd P: 512 threads in FP64 (128 registers; at 96 the kernels spill:
  // CompressibleIdealGas2D N = 6 195 against 229 us), 640 for
  // LinearShallowWater at P = 7, which does not spill there (140 against 150),
  // and 768 in FP32 (896 and 640 measured within 4 %).
  static constexpr int kOddThreads =
      sizeof(R) == 4 ? 768 : (P == 7 && NV == 3 && !Phys::kLaggedVelocity) ? 640 : 512;
  static constexpr int kMaxGroups = (P % 2)
      ? (TPE > 32 && kOddThreads / TPE > 15 ? 15 : kOddThreads / TPE)
      : (P <= 4) ? (((NV == 4 && sizeof(R) == 8) || ref_rounding<R>()) ? 15 : (sizeof(R) == 4 ? 24 : 20))
               : (P == 6 ? ((EPG == 4 && (Phys::kLaggedVelocity || NV == 4) && sizeof(R) == 8) ? 3 : 640 / TPE)
                         : ((sizeof(R) == 4) ? 14 : (NV == 3 && !ref_rounding<R>()) ? 12 : 10));
  static constexpr int kThreadsMax = kMaxGroups * TPE;
  // Per-element compute arrays (bulk type), laid out for conflict-free shared
  // accesses.  A 64-bit shared access is served per half-warp: two threads of
  // a half-warp that touch different words of one bank pair (8-byte word
  // index mod 16) cost an extra pass.
  //  * contravariant fluxes [2][NV][P][P]: a half-warp holds rows j and j + 1.
  //  * node fields of the updated solution, read one line per thread by the
  //    trace tasks: field stride FS = 8 (mod 16) and, for P = 8, the column
  //    index XOR-swizzled per (field, row) so that the column lines and the
  //    row lines of two fields fall into distinct bank pairs; other P pad
  //    rows to P + 1.
  //  * boundary-normal flux [4][SS]: sides SS values apart, SS * sizeof(R) =
  //    64 (mod 128).
  // With two elements per group their arrays follow each other (EB values
  // apart), and the divergence sums go to a separate array (NV P^2 per
  // element) instead of replacing the xi flux, since one element's
  // divergence threads may then span two warps.
  static constexpr bool kOdd = (P % 2) != 0;  // rows of an odd length need no padding
  static constexpr bool kSwz = (P == 8);
  static constexpr int RS = (kSwz || kOdd) ? P : P + 1;
  static constexpr int FS = kSwz ? PP + 8 : P * RS;
  // Node fields: over the fluxes, or (kSep) in an array of their own.  Apart,
  // a thread may write its node's fields while others still read the fluxes and
  // its next fluxes while others still form traces, which saves two of a tile's
  // five group barriers; the larger elements leave room for fewer groups.
  // us per stage on 256x256, together -> apart: P = 6 CompressibleIdealGas2D
  // FP64 141 -> 135.5, FP32 113.6 -> 109, reference rounding 150 -> 137,
  // ShallowWater FP64 103 -> 97, LinearShallowWater 94.4 -> 92.7; P = 7 FP32
  // 177 -> 165, reference 280 -> 265, LinearShallowWater FP64 144 -> 134, but
  // production ShallowWater 158 -> 170 and CompressibleIdealGas2D 195 -> 197;
  // P = 5 FP32 102 -> 96, reference 145 -> 137, production FP64 96x96 17.9 ->
  // 19.8; P = 4 FP32 ShallowWater 44.2 -> 42.1, LinearShallowWater 40.0 -> 38.4,
  // CompressibleIdealGas2D 55 -> 58, its reference roundings 95 -> 87.6, the
  // other FP64 forms within 2 %; P = 3 CompressibleIdealGas2D FP32 47.8 -> 45.1,
  // production FP64 119x119 14.3 -> 13.7, the others within 2 %; P = 8 loses
  // more groups than the barriers cost.
  static constexpr bool kProd = sizeof(R) == 8 && !ref_rounding<R>();
  static constexpr bool kSep = P == 6 || (P == 5 && !kProd) ||
                               (P == 7 && (!kProd || (NV == 3 && !Phys::kLaggedVelocity))) ||
                               (P == 4 && (sizeof(R) == 4 ? NV == 3 : NV == 4 && !kProd)) ||
                               (P == 3 && NV == 4 && (kProd || sizeof(R) == 4));
  static constexpr int kU = (!kSep && NT * FS > 2 * NV * PP) ? NT * FS : 2 * NV * PP;
  static constexpr int SS = side_stride(NV * P, (int)sizeof(R));
  static constexpr int EB = kU + 4 * SS + (kSep ? NT * FS : 0);
  static constexpr int oN = kSep ? kU + 4 * SS : 0;  // node fields within an element's arrays
  // Every thread waits for the tile's copies itself (instead of thread 0 for
  // the group): with kSep there is no barrier to wait at, and at P = 4 a
  // one-warp group that one lane waited for ran its lanes apart afterwards
  // (256x256, one -> all: reference rounding CompressibleIdealGas2D 185 -> 95,
  // ShallowWater 125 -> 65, LinearShallowWater 112 -> 60 us; production FP64
  // 74.3 -> 72.9, 54.3 -> 54.0, 47.7 -> 47.6; FP32 CompressibleIdealGas2D
  // 55.0 -> 57.4, so one lane there).
  static constexpr bool kAllWait = kSep || (P == 4 && sizeof(R) == 8);
  static constexpr int kDiv = (EPG > 1 && !kOdd) ? NV * PP : 0;  // separate divergence sums per element
  static constexpr int groupBytes = (int)(((EPG * (EB + kDiv)) * sizeof(R) + 127) / 128 * 128);
  // Weak-divergence volume sums: one thread per 2x2 block of nodes and pair
  // of variables.  The xi flux rows are stored with their value pairs
  // XOR-swizzled per row pair (P/2 a power of two), so that the paired loads
  // of a quarter-warp fall into distinct banks.
  static constexpr int HB = P / 2, NVP = (NV + 1) / 2, NB = HB * HB * NVP;
  static_assert(kOdd || EPG > 1 || NB <= 32, "one element's divergence blocks fit one warp");
  static_assert(kOdd || EPG * NB <= TPE, "every divergence block has its own thread");
  static constexpr bool kSwzF = !kOdd && (HB & (HB - 1)) == 0;
  // position of value m in row j of the xi flux
  __device__ __forceinline__ static int f0pos(int m, int j) {
    if constexpr (kSwzF) return 2 * ((m >> 1) ^ ((j >> 1) & (HB - 1))) + (m & 1);
    else return m;
  }
  // Divergence sums as FP64 tensor-core products: production and FP32-bulk
  // forms at P = 8 and 6 (one element per warp) and 4 (two), production FP64
  // at P = 7 (229 against 257 us per stage with a sum per node; at P = 5 they
  // are slower, 140 against 123)
  static constexpr bool kDmma =
      ((P == 8 && EPG == 1) || P == 6 || (P == 7 && sizeof(R) == 8)) && !ref_rounding<R>();
  static constexpr bool kDmma4 = (P == 4 && EPG == 2 && TPE == 32) && !ref_rounding<R>();
  // odd P otherwise: each node's thread forms its sums in registers, in the
  // reference's order
  // production FP64 at P = 3 and 5: a thread per line of a variable, its sums
  // along the line in registers with the matrix as kernel-parameter constants,
  // written over the line.  A line's P values are read once for its P nodes
  // (10 shared accesses instead of 40 per thread at P = 5, where the L1 pipe ran
  // at 70 %): us per stage on 256x256, a sum per node -> lines, P = 5
  // ShallowWater 98 -> 88, CompressibleIdealGas2D 123 -> 112, LinearShallowWater
  // 81 -> 76; P = 3 46.5 -> 44.7, 64.7 -> 63.5, 39.2 -> 39.0; at P = 7 192
  // against the products' 195, but ShallowWater 184 against 158.
  static constexpr bool kLines = kOdd && kProd && !kDmma;
  static constexpr bool kRegDiv = kOdd && !kDmma && !kLines;
  // At P = 8 the products' operand loads read, per half-warp, four rows of
  // the xi flux, the eta flux and the transposed dgMatrix at four columns
  // each; rows two apart would share banks, so these three arrays keep the
  // column index XOR 4 in row pairs 2-3 and 6-7 (the per-node stores of
  // phase A stay conflict-free, as a half-warp stores two whole rows).
  static constexpr bool kSw8 = (P == 8) && kDmma;
  __device__ __forceinline__ static int cswz(int c, int r) { return kSw8 ? (c ^ (4 * ((r >> 1) & 1))) : c; }
  // positions of F0(m, j), F1(i, j) and dgM(m, i)
  __device__ __forceinline__ static int f0at(int m, int j) { return kSw8 ? P * j + cswz(m, j) : P * j + f0pos(m, j); }
  __device__ __forceinline__ static int f1at(int i, int j) { return kLines ? P * i + j : P * j + cswz(i, j); }
  __device__ __forceinline__ static int dgat(int m, int i) { return P * m + cswz(i, m); }
  // The auxiliaries of the volume flux.  FP32 bulk at odd P forms the full node
  // state, as its per-element kernel does (the compiler contracts the pressure
  // of the shorter form differently, in the last bit).
  // The traced fields of a node's solution f[0..NV).  (ShallowWater's are the
  // solution itself: with the velocities formed and stored along, as the flux
  // needs them, its stages took 1-4 % longer.)
  __device__ __forceinline__ static void trace_fields(R* f, const StageArgs& a) {
    if constexpr (NT > NV) Phys::template node<R>(f, a);
  }
  __device__ __forceinline__ static void flux_fields(R* f, const StageArgs& a) {
    if constexpr (kOdd && sizeof(R) == 4) Phys::template node<R>(f, a);
    else Phys::template node_flux<R>(f, a);
  }
  // Trace tasks of a tile, one per (element, direction, field, line), in rounds
  // of a task per thread.  Where a thread has several, it reads each one's
  // offsets from a table made once per CTA: working them out (divisions by 2 NT
  // P, NT P and P) cost as much as the sums.  us per stage on 256x256, without
  // -> with: CompressibleIdealGas2D P = 6 FP32 109 -> 101.5, FP64 135 -> 129,
  // reference roundings 183 -> 171; P = 4 FP32 54.8 -> 49.4; P = 5 FP32 96.2 ->
  // 89.5; P = 3 FP32 47.8 -> 43.2; P = 7 FP32 165 -> 160; ShallowWater FP32 P =
  // 4 44.2 -> 41.0.  With one round (ShallowWater and LinearShallowWater at P =
  // 5 to 7) the table's load is one more step before the tile's end, 1-7 %
  // slower but for FP32 at P = 7 (134 -> 129), and ShallowWater at P = 3 lost
  // 2-3 % too.
  static constexpr int kTasks = EPG * 2 * NT * P, kRounds = (kTasks + TPE - 1) / TPE;
  static constexpr int kTaskTab = !kSwz && (kRounds > 1 ? !(P == 3 && Phys::kLaggedVelocity) : P == 7 && sizeof(R) == 4)
                                      ? kRounds * TPE
                                      : 0;
  // P = 8: an orientation per warp (tile_traces).  us per stage, tasks in
  // common -> per warp: CompressibleIdealGas2D FP64 128x128 47.7 -> 46.9, 256x256
  // 171.9 -> 170.4, FP32 37.4 -> 36.2 and 128.9 -> 127.3, ShallowWater FP32 32.1
  // -> 31.5; but LinearShallowWater FP64 122.4 -> 124.7, reference roundings 222
  // -> 226, ShallowWater FP64 134.5 -> 135.3.
  static constexpr bool kWarpTraces = kSwz && (sizeof(R) == 4 || (kProd && NV == 4));
  // offset of node (i, j) in field f's block of the node-field array
  __device__ __forceinline__ static int nf(int f, int i, int j) {
    if constexpr (kSwz) return P * j + (i ^ (((j >> 1) ^ (4 * (f & 1))) & (P - 1)));
    else return RS * j + i;
  }
};

// Weak-divergence volume sums of a tile whose contravariant fluxes are in
// shared memory (phase B, alongside the face phase; gBase is the group's array
// of EB values per element), the
// reference's order per node and variable (VectorDGDivergence_2D,
// src/SELF_Lagrange.f90):
//   d = 0;  for m ascending: d = (d + dgM(m,i) F0(m,j)) + dgM(m,j) F1(i,m).
// A thread sums a 2x2 block of nodes for two variables, so every loaded
// flux pair and dgMatrix pair serves two nodes.  One-element groups write
// the sums over the xi flux ([NV][P^2], node-major) once the warp has read
// it; two-element groups write them to their separate array.
// Production FP64 and FP32-bulk forms at P = 8 and P = 6: the same sums
// as FP64 tensor-core products (mma.sync m8n8k4 f64), D(j,i) = sum_m
// F0(m,j) dgM(m,i) + dgM(m,j) F1(i,m), four chained products per variable
// over one warp per element (a P = 6 element is padded with zeros to the
// 8x8 shape; FP32-bulk fluxes are widened exactly to FP64 and the sums
// rounded back once).  The order of the additions inside a product is the
// hardware's, so only the forms without the reference's rounding use it.
// At P = 4 one product covers both elements of a tile: rows and columns
// 0-3 belong to the first element, 4-7 to the second; the xi product's
// A rows and the eta product's B columns carry the element's flux, the
// dgMatrix operand is the same for both, and the two diagonal 4x4 blocks
// of the sum are the two elements' sums (the off-diagonal ones mix the
// elements and are dropped).
template <int P, class Phys, typename R>
__device__ __forceinline__ void tile_volume_sums(R* gBase, const double* sdg, int t, int faceWarp, int nLive,
                                                 const StageArgs& a) {
  using T = TmaTraits<P, Phys, R>;
  constexpr int NV = T::NV, PP = T::PP, EPG = T::EPG, EB = T::EB, TPE = T::TPE;
  if constexpr (T::kLines) {
    constexpr int LE = 2 * NV * P;  // lines of an element: xi lines of the xi flux, eta lines of the eta flux
    for (int k = t; k < EPG * LE; k += TPE) {
      const int eE = k / LE;
      if (eE >= nLive) break;
      R* line = gBase + eE * EB + P * (k - eE * LE);
      R x[P];
#pragma unroll
      for (int m = 0; m < P; ++m) x[m] = line[m];
#pragma unroll
      for (int l = 0; l < P; ++l) {
        R s = a.dgM[P * l] * x[0];  // (kernel-parameter constants)
#pragma unroll
        for (int m = 1; m < P; ++m) s = s + a.dgM[m + P * l] * x[m];
        line[l] = s;
      }
    }
  } else if constexpr (T::kDmma4) {
    const int lane = t & 31, gq = lane >> 2, kq = lane & 3;
    const int eR = gq >> 2, jr = gq & 3;   // the element and node row of this lane's A row / B column
    const R* bU = gBase + eR * EB;
    const R* bF1 = bU + NV * PP;
    const double dg = sdg[T::dgat(kq, jr)];    // dgM(m = kq, jr): B of the xi product, A of the eta product
    // this lane's sums: row gq, columns 2 kq, 2 kq + 1 -> element kq >> 1
    const bool diag = (eR == (kq >> 1)) && eR < nLive;
    R* bD = gBase + EPG * EB + eR * NV * PP;
    using R2 = typename std::conditional<sizeof(R) == 8, double2, float2>::type;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      double c0 = 0.0, c1 = 0.0;
      const double aF0 = (double)bU[v * PP + T::f0at(kq, jr)];  // F0 at (m = kq, j = jr)
      const double bF = (double)bF1[v * PP + T::f1at(jr, kq)];   // F1 at (i = jr, m = kq)
      asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                   : "+d"(c0), "+d"(c1)
                   : "d"(aF0), "d"(dg));
      asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                   : "+d"(c0), "+d"(c1)
                   : "d"(dg), "d"(bF));
      if (diag) {  // D(j = jr, i = 2 (kq & 1)), D(jr, 2 (kq & 1) + 1)
        R2 x;
        x.x = (R)c0;
        x.y = (R)c1;
        reinterpret_cast<R2*>(bD + v * PP + P * jr)[kq & 1] = x;
      }
    }
  } else if constexpr (T::kDmma) {
    // the warps a tile's face threads leave free take its elements in turn
    // (a one-element group: the warp that is not the face warp)
    constexpr int kDW = (EPG == 1) ? 1 : ((TPE - EPG * 4 * P) / 32 > 0 ? (TPE - EPG * 4 * P) / 32 : 1);
    const int w = t >> 5;
    const bool run = (EPG == 1) ? (w != faceWarp) : (w < kDW);
    for (int eB = (EPG == 1) ? 0 : w; run && eB < nLive; eB += kDW) {  // uniform over the warp
      const R* bU = gBase + eB * EB;
      const R* bF1 = bU + NV * PP;
      R* bD = T::kDiv ? gBase + EPG * EB + eB * NV * PP : gBase + eB * EB;
      const int lane = t & 31, gq = lane >> 2, kq = lane & 3;
      double dv[NV][2];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        double c0 = 0.0, c1 = 0.0;
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
          const int m = 4 * kk + kq;
          const bool in = (P == 8) || (gq < P && m < P);  // the zero padding of P = 6
          const double aF0 = in ? (double)bU[v * PP + T::f0at(m, gq)] : 0.0;  // F0 at (m, j = gq)
          const double dg = in ? sdg[T::dgat(m, gq)] : 0.0;                    // dgM(m, gq)
          const double bF = in ? (double)bF1[v * PP + T::f1at(gq, m)] : 0.0;   // F1 at (i = gq, m)
          asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                       : "+d"(c0), "+d"(c1)
                       : "d"(aF0), "d"(dg));
          asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                       : "+d"(c0), "+d"(c1)
                       : "d"(dg), "d"(bF));
        }
        dv[v][0] = c0;  // D(j = gq, i = 2 kq), D(gq, 2 kq + 1)
        dv[v][1] = c1;
      }
      if constexpr (T::kDiv == 0) __syncwarp();  // the warp has read the xi flux it overwrites
      using R2 = typename std::conditional<sizeof(R) == 8, double2, float2>::type;
      if constexpr (T::kOdd) {
        if (gq < P) {
#pragma unroll
          for (int v = 0; v < NV; ++v) {
            if (2 * kq < P) bD[v * PP + P * gq + 2 * kq] = (R)dv[v][0];
            if (2 * kq + 1 < P) bD[v * PP + P * gq + 2 * kq + 1] = (R)dv[v][1];
          }
        }
      } else if (gq < P && 2 * kq + 1 < P) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          R2 x;
          x.x = (R)dv[v][0];
          x.y = (R)dv[v][1];
          reinterpret_cast<R2*>(bD + v * PP + P * gq)[kq] = x;
        }
      }
    }
  } else if constexpr (!T::kRegDiv) {
    const bool mine = (EPG == 1) ? (TPE < 64 || (t >> 5) != faceWarp) : (t < EPG * T::NB);
    if (mine) {
      using R2 = typename std::conditional<sizeof(R) == 8, double2, float2>::type;
      constexpr int HB = T::HB;
      const int eB = (EPG == 1) ? 0 : t / T::NB;
      const int tb = (EPG == 1) ? (t & 31) : t - eB * T::NB;
      const bool on = (EPG == 1) ? (tb < T::NB) : (eB < nLive);
      const R* bU = gBase + eB * EB;
      const R* bF1 = bU + NV * PP;
      R* bD = (EPG > 1) ? gBase + EPG * EB + eB * NV * PP : gBase;
      const int vp = tb / (HB * HB), rem = tb - vp * (HB * HB), bj = rem / HB, bi = rem - bj * HB;
      const int v0 = 2 * vp;
      const bool two = v0 + 1 < NV;
      R acc[2][2][2];  // [variable of the pair][row offset r (j)][column offset c (i)]
#pragma unroll
      for (int vv = 0; vv < 2; ++vv)
#pragma unroll
        for (int r = 0; r < 2; ++r) acc[vv][r][0] = acc[vv][r][1] = (R)0;
      if (on) {
        const double2* sdg2 = reinterpret_cast<const double2*>(sdg);
#pragma unroll
        for (int mp = 0; mp < HB; ++mp) {
          R f0[2][2][2];  // [vv][r][k]: F0(2 mp + k, 2 bj + r)
          R f1[2][2][2];  // [vv][k][c]: F1(2 bi + c, 2 mp + k)
#pragma unroll
          for (int vv = 0; vv < 2; ++vv) {
            const int v = (vv == 0 || two) ? v0 + vv : v0;
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const int row = 2 * bj + r;
              const R2 x = reinterpret_cast<const R2*>(bU + v * PP + P * row)[T::f0pos(2 * mp, row) >> 1];
              f0[vv][r][0] = x.x;
              f0[vv][r][1] = x.y;
            }
#pragma unroll
            for (int kq = 0; kq < 2; ++kq) {
              const R2 x = reinterpret_cast<const R2*>(bF1 + v * PP + P * (2 * mp + kq))[bi];
              f1[vv][kq][0] = x.x;
              f1[vv][kq][1] = x.y;
            }
          }
#pragma unroll
          for (int kq = 0; kq < 2; ++kq) {
            const int m = 2 * mp + kq;
            const double2 dI = sdg2[bi + HB * m], dJ = sdg2[bj + HB * m];
            const R gi[2] = {(R)dI.x, (R)dI.y}, gj[2] = {(R)dJ.x, (R)dJ.y};
#pragma unroll
            for (int vv = 0; vv < 2; ++vv)
#pragma unroll
              for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int c = 0; c < 2; ++c)
                  acc[vv][r][c] = acc[vv][r][c] + gi[c] * f0[vv][r][kq] + gj[r] * f1[vv][kq][c];
          }
        }
      }
      if constexpr (EPG == 1) __syncwarp();  // the warp has read the xi flux it overwrites
      if (on) {
#pragma unroll
        for (int vv = 0; vv < 2; ++vv)
          if (vv == 0 || two)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              R2 x;
              x.x = acc[vv][r][0];
              x.y = acc[vv][r][1];
              reinterpret_cast<R2*>(bD + (v0 + vv) * PP + P * (2 * bj + r))[bi] = x;
            }
      }
    }
  }
}

// End traces of the node fields of a tile of `elems` elements (`live` of them
// real), whose field arrays lie `stride` values apart: BoundaryInterp
// (src/SELF_Lagrange.f90:2241-2270).  One task per (element, field, line,
// orientation) reads the line's P values once and forms both of its end
// traces: column l gives S (side 0) and N (side 2), row l gives W (3) and E
// (1).  This thread takes the tasks k0, k0 + step, ... and passes each result
// to emit(element, field, line, row, lo, hi).  P = 8 numbers the tasks by
// field pair, orientation, field, line (an odd NT leaves the last pair's
// second half idle), so that a half-warp reads the column lines (or the row
// lines) of two fields; the padded layouts of the other P number them by
// orientation, field, line, with no idle tasks.  With kWarp (P = 8) each warp
// has one orientation instead, so that no address depends on the task: fewer
// instructions, but an uneven last round is not shared out.
template <int P, class Phys, typename R, bool kWarp, class Emit>
__device__ __forceinline__ void tile_traces(const R* fields, int stride, int elems, int live, int k0, int step,
                                            const StageArgs& a, Emit emit) {
  using T = TmaTraits<P, Phys, R>;
  constexpr int NT = T::NT;
  if constexpr (kWarp) {
    static_assert(P == 8, "64 threads per element");
    // lane l + 8 f takes line l of fields f, f + 4, ..., whose swizzle is the
    // same, so that a lane's eight offsets serve all its tasks
    const int l = k0 & 7, f0 = (k0 & 31) >> 3;
    const bool row = (k0 >> 5) & 1;
    for (int eE = k0 >> 6; eE < live; eE += step >> 6) {
      const R* fv = fields + eE * stride + f0 * T::FS;
      int at[P];
#pragma unroll
      for (int m = 0; m < P; ++m) at[m] = row ? T::nf(f0, m, l) : T::nf(f0, l, m);
#pragma unroll
      for (int f = 0; f < NT; f += 4) {
        if (f0 + f >= NT) break;
        R lo = (R)0, hi = (R)0;
#pragma unroll
        for (int m = 0; m < P; ++m) {
          const R x = fv[f * T::FS + at[m]];
          lo = lo + bm_left<R>(a, m) * x;  // kernel-parameter constants (m is unrolled)
          hi = hi + bm_right<R, P>(a, m) * x;
        }
        emit(eE, f0 + f, l, row, lo, hi);
      }
    }
  } else {
    constexpr int NTp = T::kSwz ? (NT + 1) / 2 * 2 : NT;
    constexpr int TPEl = 2 * NTp * P;  // tasks per element
    for (int kk = k0; kk < elems * TPEl; kk += step) {
      const int eE = kk / TPEl, ks = kk - eE * TPEl;
      if (eE >= live) continue;
      int row, fi, l;
      if constexpr (T::kSwz) {
        const int fp = ks / (4 * P), r = ks - fp * 4 * P, r2 = r - (r / (2 * P)) * 2 * P, fs = r2 / P;
        row = r / (2 * P);
        l = r2 - fs * P;
        fi = 2 * fp + fs;
        if (fi >= NT) continue;
      } else {
        row = ks / (NT * P);
        const int r = ks - row * NT * P;
        fi = r / P;
        l = r - fi * P;
      }
      const R* fv = fields + eE * stride + fi * T::FS;
      R lo = (R)0, hi = (R)0;
#pragma unroll
      for (int m = 0; m < P; ++m) {
        const R x = fv[row ? T::nf(fi, m, l) : T::nf(fi, l, m)];
        lo = lo + bm_left<R>(a, m) * x;  // kernel-parameter constants (m is unrolled)
        hi = hi + bm_right<R, P>(a, m) * x;
      }
      emit(eE, fi, l, row != 0, lo, hi);
    }
  }
}

// The same from a table of tasks: line's first node (17 bits up), its direction
// (bit 16) and the offset of its value in the tile's trace blocks (16 bits;
// 0xffff: no task).
template <int P, class Phys, typename R>
__device__ __forceinline__ uint32_t trace_task(int k) {
  using T = TmaTraits<P, Phys, R>;
  constexpr int NT = T::NT;
  if (k >= T::kTasks) return 0xffffu;
  const int eE = k / (2 * NT * P), ks = k - eE * 2 * NT * P, row = ks / (NT * P), r = ks - row * NT * P;
  const int fi = r / P, l = r - fi * P;
  const uint32_t src = eE * T::EB + fi * T::FS + (row ? T::RS * l : l);
  return src << 17 | (uint32_t)row << 16 | (uint32_t)(4 * T::TS * eE + l + P * fi);
}
template <int P, class Phys, typename R>
__device__ __forceinline__ void table_traces(const R* fields, const uint32_t* tasks, int live, int t,
                                             const StageArgs& a, R* out) {
  using T = TmaTraits<P, Phys, R>;
  static_assert(T::EPG * T::EB < (1 << 15) && 4 * T::TS * T::EPG < 0xffff, "a task fits its table entry");
#pragma unroll
  for (int r = 0; r < T::kRounds; ++r) {
    const uint32_t k = tasks[r * T::TPE + t];
    const int o = k & 0xffffu;
    if (o >= 4 * T::TS * live) continue;
    const bool row = k & 0x10000u;
    const R* fv = fields + (k >> 17);
    const int step = row ? 1 : T::RS;
    R lo = (R)0, hi = (R)0;
#pragma unroll
    for (int m = 0; m < P; ++m) {
      const R x = fv[m * step];
      lo = lo + bm_left<R>(a, m) * x;  // kernel-parameter constants (m is unrolled)
      hi = hi + bm_right<R, P>(a, m) * x;
    }
    out[o + T::TS * (row ? 3 : 0)] = lo;
    out[o + T::TS * (row ? 1 : 2)] = hi;
  }
}

// PhysCIG::node in FP32 with every product rounded by itself, whatever the
// compiler would contract: the traces of a state set from outside are the
// first stage's input, and a last-bit difference there is visible in the
// solution (2e-9 relative after twelve steps).
__device__ __forceinline__ void cig_fields_rounded(float* f, float gamma) {
  const float r = 1.0f / f[2];
  f[4] = __fmul_rn(f[0], r);
  f[5] = __fmul_rn(f[1], r);
  const float ke = __fmul_rn(0.5f, __fadd_rn(__fmul_rn(f[0], f[4]), __fmul_rn(f[1], f[5])));
  f[6] = __fmul_rn(gamma - 1.0f, __fsub_rn(f[3], ke));
  f[7] = __fadd_rn(f[3], f[6]);
  f[8] = sqrtf(__fmul_rn(__fmul_rn(gamma, f[6]), r));
}

// The trace cache (and, ShallowWater, the lagged velocity traces, which start
// as those of this solution: SetSolution leaves solution%boundary =
// BoundaryInterp(solution)) of a solution set from outside.  Bound by memory:
// the solution read, the traces written.  Blocks of 256 threads, one node per
// thread, with only the node fields in shared memory: 2 048 threads per SM.
// At P = 8 CompressibleIdealGas2D's sums take an orientation per warp (FP32
// 256x256 77.9 -> 71.8 us, FP64 128x128 19.7 -> 18.6; ShallowWater 25.8 -> 26.8).
// Persistent blocks that load the next elements during the sums were slower
// (FP64 128x128 24.7-26.7 us).
template <int P, class Phys, typename R>
struct TraceBlock {
  static constexpr int elems = 256 / (P * P), threads = elems * P * P;
};
template <int P, class Phys, typename R>
__global__ void __launch_bounds__(TraceBlock<P, Phys, R>::threads) k_traces(const StageArgs a) {
  using T = TmaTraits<P, Phys, R>;
  constexpr int NV = T::NV, NT = T::NT, PP = T::PP, TS = T::TS, FS = T::FS;
  constexpr int EPB = TraceBlock<P, Phys, R>::elems, NTH = TraceBlock<P, Phys, R>::threads;
  __shared__ R sm[EPB * NT * FS];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // (the stage kernel waits itself)
  const int t = threadIdx.x, slot = t / PP, n = t - slot * PP;
  const long long e0 = (long long)blockIdx.x * EPB;
  const int live = a.nEl - e0 < EPB ? (int)(a.nEl - e0) : EPB;
  if (slot < live) {
    R f[NT];
#pragma unroll
    for (int v = 0; v < NV; ++v) f[v] = (R)a.q[n + (long long)PP * (v + NV * (e0 + slot))];
    if constexpr (NV == 4 && sizeof(R) == 4) cig_fields_rounded(f, (float)a.gamma);
    else T::trace_fields(f, a);
#pragma unroll
    for (int v = 0; v < NT; ++v) sm[(slot * NT + v) * FS + T::nf(v, n % P, n / P)] = f[v];
  }
  __syncthreads();
  R* trOut = reinterpret_cast<R*>(a.trOut) + (size_t)4 * TS * e0;
  tile_traces<P, Phys, R, P == 8 && NV == 4>(sm, NT * FS, EPB, live, t, NTH, a,
                                             [&](int eE, int fi, int l, bool row, R lo, R hi) {
    R* o = trOut + 4 * TS * eE + l + P * fi;
    o[TS * (row ? 3 : 0)] = lo;
    o[TS * (row ? 1 : 2)] = hi;
  });
  if constexpr (Phys::kLaggedVelocity) {
    __syncthreads();
    R* vOut = reinterpret_cast<R*>(a.velOut) + (size_t)8 * P * e0;
    for (int k = t; k < live * 4 * P; k += NTH) {
      const int es = k / P, ii = k - es * P;  // (element, side)
      const R* o = trOut + TS * es + ii;
      const R H = o[2 * P];
      vOut[2 * P * es + ii] = o[0] / H;
      vOut[2 * P * es + ii + P] = o[P] / H;
    }
  }
}

template <int P, class Phys, typename R>
cudaError_t launch_traces(const StageArgs& a, cudaStream_t st) {
  using B = TraceBlock<P, Phys, R>;
  k_traces<P, Phys, R><<<(a.nEl + B::elems - 1) / B::elems, B::threads, 0, st>>>(a);
  return cudaGetLastError();
}

template <int P, class Phys, typename R, bool kMulti = false>
__global__ void __launch_bounds__(TmaTraits<P, Phys, R>::kThreadsMax, 1)
    k_fused_stage_tma(const StageArgs a, const TmaPlan pl, const TmaSteps ms) {
  using T = TmaTraits<P, Phys, R>;
  constexpr int NV = T::NV, NT = T::NT, NF = T::NF, PP = T::PP, TS = T::TS, TPE = T::TPE, N = P - 1;
  constexpr int FS = T::FS, SS = T::SS, EPG = T::EPG, EB = T::EB;
  constexpr bool kLSW = (NV == 3 && !Phys::kLaggedVelocity);
  constexpr bool kSW = Phys::kLaggedVelocity;
  // Neighbour traces loaded before phase A (measured per configuration: a
  // gain at P = 8 and for ShallowWater FP64 at P = 6; a loss where the
  // registers they hold across phase A make the kernel spill or crowd it --
  // reference-rounding CompressibleIdealGas2D at P = 8, CompressibleIdealGas2D
  // at P = 6, every model at P = 4)
  constexpr bool kNbrEarly =
      (P == 8) ? !(NV == 4 && ref_rounding<R>()) : (P == 6 && kSW && sizeof(R) == 8);
  // The RK register's tile requested into L2 two tiles ahead of its use, so
  // that phase D's loads wait for L2 and not for HBM.  At P = 8 and 6 in the
  // production and FP32-bulk forms, and only where the stage's data exceed L2
  // (us per stage, without -> with: 256x256 CompressibleIdealGas2D P = 8 FP64
  // 175.9 -> 172.5, FP32 133.6 -> 129.4, ShallowWater P = 8 FP32 111.7 ->
  // 105.4, P = 6 FP32 90.5 -> 83.4; on 96x96, where they fit, 1-4 % slower;
  // P = 4 within 1 %; the reference-rounding kernels 3 % slower).  Loading the
  // register into the node threads' registers before the face phase instead was
  // slower (ShallowWater P = 8 FP32 117.6 us).
  constexpr bool kPrefetch = (P == 8 || P == 6) && !ref_rounding<R>();
  auto f0at = [](int m, int j) { return T::f0at(m, j); };
  auto f1at = [](int i, int j) { return T::f1at(i, j); };
  auto dgat = [](int m, int i) { return T::dgat(m, i); };
  extern __shared__ __align__(128) unsigned char smem[];
  const int C = pl.groups;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  double* sdg = reinterpret_cast<double*>(smem + pl.oMats);
  double* sb = sdg + PP;
  double* sqw = sb + 2 * P;
  double* sqwr = sqw + P;  // 1/w (the FP32-bulk and production FP64 forms)
  // bMatrix and 1/w in the bulk type (FP32-bulk form: rounded copies after 1/w)
  R* sbR = sizeof(R) == 8 ? reinterpret_cast<R*>(sb) : reinterpret_cast<R*>(sqwr + P);
  R* sqwrR = sizeof(R) == 8 ? reinterpret_cast<R*>(sqwr) : sbR + 2 * P;
  R* sdgR = sizeof(R) == 8 ? reinterpret_cast<R*>(sdg) : sqwrR + P;  // (kRegDiv)
  volatile int* gflag = reinterpret_cast<volatile int*>(smem + pl.oFlags);
  unsigned char* slots = smem + pl.oSlots;

  if (threadIdx.x == 0) {
    for (int k = 0; k < 2 * C; ++k) mbar_init(&full[k], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // dgMatrix transposed (sdg[i + P m] = dgM(m, i), the column index swizzled
  // where kSw8): a warp's reads of the columns of its nodes' i (or j) are then
  // consecutive
  for (int k = threadIdx.x; k < PP; k += blockDim.x) {
    const double d = a.dgM[k / P + P * (k % P)];
    sdg[dgat(k / P, k % P)] = d;
    if constexpr (T::kRegDiv && sizeof(R) == 4) sdgR[dgat(k / P, k % P)] = (R)d;
  }
  for (int k = threadIdx.x; k < 2 * P; k += blockDim.x) {
    sb[k] = a.bM[k];
    if constexpr (sizeof(R) == 4) sbR[k] = a.bMf[k];
  }
  uint32_t* tasks = reinterpret_cast<uint32_t*>(smem + pl.oTasks);
  for (int k = threadIdx.x; k < T::kTaskTab; k += blockDim.x) tasks[k] = trace_task<P, Phys, R>(k);
  if (T::kAllWait)
    for (int k = threadIdx.x; k < C; k += blockDim.x) gflag[k] = 1;
  for (int k = threadIdx.x; k < P; k += blockDim.x) {
    sqw[k] = a.qw[k];
    sqwr[k] = 1.0 / a.qw[k];
    if constexpr (sizeof(R) == 4) sqwrR[k] = (R)(1.0 / a.qw[k]);
  }
  __syncthreads();
  // Launched as a programmatic dependent of the previous kernel on the stream:
  // let the next launch start its own prologue, then wait until the previous
  // kernel has completed and its writes are visible.  Everything above reads
  // only set-up constants; everything below may read what it wrote or write
  // what it read.  (Both are no-ops for an ordinary launch.)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // Work items are tiles of EPG consecutive elements; the CTA takes tiles
  // blockIdx.x, blockIdx.x + gridDim.x, ...
  const long long nTiles = ((long long)a.nEl + EPG - 1) / EPG;
  const long long nMine =
      (long long)blockIdx.x < nTiles ? (nTiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
  static_assert(!kMulti || EPG == 1, "several stages per launch: one face warp per tile");
  const bool rk = kMulti || (a.mode == MODE_RK);
  const int g = threadIdx.x / TPE;
  const int t = threadIdx.x % TPE;
  if (g >= C) return;
  // work items of group g: its tiles g, g + C, ... of the CTA (nMineG per
  // stage), stage after stage
  const long long nMineG = (long long)g < nMine ? (nMine - g + C - 1) / C : 0;
  const long long nItems = kMulti ? nMineG * ms.nStages : nMineG;
  auto cache_of = [&](void* const* pair, int c0, int st, const void* one) -> const void* {
    return kMulti ? (((c0 + st) & 1) ? pair[1] : pair[0]) : one;  // a stage's input cache (no dynamic index)
  };

  // Group g consumes the CTA's tiles g, g + C, g + 2C, ... through its two
  // buffers; its thread 0 issues the copies of local tile jj + 2 into the
  // buffer that tile jj has just released.  Every piece of a tile is
  // contiguous in global memory (element-major arrays), so a tile is still
  // one bulk copy per piece.
  // the geometry record's kind: FP32 metrics and an FP64 1/J in the FP32-bulk
  // form; FP64 metrics with J (reference roundings), 1/J (production FP64 at
  // P < 8) or no J slot (production FP64 at P = 8, which forms 1/J from dsdx:
  // measured faster there, slower at P = 6)
  constexpr int kGeo = geo_kind<P, R>();
  constexpr GeoRec kRec = geo_rec(P, kGeo);
  const uint32_t qb = NV * PP * 8, gb = kRec.bytes, ob = 4 * TS * sizeof(R);
  const uint32_t vb = kSW ? 8 * P * sizeof(R) : 0;
  uint32_t xb[5] = {0, 0, 0, 0, 0};  // per element
  if constexpr (kLSW) {
    xb[0] = PP * 8;
    xb[1] = 4 * P * 8;
    xb[2] = a.fld[2] ? PP * 8 : 0;
  } else if constexpr (kSW) {
    xb[0] = a.fld[0] ? 4 * P * 8 : 0;
    xb[1] = a.fld[1] ? 2 * PP * 8 : 0;
  } else {
    xb[0] = a.fld[0] ? 2 * PP * 8 : 0;
    xb[1] = a.fld[1] ? (T::kOdd ? 2 : 1) * PP * 8 : 0;
    xb[2] = xb[3] = xb[4] = a.fld[2] ? 16 * P * 8 : 0;
  }
  auto tile_live = [&](long long k) -> int {  // live elements of the CTA's local tile k
    const long long e0 = (blockIdx.x + k * gridDim.x) * EPG;
    const long long r = (long long)a.nEl - e0;
    return r < EPG ? (int)r : EPG;
  };
  // item w = tile jj of stage st (thread 0 only)
  auto issue = [&](long long w, int st, long long jj) {
    if (w >= nItems) return;
    const long long k = g + jj * C;
    const int buf = (int)(w & 1);
    const long long e = (blockIdx.x + k * gridDim.x) * EPG;  // first element of the tile
    const uint32_t nl = (EPG == 1) ? 1u : (uint32_t)tile_live(k);
    unsigned char* sl = slots + (size_t)(2 * g + buf) * pl.slotBytes;
    uint64_t* bar = &full[2 * g + buf];
    // An odd number of elements of odd P (the last tile of a mesh) leaves a
    // piece 8 bytes short of a multiple of 16: this thread then moves the last
    // value itself.
    auto whole = [&](uint32_t n) { return T::kOdd ? n & ~15u : n; };
    auto copy = [&](unsigned char* dst, const void* src, uint32_t n) { bulk_g2s(dst, src, whole(n), bar); };
    if (T::kOdd && (nl & 1)) {  // before the arrival on the barrier, which releases the stores
      auto tail = [&](unsigned char* dst, const double* src, uint32_t n) {
        if (n & 8) *reinterpret_cast<double*>(dst + whole(n)) = src[n / 8 - 1];
      };
      tail(sl + pl.oQ, a.q + (size_t)e * NV * PP, nl * qb);
      if constexpr (kLSW) {
        tail(sl + pl.oX[0], a.fld[0] + (size_t)e * PP, nl * xb[0]);
        if (xb[2]) tail(sl + pl.oX[2], a.fld[2] + (size_t)e * PP, nl * xb[2]);
      }
    }
    uint32_t bytes = nl * (gb + ob + vb) + whole(nl * qb);
#pragma unroll
    for (int x = 0; x < 5; ++x) bytes += whole(nl * xb[x]);
    mbar_arrive_expect_tx(bar, bytes);
    if (a.debugStarve == 1 && blockIdx.x == 0 && k == 0) return;
    const R* trIn = reinterpret_cast<const R*>(cache_of(ms.tr, ms.cur0, st, a.trIn));
    copy(sl + pl.oQ, a.q + (size_t)e * NV * PP, nl * qb);
    if constexpr (kPrefetch)
      if (pl.prefetch && rk) {  // the register, which the node threads load themselves in phase D
        if constexpr (sizeof(R) == 4) prefetch_l2(a.Gf + (size_t)e * NV * PP, nl * NV * PP * 4);
        else prefetch_l2(a.G + (size_t)e * NV * PP, nl * NV * PP * 8);
      }
    bulk_g2s(sl + pl.oDsdx, reinterpret_cast<const unsigned char*>(a.geo) + (size_t)e * gb, nl * gb, bar);
    bulk_g2s(sl + pl.oOwn, trIn + (size_t)4 * TS * e, nl * ob, bar);
    if constexpr (kSW)
      bulk_g2s(sl + pl.oVelOwn,
               reinterpret_cast<const R*>(cache_of(ms.vel, ms.vcur0, st, a.velIn)) + (size_t)e * 8 * P, nl * vb,
               bar);
    if constexpr (kLSW) {
      copy(sl + pl.oX[0], a.fld[0] + (size_t)e * PP, nl * xb[0]);
      bulk_g2s(sl + pl.oX[1], a.fld[1] + (size_t)e * 4 * P, nl * xb[1], bar);
      if (xb[2]) copy(sl + pl.oX[2], a.fld[2] + (size_t)e * PP, nl * xb[2]);
    } else if constexpr (kSW) {
      if (xb[0]) bulk_g2s(sl + pl.oX[0], a.fld[0] + (size_t)e * 4 * P, nl * xb[0], bar);
      if (xb[1]) bulk_g2s(sl + pl.oX[1], a.fld[1] + (size_t)e * 2 * PP, nl * xb[1], bar);
    } else {
      // environmentalsGradient (2,P,P,2,nEl): variable 1, both components, of each element
      if (xb[0])
        for (uint32_t x = 0; x < nl; ++x)
          bulk_g2s(sl + pl.oX[0] + x * xb[0], a.fld[0] + (size_t)(e + x) * 4 * PP, xb[0], bar);
      // environmentals (P,P,2,nEl): variable 2 (drag) of each element; both
      // variables where P is odd (the second alone is not 16-byte aligned)
      if (xb[1] && T::kOdd) bulk_g2s(sl + pl.oX[1], a.fld[1] + (size_t)e * 2 * PP, nl * xb[1], bar);
      else if (xb[1])
        for (uint32_t x = 0; x < nl; ++x)
          bulk_g2s(sl + pl.oX[1] + x * xb[1], a.fld[1] + (size_t)(e + x) * 2 * PP + PP, xb[1], bar);
      if (xb[2])
        for (int x = 2; x < 5; ++x) bulk_g2s(sl + pl.oX[x], a.fld[x] + (size_t)e * 16 * P, nl * xb[x], bar);
    }
  };
  if (t == 0) {
    issue(0, 0, 0);  // (a group has at least three tiles per stage when there are several stages)
    issue(1, 0, 1);
  }

  const int barId = 1 + g;
  // a one-warp group synchronises with the warp barrier (no named-barrier
  // limit on the number of groups); larger groups use named barrier 1 + g
  auto group_bar = [&]() {
    if constexpr (TPE == 32) __syncwarp();
    else named_bar(barId, TPE);
  };
  // node phases: thread t serves node n of element ee of the tile
  const int ee = t / PP;
  const int n = t - ee * PP;
  const int i = n % P, j = n / P;
  // Which warp of a one-element group runs the face phase (the other one sums
  // the divergence meanwhile): alternated in pairs of groups so that both
  // kinds of work spread over the SM's four schedulers (warp w runs on w mod
  // 4).  Two-element groups give the divergence blocks to their first
  // threads and the face nodes to their last ones.
  const int faceWarp = (EPG == 1 && TPE >= 64) ? ((g >> 1) & 1) : 0;
  R* gBase = reinterpret_cast<R*>(smem + pl.oGroups + (size_t)g * pl.groupBytes);
  R* gU = gBase + ee * EB;      // this thread's element: fluxes, later node fields
  R* gN = gU + T::oN;           // node fields
  R* gF1 = gU + NV * PP;        // eta flux [NV][P][P]
  R* gfb = gU + T::kU;          // [4][SS]: [NV][P] per side
  R* gD = T::kDiv ? gBase + EPG * EB + ee * NV * PP : gU;  // divergence sums
  constexpr int rNhat = kRec.oNhat, rNs = kRec.oNs, rJ = kRec.oJ, rSi = kRec.oSi;

  int st = 0;        // stage of item w
  long long jj = -1;  // index of item w's tile among the group's tiles
  for (long long w = 0; w < nItems; ++w) {
    if constexpr (kMulti) {
      if (++jj == nMineG) {
        jj = 0;
        ++st;
      }
    } else {
      jj = w;
    }
    const long long k = g + jj * C;
    // this stage's caches and RK coefficients
    const R* trIn = reinterpret_cast<const R*>(cache_of(ms.tr, ms.cur0, st, a.trIn));
    R* trOut = reinterpret_cast<R*>(const_cast<void*>(cache_of(ms.tr, ms.cur0, st + 1, a.trOut)));
    const R* velIn = reinterpret_cast<const R*>(cache_of(ms.vel, ms.vcur0, st, a.velIn));
    R* velOut = reinterpret_cast<R*>(const_cast<void*>(cache_of(ms.vel, ms.vcur0, st + 1, a.velOut)));
    const int m3 = st % 3;
    const double rkA = kMulti ? (m3 == 0 ? ms.rkA[0] : (m3 == 1 ? ms.rkA[1] : ms.rkA[2])) : a.rk_a;
    const double rkG = kMulti ? (m3 == 0 ? ms.rkG[0] : (m3 == 1 ? ms.rkG[1] : ms.rkG[2])) : a.rk_g;
    const double rkGdt = kMulti ? rkG * ms.dt : a.rk_gdt;
    // the stage's first tile reads other CTAs' traces of the previous stage
    const bool gridWait = kMulti && st > 0 && jj == 0;
    const long long e0 = (blockIdx.x + k * gridDim.x) * EPG;
    const int nLive = (EPG == 1) ? 1 : tile_live(k);
    const long long e = e0 + ee;
    const bool active = (t < EPG * PP) && (ee < nLive);
    const int buf = (int)(w & 1);
    const uint32_t par = (uint32_t)((w >> 1) & 1);
    const unsigned char* sl = slots + (size_t)(2 * g + buf) * pl.slotBytes;
    bool copied = true;  // (kAllWait: as this thread saw it; the group agrees at its next barrier)
    if constexpr (T::kAllWait) {
      copied = mbar_wait(&full[2 * g + buf], par, a.waitCycles);
      if (!copied) gflag[g] = 0;
      if constexpr (!T::kSep) group_bar();
    } else {
      if (t == 0) gflag[g] = mbar_wait(&full[2 * g + buf], par, a.waitCycles) ? 1 : 0;
      group_bar();
    }
    auto give_up = [&]() {
      if (t == 0) {
        if (a.err) atomicExch(a.err, 1);
        // Wait (bounded) once more for this buffer's copies and for those of
        // the group's other buffer, so that none is pending when the CTA exits.
        mbar_wait(&full[2 * g + buf], par, a.waitCycles);
        if (w + 1 < nItems) mbar_wait(&full[2 * g + (buf ^ 1)], (uint32_t)(((w + 1) >> 1) & 1), a.waitCycles);
      }
    };
    if (!T::kSep && !gflag[g]) {
      give_up();
      break;
    }
    const unsigned char* rec = sl + pl.oDsdx + (size_t)ee * gb;  // this thread's element's geometry record
    const double* sq = reinterpret_cast<const double*>(sl + pl.oQ + (size_t)ee * qb);
    // node auxiliaries of this element, read from the buffer where they are used
    auto node_aux = [&](double na[3]) {
      na[0] = na[1] = na[2] = 0.0;
      if constexpr (kLSW) {
        na[0] = reinterpret_cast<const double*>(sl + pl.oX[0] + ee * xb[0])[n];
        if (pl.oX[2] >= 0) na[1] = reinterpret_cast<const double*>(sl + pl.oX[2] + ee * xb[2])[n];
      } else if constexpr (kSW) {
        if (pl.oX[1] >= 0) {
          const double* gg = reinterpret_cast<const double*>(sl + pl.oX[1] + ee * xb[1]);
          na[0] = gg[2 * n];
          na[1] = gg[2 * n + 1];
        }
      } else {
        if (pl.oX[0] >= 0) {
          const double* gg = reinterpret_cast<const double*>(sl + pl.oX[0] + ee * xb[0]);
          na[0] = gg[2 * n];
          na[1] = gg[2 * n + 1];
        }
        if (pl.oX[1] >= 0)
          na[2] = reinterpret_cast<const double*>(sl + pl.oX[1] + ee * xb[1])[n + (T::kOdd ? PP : 0)];
      }
    };

    // Face threads of this tile (phase C): each serves one face node of one
    // element.  Their neighbour traces (and, ShallowWater, the neighbour's
    // lagged velocity traces) are plain global loads; where kNbrEarly they
    // are issued here, before phase A, so that their latency overlaps the
    // flux computation, otherwise at the start of phase C.
    const int c0 = TPE - EPG * 4 * P;  // first face thread of a multi-element group
    const int cf = (EPG == 1) ? (t & 31) : t - c0;
    const int eC = cf / (4 * P);
    const bool faceOn = ((EPG == 1) ? ((t >> 5) == faceWarp && (t & 31) < 4 * P) : (t >= c0)) && eC < nLive;
    const int cc = cf - eC * 4 * P;
    const int s1 = cc / P, ii = cc % P;
    const unsigned char* recC = sl + pl.oDsdx + (size_t)eC * gb;
    const int* ssi = reinterpret_cast<const int*>(recC + rSi) + 5 * s1;
    R X[NT], velR[2] = {(R)0, (R)0};
    auto load_neighbour = [&]() {
      const long long nb =
          (ssi[4] == 0) ? (long long)TS * (ssi[3] / 10 - 1 + 4 * (long long)(ssi[2] - 1)) : -1;
      const int i2 = (ssi[3] % 10) ? N - ii : ii;
      // (several stages in one launch: through L2, as the SM's L1 may still
      // hold these lines from two stages back)
      auto ld = [](const R* x) -> R { return kMulti ? __ldcg(x) : *x; };
      const R* nbr = trIn + (nb < 0 ? 0 : nb);
#pragma unroll
      for (int kf = 0; kf < NT; ++kf) X[kf] = (nb >= 0) ? ld(nbr + i2 + P * kf) : (R)0;
      if constexpr (kSW)
        if (nb >= 0) {
          const R* vn = velIn + (size_t)2 * P * (ssi[3] / 10 - 1 + 4 * (size_t)(ssi[2] - 1));
          velR[0] = ld(vn + i2);
          velR[1] = ld(vn + i2 + P);
        }
    };
    if constexpr (kNbrEarly)
      if (faceOn && !gridWait && copied) load_neighbour();

    // ---- A: flux auxiliaries, contravariant flux.  The buffer stays valid
    // until the end of phase D, so the solution, J and the node auxiliaries
    // are read again where they are needed instead of living in registers
    // across the face phase.
    R f[NF];
    if (active && copied) {
#pragma unroll
      for (int v = 0; v < NV; ++v) f[v] = (R)sq[n + PP * v];
      T::flux_fields(f, a);
      double na[3];
      node_aux(na);
      R Fx[NV], Fy[NV];
      Phys::template flux<R>(f, na, a, Fx, Fy);
      // dsdx planes: (dsdx11, dsdx21) of every node, then (dsdx12, dsdx22)
      R m11, m21, m12, m22;
      if constexpr (kRec.wm == 4) {  // FP32 record: the metric terms already rounded
        const float2* gp = reinterpret_cast<const float2*>(rec);
        const float2 c1 = gp[n], c2 = gp[PP + n];
        m11 = c1.x, m21 = c1.y, m12 = c2.x, m22 = c2.y;
      } else {
        const double2* gp = reinterpret_cast<const double2*>(rec);
        const double2 c1 = gp[n], c2 = gp[PP + n];
        m11 = (R)c1.x, m21 = (R)c1.y, m12 = (R)c2.x, m22 = (R)c2.y;
      }
      R F0[NV], F1[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        F0[v] = m11 * Fx[v] + m21 * Fy[v];
        F1[v] = m12 * Fx[v] + m22 * Fy[v];
      }
      if constexpr (NV == 4)
        if (a.av) av_volume_add<P, R>(a, n, e, F0, F1);
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        gU[v * PP + f0at(i, j)] = F0[v];
        gF1[v * PP + f1at(i, j)] = F1[v];
      }
    }
    group_bar();  // contravariant fluxes ready
    if (T::kSep && !gflag[g]) {
      give_up();
      break;
    }

    // ---- B (alongside the face phase C): weak-divergence volume sums
    if constexpr (T::kRegDiv || T::kLines)
      if (faceOn && !kNbrEarly) load_neighbour();  // in flight during the sums
    tile_volume_sums<P, Phys, R>(gBase, sdg, t, faceWarp, nLive, a);

    // ---- C: faces; own traces of this stage's solution come from the cache,
    // the neighbour's were loaded before phase A
    R dreg[NV];
    if constexpr (T::kRegDiv) {
      if (active) {
#pragma unroll
        for (int v = 0; v < NV; ++v) dreg[v] = (R)0;
#pragma unroll
        for (int m = 0; m < P; ++m) {
          const R gi = sdgR[dgat(m, i)], gj = sdgR[dgat(m, j)];
#pragma unroll
          for (int v = 0; v < NV; ++v)
            dreg[v] = dreg[v] + gi * gU[v * PP + f0at(m, j)] + gj * gF1[v * PP + f1at(i, m)];
        }
      }
    }
    {
      if (faceOn) {
        if (gridWait) {
          // every group has ended the previous stage (its traces are final):
          // the face warp waits alone, the divergence warp goes on meanwhile
          if ((t & 31) == 0 && !wait_at_least(ms.bar, (unsigned)st * (unsigned)ms.nGroups, a.waitCycles))
            gflag[g] = 0;  // checked after phase C
          __syncwarp();
        }
        if ((!kNbrEarly && !T::kRegDiv && !T::kLines) || gridWait) load_neighbour();
        const long long eF = e0 + eC;
        const int bcid = ssi[4];
        const bool physical = (bcid != 0) && (ssi[2] == 0);
        const R* own = reinterpret_cast<const R*>(sl + pl.oOwn + (size_t)eC * ob) + s1 * TS;
        R L[NT];
#pragma unroll
        for (int kf = 0; kf < NT; ++kf) L[kf] = own[ii + P * kf];
        double2 nh;  // the face functions round the normal to R first: FP32 records hold it rounded
        double ns;
        if constexpr (kRec.wm == 4) {
          const float2 nf = reinterpret_cast<const float2*>(recC + rNhat)[ii + P * s1];
          nh = make_double2(nf.x, nf.y);
          ns = reinterpret_cast<const float*>(recC + rNs)[ii + P * s1];
        } else {
          nh = reinterpret_cast<const double2*>(recC + rNhat)[ii + P * s1];
          ns = reinterpret_cast<const double*>(recC + rNs)[ii + P * s1];
        }
        double fx[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        if constexpr (kLSW) {
          fx[0] = reinterpret_cast<const double*>(sl + pl.oX[1] + eC * xb[1])[ii + P * s1];
        } else if constexpr (kSW) {
          if (physical && pl.oX[0] >= 0)
            fx[0] = reinterpret_cast<const double*>(sl + pl.oX[0] + eC * xb[0])[ii + P * s1];
        } else {
          if (physical && pl.oX[2] >= 0) {
            const double* ps = reinterpret_cast<const double*>(sl + pl.oX[2] + eC * xb[2]);
            const double* pp = reinterpret_cast<const double*>(sl + pl.oX[3] + eC * xb[3]);
            const double* pd = reinterpret_cast<const double*>(sl + pl.oX[4] + eC * xb[4]);
            const int b = ii + P * 4 * s1;
            for (int v = 0; v < 4; ++v) fx[v] = ps[b + v * P];
            fx[4] = pp[b];
            fx[5] = pp[b + P];
            fx[6] = pp[b + 3 * P];
            fx[7] = pd[b + P];
            fx[8] = pd[b + 2 * P];
          }
        }
        R velL[2] = {(R)0, (R)0};
        if constexpr (kSW) {
          const R* vo = reinterpret_cast<const R*>(sl + pl.oVelOwn + (size_t)eC * vb);
          velL[0] = vo[ii + P * (0 + 2 * s1)];
          velL[1] = vo[ii + P * (1 + 2 * s1)];
          R* vOut = velOut;
          if constexpr (ref_rounding<R>() || (T::kOdd && sizeof(R) == 4)) {
            vOut[ii + P * (0 + 2 * (s1 + 4 * eF))] = L[0] / L[2];
            vOut[ii + P * (1 + 2 * (s1 + 4 * eF))] = L[1] / L[2];
          } else {
            const R rH = (R)1 / L[2];
            vOut[ii + P * (0 + 2 * (s1 + 4 * eF))] = L[0] * rH;
            vOut[ii + P * (1 + 2 * (s1 + 4 * eF))] = L[1] * rH;
          }
        }
        R out[NV];
        Phys::template face<R>(bcid, physical, L, X, velL, velR, nh.x, nh.y, ns, fx,
                               Phys::template face_constants<R>(fx, a), a, out);
        if constexpr (NV == 4)
          if (a.av) av_face_add<P, R>(a, s1, ii, eF, ssi, nh.x, nh.y, ns, out);
        R* fb = gBase + eC * EB + T::kU;
#pragma unroll
        for (int v = 0; v < NV; ++v) fb[s1 * SS + v * P + ii] = out[v];
      }
    }
    group_bar();  // flux and face values ready
    if (gridWait && !gflag[g]) {  // the stage-end wait ran out
      if (t == 0) {
        if (a.err) atomicExch(a.err, 1);
        if (w + 1 < nItems) mbar_wait(&full[2 * g + (buf ^ 1)], (uint32_t)(((w + 1) >> 1) & 1), a.waitCycles);
      }
      break;
    }

    // ---- D: weak divergence + lift, 1/J, source, RK update
    double dsdt[NV], qv[NV], Gv[NV];
    if (active) {
      if (rk) {  // RK register from global memory; the lift below hides the latency
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          const size_t gi = n + (size_t)PP * (v + NV * (size_t)e);
          Gv[v] = sizeof(R) == 4 ? (double)a.Gf[gi] : a.G[gi];  // FP32-bulk form: an FP32 register
        }
      }
#pragma unroll
      for (int v = 0; v < NV; ++v) qv[v] = sq[n + PP * v];
      // J of the node (reference-rounding build) or 1/J (the other forms:
      // from the record, or for production FP64 at P = 8 the reciprocal of
      // det(dsdx) = J)
      double Jij;
      if constexpr (kGeo != GEO_NOJ) {
        Jij = reinterpret_cast<const double*>(rec + rJ)[n];
      } else {
        const double2* gp = reinterpret_cast<const double2*>(rec);
        const double2 c1 = gp[n], c2 = gp[PP + n];
        Jij = 1.0 / (c1.x * c2.y - c2.x * c1.y);
      }
      // sources in FP64 in every form (well-balanced topography / gravity terms)
      double Src[NV], na[3];
      node_aux(na);
      Phys::template source<double>(qv, na, a, Src);
      R d[NV];  // volume sums from phase B
#pragma unroll
      for (int v = 0; v < NV; ++v) d[v] = T::kRegDiv ? dreg[v] : T::kLines ? gU[v * PP + n] + gF1[v * PP + f1at(i, j)] : gD[v * PP + n];
      if constexpr (ref_rounding<R>()) {
        // the reference's divisions, rounded as it rounds them (bit-exact form)
        const R wi = (R)sqw[i], wj = (R)sqw[j];
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          const R dv = d[v] + ((R)sb[i + P] * gfb[1 * SS + v * P + j] + (R)sb[i] * gfb[3 * SS + v * P + j]) / wi +
                       ((R)sb[j + P] * gfb[2 * SS + v * P + i] + (R)sb[j] * gfb[0 * SS + v * P + i]) / wj;
          dsdt[v] = Src[v] - (double)dv / Jij;
        }
      } else {
        // FP32 bulk and production FP64: products with the reciprocals of the
        // weights, and by 1/J
        const R rwi = sqwrR[i], rwj = sqwrR[j];
        const R bi0 = sbR[i], bi1 = sbR[i + P], bj0 = sbR[j], bj1 = sbR[j + P];
        const double rJ = Jij;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          const R dv = d[v] + (bi1 * gfb[1 * SS + v * P + j] + bi0 * gfb[3 * SS + v * P + j]) * rwi +
                       (bj1 * gfb[2 * SS + v * P + i] + bj0 * gfb[0 * SS + v * P + i]) * rwj;
          dsdt[v] = fma(-(double)dv, rJ, Src[v]);  // (explicit: Src may be a product too)
        }
      }
    }
    auto refill = [&]() {  // the buffer: generic-proxy reads before the async-proxy writes
      if (t != 0) return;
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      if (!kMulti || jj + 2 < nMineG) issue(w + 2, st, jj + 2);
      else issue(w + 2, st + 1, jj + 2 - nMineG);
    };
    if (!T::kSep || !rk) {
      group_bar();  // every thread is done reading the flux arrays and the buffer
      refill();
    }
    if (!rk) {
      if (active)
#pragma unroll
        for (int v = 0; v < NV; ++v) a.dSdt[n + (size_t)PP * (v + NV * (size_t)e)] = dsdt[v];
      continue;
    }
    if (active) {
      const double gdt = a.dtElem ? rkG * a.dtElem[e] : rkGdt;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const size_t gi = n + (size_t)PP * (v + NV * (size_t)e);
        const double Gn = rkA * Gv[v] + dsdt[v];
        if constexpr (sizeof(R) == 4) a.Gf[gi] = (float)Gn;  // the solution update uses the FP64 value
        else a.G[gi] = Gn;
        const double qn = qv[v] + gdt * Gn;
        a.q[gi] = qn;
        f[v] = (R)qn;
      }
      T::trace_fields(f, a);
#pragma unroll
      for (int v = 0; v < NT; ++v) gN[v * FS + T::nf(v, i, j)] = f[v];
    }
    group_bar();
    if constexpr (T::kSep) refill();

    // ---- E: traces of the updated solution -> trace cache.  (Without kWarp a
    // one-element group's face warp starts one warp later, so the other warp
    // takes the last, partial round.)
    if constexpr (T::kTaskTab > 0) {
      table_traces<P, Phys, R>(gBase + T::oN, tasks, nLive, t, a, trOut + (size_t)4 * TS * e0);
    } else {
      const int k0 = (EPG == 1 && !T::kWarpTraces) ? (faceWarp ? t : (t + 32) % TPE) : t;
      tile_traces<P, Phys, R, T::kWarpTraces>(gBase + T::oN, EB, EPG, nLive, k0, TPE, a,
                                              [&](int eE, int fi, int l, bool row, R lo, R hi) {
        R* o = trOut + (size_t)4 * TS * (e0 + eE);
        o[l + P * fi + TS * (row ? 3 : 0)] = lo;
        o[l + P * fi + TS * (row ? 1 : 2)] = hi;
      });
    }
    // no barrier here: the next tile's post-wait barrier orders the reuse of the arrays
    if constexpr (kMulti) {
      // This tile's solution, traces and velocity traces are read again by
      // bulk copies (async proxy) in the next stage: the copies of tiles 0
      // and 1 go out during this stage's last two tiles, the others during
      // the next stage, so a proxy fence after tiles 0, 1 and the last one
      // orders every write before the copy that reads it.
      if (jj <= 1 || jj == nMineG - 1) asm volatile("fence.proxy.async.global;" ::: "memory");
      if (jj == nMineG - 1 && st + 1 < ms.nStages) {  // the group's stage ends: announce it
        group_bar();
        if (t == 0 && !(a.debugStarve == 2 && blockIdx.x == 0 && g == 0)) {
          __threadfence();
          atomicAdd(ms.bar, 1u);
        }
      }
    }
  }
}

// Host-side plan for k_fused_stage_tma given the smem budget.
template <int P, class Phys, typename R>
inline bool make_tma_plan(const StageArgs& a, int smemLimit, long long l2Bytes, TmaPlan& pl, int maxGroups = 0) {
  using T = TmaTraits<P, Phys, R>;
  constexpr int PP = T::PP, NV = T::NV, TS = T::TS, EPG = T::EPG;
  constexpr bool kLSW = (NV == 3 && !Phys::kLaggedVelocity);
  constexpr bool kSW = Phys::kLaggedVelocity;
  int o = 0;
  auto put = [&](int bytes) {  // one piece of a tile: EPG elements' blocks back to back
    int at = o;
    o += (EPG * bytes + 15) / 16 * 16;
    return at;
  };
  if (!a.geo) return false;
  pl.oQ = put(NV * PP * 8);
  constexpr GeoRec gr = geo_rec(P, geo_kind<P, R>());
  pl.oDsdx = put(gr.bytes);  // records: dsdx, nHat, nScale, [J or 1/J,] sideInfo
  pl.oNhat = pl.oDsdx + gr.oNhat;  // (offsets within the first element's record)
  pl.oNs = pl.oDsdx + gr.oNs;
  pl.oJ = pl.oDsdx + gr.oJ;
  pl.oSi = pl.oDsdx + gr.oSi;
  pl.oOwn = put(4 * TS * (int)sizeof(R));
  for (int x = 0; x < 5; ++x) pl.oX[x] = -1;
  pl.oVelOwn = -1;
  if (kLSW) {
    pl.oX[0] = put(PP * 8);
    pl.oX[1] = put(4 * P * 8);
    if (a.fld[2]) pl.oX[2] = put(PP * 8);
  } else if (kSW) {
    if (a.fld[0]) pl.oX[0] = put(4 * P * 8);
    if (a.fld[1]) pl.oX[1] = put(2 * PP * 8);
    pl.oVelOwn = put(8 * P * (int)sizeof(R));
  } else {
    if (a.fld[0]) pl.oX[0] = put(2 * PP * 8);
    if (a.fld[1]) pl.oX[1] = put((P % 2 ? 2 : 1) * PP * 8);
    if (a.fld[2])
      for (int x = 2; x < 5; ++x) pl.oX[x] = put(16 * P * 8);
  }
  // one stage's data: the tiles' copies, the register, and the traces written
  pl.prefetch =
      (long long)a.nEl * (o / EPG + NV * PP * (int)sizeof(R) + 4 * TS * (int)sizeof(R)) > l2Bytes ? 1 : 0;
  pl.slotBytes = (o + 127) / 128 * 128;
  pl.groupBytes = T::groupBytes;
  const int cMax = (maxGroups > 0 && maxGroups < T::kMaxGroups) ? maxGroups : T::kMaxGroups;
  for (int C = cMax; C >= 1; --C) {
    int s = 0;
    s += 2 * C * 8;  // barriers
    s = (s + 15) / 16 * 16;
    const int oMats = s;
    s += (PP + 4 * P) * 8;  // dgMatrix, bMatrix, weights, reciprocal weights
    if (sizeof(R) == 4) s += ((3 * P + (T::kRegDiv ? PP : 0)) * 4 + 15) / 16 * 16;  // their FP32 copies
    const int oTasks = s;
    s += T::kTaskTab * 4;
    const int oFlags = s;
    s += C * 4;  // group flags
    s = (s + 127) / 128 * 128;
    const int oSlots = s;
    s += 2 * C * pl.slotBytes;
    const int oGroups = s;
    s += C * pl.groupBytes;
    if (s <= smemLimit) {
      pl.groups = C;
      pl.oMats = oMats;
      pl.oTasks = oTasks;
      pl.oFlags = oFlags;
      pl.oSlots = oSlots;
      pl.oGroups = oGroups;
      pl.smemBytes = s;
      return true;
    }
  }
  return false;
}

}  // namespace selfgpu
