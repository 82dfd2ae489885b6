// bruteforce_tc.cuh -- float brute force with the distance filter on the
// tensor cores (tcgen05).
//
// The filter of k_knn_bruteforce, a = |p|^2 - 2 q.p against a threshold with
// an error bound, is a matrix product: D + 1 terms per (query, point) pair.
// Its operands are split into two fp16 halves each (22 bits), the products
// exact and accumulated in fp32, so that a pair's filter value costs a
// handful of tensor-core slots and half an instruction of epilogue -- a
// 3-input minimum over two accumulators -- instead of D FMAs, a minimum and a
// share of a shared-memory read. Groups with a value at or below the
// threshold take the reference's distance and the exact (dist2, index) test,
// so results are those of k_knn_bruteforce, bit for bit.
//
// Bound by the ALU pipe (64 % busy: the minimum, the tests, the waits' polls)
// and the exact tests. A search's ms, k_knn_bruteforce -> here: 100 k x 100 k
// 3-D points, k = 1 2.80 -> 1.15, 5 3.51 -> 1.54, 10 4.81 -> 2.00, 16 7.13 ->
// 2.17, 32 17.3 -> 3.56; 50 k points, 40 k queries in 8-D, k = 5 1.90 -> 0.51;
// 30 k x 30 k in 16-D, k = 10 2.71 -> 0.43; 100 k points, one query 0.18 -> 0.08.
//
// Coordinates enter as x' = s (x - c), with c and the power of 2 s from a
// sample of the points (tc_scale: all but a few of them within 8 of c), each
// as h + l with h and l fp16: |x' - h - l| <= 2^-22 |x'| + 2^-25. Per
// dimension the product takes three slots, (-2 qh) ph + (-2 ql) ph + (-2 qh)
// pl, and |p'|^2 two more against ones. With X = |q'|^2 + P, P >= |p'|^2 for
// the points of a stage (P >= 1/4), the value's error is at most
//   2^-22 X          the dropped ql pl,
//   2^-20 X          the split's and the centring's rounding (the fp16
//                    subnormals' 2^-25 included, P being at least 1/4),
//   (S + 2) 2^-22 X  fp32 accumulation of S slots, every addition taken as
//                    truncated to 2^-23 of the largest partial sum,
// and a reference distance e <= thr has s^2 e within 2^-19 (s^2 thr + X) of
// the exact scaled distance for D <= 16. The threshold's slack is
// 2^-16 (S / 16) (s^2 thr + 2 X): over twice the sum for every S from 16 on.
// (Measured against 64 bits over 2-D to 16-D points: at most 2^-21.3 X.)
//
// The slack grows with P, so P is a stage's own, and a point farther out than
// nearly all the others (|p'|^2 above TcShape::kFar) leaves it: its value is
// minus infinity, below every threshold, so that every query takes its exact
// distance. One far return among a scan's points costs each query one distance
// (with one centre, scale and P for the whole cloud most points passed every
// threshold). A query that the filter cannot hold is searched after the others,
// by its warp without the pipeline.
// (82,762 lidar points and as many queries, k = 5, ms, k_knn_bruteforce / one
// range for the whole cloud / here: the scan 6.39 / 3.95 / 3.05, one return at
// 10 km 6.54 / 17.85 / 3.10, 2 % at 1 km 7.40 / 12.89 / 3.6; 80 k points of a
// Cauchy law 7.46 / 15.25 / 2.73, log-normal 7.45 / 14.85 / 5.54.)
#pragma once

#include <cuda_fp16.h>

#include "internal.cuh"
#include "search.cuh"

namespace nabo_gb300 {

constexpr int kTcQueries = 128;  // per block: the accumulator's rows, one per epilogue thread
constexpr int kTcStages = 3;     // runs of tiles in shared memory
constexpr int kTcThreads = 160;  // four epilogue warps, one that copies and multiplies
constexpr int kTcSeedStride = 8;  // every 8th stage is read first for a starting threshold
constexpr float kTcQueryMax = 32736.0f;  // largest |x'| of a query that the filter holds (-2 x' is an fp16)
constexpr int kTcDrainPolls = 1 << 26;  // for the block's own products and copies, after a wait ran out

// Slots of a record of D dimensions, in whole steps of 16.
template <int D>
struct TcShape {
  static constexpr int kSlots = (3 * D + 2 + 15) / 16 * 16;
  static constexpr int kSteps = kSlots / 16;
  static constexpr float kFar = 128.0f * D;  // all coordinates within 11 of the centre are below
  static constexpr int kRowBytes = kSlots * 2;
  static constexpr size_t operandBytes(int rows) { return (size_t)rows * kRowBytes; }
};

// Points copied at a time: several tiles, so that the copying thread's work
// per tile stays below what the multiplying needs. Their operand is followed
// by their P in 16 bytes, its sign set when some of them are far.
template <int D>
struct TcStage {
  static constexpr int kPoints = D <= 4 ? 256 : 128;
  static constexpr int kBytes = (int)TcShape<D>::operandBytes(kPoints) + 16;
};

// Shared-memory operand layout (K-major, no swizzle): 8 rows by 16 bytes are
// 128 contiguous bytes, the kSlots / 8 such blocks of the same rows one after
// another, the next 8 rows after them.
template <int D>
__host__ __device__ __forceinline__ int64_t tc_offset(int64_t row, int slot8) {
  return ((row >> 3) * (TcShape<D>::kSlots / 8) + slot8) * 128 + (row & 7) * 16;
}

// Writes one row of an operand, its 16-byte blocks through `put(block, uint4)`.
// Queries: -2 q'; points: p' and |p'|^2 (a far point, x = 0: minus infinity).
template <int D, bool QUERY, typename Put>
__device__ __forceinline__ void tc_row(const float (&x)[D], bool far, Put&& put) {
  __half slot[TcShape<D>::kSlots];
#pragma unroll
  for (int i = 0; i < TcShape<D>::kSlots; ++i) slot[i] = __float2half(0.0f);
  float n2 = 0.0f;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const float v = QUERY ? -2.0f * x[d] : x[d];
    const __half h = __float2half_rn(v);
    const __half l = __float2half_rn(v - __half2float(h));
    slot[3 * d] = h;
    slot[3 * d + 1] = QUERY ? l : h;
    slot[3 * d + 2] = QUERY ? h : l;
    n2 = fmaf(x[d], x[d], n2);
  }
  const __half nh = __float2half_rn(n2);
  slot[3 * D] = QUERY ? __float2half(1.0f) : (far ? __ushort_as_half(0xfc00u) : nh);
  slot[3 * D + 1] = QUERY ? __float2half(1.0f) : __float2half_rn(n2 - __half2float(nh));
#pragma unroll
  for (int b = 0; b < TcShape<D>::kSlots / 8; ++b) {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      w[j] = (uint32_t)__half_as_ushort(slot[8 * b + 2 * j]) | (uint32_t)__half_as_ushort(slot[8 * b + 2 * j + 1]) << 16;
    put(b, make_uint4(w[0], w[1], w[2], w[3]));
  }
}

// The points' operand, a block per stage, padded to whole stages (the padding
// is never tested). It depends on the cloud only, so an object holds it from
// its creation and a search needs no scratch for it.
template <int D>
__global__ void __launch_bounds__(TcStage<D>::kPoints)
    k_bf_tc_points(const Rec<float, D>* __restrict__ recs, int64_t n, int dim, TcScale s, unsigned char* out) {
  __shared__ unsigned largest;  // a non-negative float's bits order like its value
  if (threadIdx.x == 0) largest = 0u;
  const int64_t p = blockIdx.x * (int64_t)TcStage<D>::kPoints + threadIdx.x;
  unsigned char* const stage = out + blockIdx.x * (int64_t)TcStage<D>::kBytes;
  float x[D];
#pragma unroll
  for (int d = 0; d < D; ++d) x[d] = 0.0f;
  if (p < n) {
    Rec<float, D> r;
    load_rec(recs, p, r);
#pragma unroll
    for (int d = 0; d < D; ++d) x[d] = d < dim ? (r.p.c[d] - s.centre[d]) * s.scale : 0.0f;
  }
  float n2 = 0.0f;
#pragma unroll
  for (int d = 0; d < D; ++d) n2 = fmaf(x[d], x[d], n2);
  const bool far = !(n2 <= TcShape<D>::kFar);
#pragma unroll
  for (int d = 0; d < D; ++d) x[d] = far ? 0.0f : x[d];
  tc_row<D, false>(x, far, [&](int b, uint4 v) {
    *reinterpret_cast<uint4*>(stage + tc_offset<D>(threadIdx.x, b)) = v;
  });
  const int anyFar = __syncthreads_or(far);
  const unsigned most = __reduce_max_sync(0xffffffffu, __float_as_uint(far ? 0.0f : n2));
  if ((threadIdx.x & 31) == 0) atomicMax(&largest, most);
  __syncthreads();
  if (threadIdx.x == 0) {
    const float P = fmaxf(0.25f, __uint_as_float(largest) * (1.0f + 1e-5f));
    *reinterpret_cast<float4*>(stage + TcStage<D>::kBytes - 16) = make_float4(anyFar ? -P : P, 0.0f, 0.0f, 0.0f);
  }
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Waits for the phase; false after that many polls.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int polls) {
  uint32_t ok;
#pragma unroll 1
  do {
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  } while (!ok && --polls > 0);
  return ok;
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// Descriptor of a K-major operand without swizzle: 128 bytes between the
// 16-byte columns, rowGroupBytes between groups of 8 rows.
__device__ __forceinline__ uint64_t tc_descriptor(uint32_t addr, uint32_t rowGroupBytes) {
  return (uint64_t)((addr >> 4) & 0x3fffu) | (uint64_t)(128u >> 4) << 16 | (uint64_t)(rowGroupBytes >> 4) << 32 |
         (uint64_t)1 << 46;
}
// fp16 x fp16 -> fp32, both operands K-major, M = 128, N points.
constexpr uint32_t tc_instr(int points) {
  return (1u << 4) | ((uint32_t)(points >> 3) << 17) | ((uint32_t)(kTcQueries >> 4) << 24);
}
__device__ __forceinline__ void tc_mma(uint32_t acc, uint64_t a, uint64_t b, uint32_t instr, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(acc),
      "l"(a), "l"(b), "r"(instr), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// 32 accumulator columns of this thread's row; the values are there after
// tc_wait_load (which names them, so that no use moves before it).
__device__ __forceinline__ void tc_load32(uint32_t addr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr)
      : "memory");
}
__device__ __forceinline__ void tc_wait_load(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31]) : : "memory");
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Points per tile (the accumulator's columns) and blocks per SM (two
// accumulators each of the SM's 512 columns) for a compiled list size: long
// lists take the registers of two or three blocks instead of four. One
// accumulator of 128 columns a block, the other blocks working while its
// product runs, beat two of 64 (k = 5 1.55 against 1.81 ms, half the waits a
// point) and one of 256 (1.77 ms).
template <int K>
struct TcTile {
  static constexpr int kPoints = 128;
  static constexpr int kBuffers = K <= 16 ? 1 : 2;
  static constexpr int kBlocksPerSm = K <= 10 ? 4 : K <= 16 ? 3 : 2;
  // groups of the seed pass: a power of 2 above K
  static constexpr int kSlots = K < 4 ? 4 : (K < 8 ? 8 : (K < 16 ? 16 : (K < 32 ? 32 : 64)));
};

template <int D, int K>
struct TcSmem {
  static constexpr int kStagePoints = TcStage<D>::kPoints;
  static constexpr int kTiles = kStagePoints / TcTile<K>::kPoints;
  static constexpr int kA = (int)TcShape<D>::operandBytes(kTcQueries);
  static constexpr int kCopy = TcStage<D>::kBytes;
  static constexpr int kB = (kCopy + 127) / 128 * 128;
  static constexpr int kRecs = kStagePoints * (int)sizeof(Rec<float, D>);
  static constexpr int kBytes = kA + kTcStages * (kB + kRecs);
  // enough that no more blocks share an SM than its accumulators allow
  static constexpr int kLeast = 228 * 1024 / (TcTile<K>::kBlocksPerSm + 1);
  static constexpr int kRequest = kBytes > kLeast ? kBytes : kLeast;
};

// Block (x, y): queries [128 x, 128 x + 128) against points
// [y * chunk, (y + 1) * chunk) (a multiple of the tile), results as
// k_knn_bruteforce writes them. One warp copies the tiles (operand and
// records) and issues the products, a tile ahead of the four warps that read
// the accumulators; thread t of those owns query t. A wait that runs out
// (polls) leaves the pipeline, and the block's queries are then searched
// without it, while the products and copies already issued come to their end:
// they read and write shared memory and accumulators that the next block gets.
//
// Meeting the points in cloud order, a query would insert k ln(n / k) times,
// most of them early, with loose thresholds. So every kTcSeedStride-th tile
// is read once before, only for a starting threshold: the smallest filter
// value of each of kSlots groups of its points (far ones left out). The
// (k + 1)-th smallest of those, brought back to a distance with the filter's slack, is a distance
// that k points other than the query itself reach.
template <int D, int K>
__global__ void __launch_bounds__(kTcThreads, TcTile<K>::kBlocksPerSm)
    k_bf_tc(KnnLaunch a, const unsigned char* __restrict__ operand, TcScale s, int64_t chunk, int64_t partStride,
            int polls) {
  using S = TcSmem<D, K>;
  constexpr int kTcPoints = TcTile<K>::kPoints;
  constexpr int kSlots = TcTile<K>::kSlots;
  constexpr int kParts = kTcPoints / 32;
  constexpr int kBuffers = TcTile<K>::kBuffers;
  constexpr float kSlack = 0x1p-16f * (TcShape<D>::kSlots / 16);
  constexpr int kRowGroup = TcShape<D>::kSlots / 8 * 128;
  extern __shared__ __align__(128) unsigned char tcSmem[];
  __shared__ __align__(8) uint64_t bars[2 * kTcStages + 5];
  __shared__ uint32_t accBase;
  __shared__ int failed, copiedStages, multiplied;  // copies and products issued
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* const smA = tcSmem;
  unsigned char* const smB = tcSmem + S::kA;
  const Rec<float, D>* const smR = reinterpret_cast<const Rec<float, D>*>(tcSmem + S::kA + kTcStages * S::kB);
  const Rec<float, D>* __restrict__ recs = static_cast<const Rec<float, D>*>(a.recs);
  const auto full = [&](int i) { return smem_addr(&bars[i]); };
  const auto empty = [&](int i) { return smem_addr(&bars[kTcStages + i]); };
  const auto accFull = [&](int i) { return smem_addr(&bars[2 * kTcStages + i]); };
  const auto accEmpty = [&](int i) { return smem_addr(&bars[2 * kTcStages + 2 + i]); };
  const auto drained = [&]() { return smem_addr(&bars[2 * kTcStages + 4]); };
  if (warp == 4) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&accBase)),
                 "r"(kBuffers * kTcPoints)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < kTcStages; ++i) {
      mbar_init(full(i), 1);
      mbar_init(empty(i), 4);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(accFull(i), 1);
      mbar_init(accEmpty(i), 4);
    }
    mbar_init(drained(), 1);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const float minDist = a.allowSelf ? -1.0f : Ar<float>::eps();
  const int64_t qi = blockIdx.x * (int64_t)kTcQueries + threadIdx.x;
  const bool active = warp < 4 && qi < a.nq;
  float q[D];
  float maxRadius2 = __builtin_nanf("");  // an idle slot wants nothing
  float qn = 0.0f;
  bool beyond = false;  // the filter cannot hold this query
  TopK<float, K> heap;
  heap.init(a.k);
  if (warp < 4) {
    float x[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      q[d] = active && d < a.dim ? static_cast<const float*>(a.query)[qi * a.qStride + d] : 0.0f;
      x[d] = active && d < a.dim ? (q[d] - s.centre[d]) * s.scale : 0.0f;  // (an idle slot: within the range)
      qn = fmaf(x[d], x[d], qn);
      beyond = beyond || !(fabsf(x[d]) <= kTcQueryMax);
    }
    if (active) {
      maxRadius2 = (float)a.maxRadius2;
      if (a.maxRadii) {
        const float r = static_cast<const float*>(a.maxRadii)[qi];
        maxRadius2 = Ar<float>::mul(r, r);
      }
    }
#pragma unroll
    for (int d = 0; d < D; ++d) x[d] = beyond ? 0.0f : x[d];
    qn = beyond ? 0.0f : qn;
    tc_row<D, true>(x, false, [&](int b, uint4 v) {
      *reinterpret_cast<uint4*>(smA + tc_offset<D>(threadIdx.x, b)) = v;
    });
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t acc = accBase;
  const int64_t first = (int64_t)blockIdx.y * chunk;
  const int64_t last = first + chunk < a.n ? first + chunk : a.n;
  const int stages = (int)((last - first + S::kStagePoints - 1) / S::kStagePoints);
  // stages in the order they are read: the seed's, then all
  const int seeds = stages >= kTcSeedStride ? stages / kTcSeedStride : 0;
  const int total = seeds + stages;
  const auto point_of = [&](int g) {
    return first + (int64_t)(g < seeds ? g * kTcSeedStride : g - seeds) * S::kStagePoints;
  };

  // the radius, and the seed's threshold
  float cap = beyond ? __int_as_float(0x7fffffff) : maxRadius2;
  float thr = bf_threshold(heap.head(), cap);
  // The threshold on the filter's values, s^2 thr - |q'|^2 with the slack for
  // this stage's P: one multiply-add from a query's part and the stage's. A
  // NaN threshold (an idle slot, a NaN radius, a query beyond the filter)
  // passes nothing; an infinite or overflowing one passes everything to the
  // exact test.
  const float queryPart = (2.0f * kSlack - 1.0f) * qn;
  float stagePart = queryPart, thrA = 0.0f;
  const auto set_threshold = [&]() { thrA = fmaf(thr, (1.0f + kSlack) * s.scale2, stagePart); };
  const auto offer = [&](const Rec<float, D>& r) {
    const float d = dist2_seq(q, r);
    if (d <= thr && d <= maxRadius2 && heap.accepts(d, r.p.idx) && d > minDist) {
      heap.insert(d, r.p.idx);
      thr = bf_threshold(heap.head(), cap);
      set_threshold();
    }
  };

  // A stage's P. Its copy has been complete since before its first product,
  // which the caller has read; the wait makes the copy visible to this thread,
  // the records too.
  const auto stage_bound = [&](int st, uint32_t round) {
    mbar_wait(full(st), round, kTcDrainPolls);
    return *reinterpret_cast<const float*>(smB + st * S::kB + S::kCopy - 16);
  };

  bool ok = polls > 0;
  if (warp == 4) {
    if (lane == 0) {
      const auto copy = [&](int g, int st) {
        const int64_t p = point_of(g);
        const int m = last - p < S::kStagePoints ? (int)(last - p) : S::kStagePoints;
        const uint32_t recBytes = (uint32_t)m * sizeof(Rec<float, D>);
        mbar_expect(full(st), S::kCopy + recBytes);
        bulk_load(smem_addr(smB + st * S::kB), operand + p / S::kStagePoints * S::kCopy, S::kCopy, full(st));
        bulk_load(smem_addr(smR + st * S::kStagePoints), recs + p, recBytes, full(st));
      };
      const uint64_t da = tc_descriptor(smem_addr(smA), kRowGroup);
      int copied = 0;
      for (; copied < total && copied < kTcStages; ++copied) copy(copied, copied);
      int st = 0;
      uint32_t round = 0;  // uses of stage st so far, parity
      bool product = false;
      for (int g = 0; g < total && ok; ++g) {
        ok = mbar_wait(full(st), round, polls);
        const uint64_t db = tc_descriptor(smem_addr(smB + st * S::kB), kRowGroup);
#pragma unroll
        for (int i = 0; i < S::kTiles; ++i) {
          const int buf = (g * S::kTiles + i) % kBuffers;
          // the accumulator's previous tile has been read: use n waits for n - 1
          const int use = (g * S::kTiles + i) / kBuffers;
          if (use > 0) ok = ok && mbar_wait(accEmpty(buf), (use - 1) & 1, polls);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int k = 0; k < TcShape<D>::kSteps; ++k)
            tc_mma(acc + buf * kTcPoints, da + k * 16, db + (i * (kTcPoints / 8) * kRowGroup) / 16 + k * 16,
                   tc_instr(kTcPoints), k > 0 ? 1u : 0u);
          tc_commit(accFull(buf));
          product = true;
          // the stage before this one is done with once this one's second tile is due
          if (i == S::kTiles - 1 && g > 0 && copied < total) {
            const int prev = st == 0 ? kTcStages - 1 : st - 1;
            ok = mbar_wait(empty(prev), prev < st ? round : round ^ 1, polls);
            if (ok) copy(copied++, prev);
          }
        }
        if (++st == kTcStages) {
          st = 0;
          round ^= 1;
        }
      }
      if (!ok) failed = 1;
      copiedStages = copied;
      multiplied = product;
    }
    __syncwarp();
  } else {
    const uint32_t row = acc + ((uint32_t)(warp * 32) << 16);
    if (seeds > 0) {
      float slot[kSlots];
#pragma unroll
      for (int g = 0; g < kSlots; ++g) slot[g] = __int_as_float(0x7f800000);
      int st = 0;
      float P = 0.25f;  // of all seeds
      // (a seed's stage is whole: at least kTcSeedStride - 1 more follow it)
      for (int g = 0; g < seeds && ok; ++g) {
        bool far = false;
#pragma unroll 1
        for (int i = 0; i < S::kTiles; ++i) {
          const int buf = (g * S::kTiles + i) % kBuffers;
          ok = ok && mbar_wait(accFull(buf), (g * S::kTiles + i) / kBuffers & 1, polls);
          if (!__all_sync(0xffffffffu, ok)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (i == 0) {
            const float p = stage_bound(st, g / kTcStages & 1);
            far = p < 0.0f;
            P = fmaxf(P, fabsf(p));
          }
#pragma unroll
          for (int part = 0; part < kTcPoints / 32; ++part) {
            uint32_t v[32];
            tc_load32(row + buf * kTcPoints + 32 * part, v);
            tc_wait_load(v);
            if (far) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = v[j] == 0xff800000u ? 0x7f800000u : v[j];
            }
            // value j to slot (32 part + j) % kSlots, two at a time where two
            // of the 32 share a slot
            if constexpr (kSlots >= 32) {
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                const int sl = (32 * part + j) % kSlots;
                slot[sl] = fminf(slot[sl], __uint_as_float(v[j]));
              }
            } else {
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                const int x = j / kSlots * 2 * kSlots + j % kSlots;
                slot[j % kSlots] = min3(slot[j % kSlots], __uint_as_float(v[x]), __uint_as_float(v[x + kSlots]));
              }
            }
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(accEmpty(buf));
        }
        if (lane == 0) mbar_arrive(empty(st));
        st = st + 1 == kTcStages ? 0 : st + 1;
      }
      if (ok) {
        // the (k + 1)-th smallest slot, unless two of them may be the query
        // itself (which a search without self matches does not take)
        int near = 0;
        float bound = __int_as_float(0x7f800000);
        const float selfMax = minDist < 0.0f ? -__int_as_float(0x7f800000)
                                             : (minDist * s.scale2 - qn) + kSlack * (minDist * s.scale2 + 2.0f * (P + qn));
#pragma unroll 1
        for (int i = 0; i < a.k + 1; ++i) {  // take the smallest out, k + 1 times
          bound = slot[0];
#pragma unroll
          for (int g = 1; g < kSlots; ++g) bound = fminf(bound, slot[g]);
          near += bound <= selfMax ? 1 : 0;
          bool out = false;
#pragma unroll
          for (int g = 0; g < kSlots; ++g) {
            const bool hit = !out && slot[g] == bound;
            slot[g] = hit ? __int_as_float(0x7f800000) : slot[g];
            out = out || hit;
          }
        }
        if (near <= 1) {
          // s^2 e <= bound + |q'|^2 + slack, rounded up
          const float e = (bound + qn) + kSlack * (fabsf(bound + qn) + 2.0f * (P + qn));
          const float seed = __fmul_ru(fmaxf(e, 0.0f) * (1.0f + 0x1p-20f), 1.0f / s.scale2);
          if (seed < cap || !(cap == cap)) cap = cap == cap ? seed : cap;
          thr = bf_threshold(heap.head(), cap);
        }
      }
    }
    int st = seeds % kTcStages;
    uint32_t round = (seeds / kTcStages) & 1;
    for (int g = seeds; g < total && ok; ++g) {
      const int64_t p0 = point_of(g);
      const int m = last - p0 < S::kStagePoints ? (int)(last - p0) : S::kStagePoints;
#pragma unroll 1
      for (int i = 0; i < S::kTiles; ++i) {
        const int buf = (g * S::kTiles + i) % kBuffers;
        ok = mbar_wait(accFull(buf), (g * S::kTiles + i) / kBuffers & 1, polls);
        if (!__all_sync(0xffffffffu, ok)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (i == 0) {
          stagePart = fmaf(2.0f * kSlack, fabsf(stage_bound(st, round)), queryPart);
          set_threshold();
          thrA = thr != thr ? -__int_as_float(0x7f800000) : thrA;
        }
        // the columns that pass, 32 at a time, the next ones on their way
        // meanwhile (one copy of the exact test serves all of them: inlined
        // per 32 columns it overflowed the instruction cache)
        unsigned mask[kParts];
        uint32_t w[2][32];
        tc_load32(row + buf * kTcPoints, w[0]);
#pragma unroll
        for (int part = 0; part < kParts; ++part) {
          uint32_t(&v)[32] = w[part & 1];
          tc_wait_load(v);
          if (part + 1 < kParts) {
            tc_load32(row + buf * kTcPoints + 32 * (part + 1), w[(part + 1) & 1]);
          } else {  // the accumulators have been read
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(accEmpty(buf));
          }
          const auto value = [&](int j) { return __uint_as_float(v[j]); };
          float m4[4];
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            m4[q4] = min3(value(8 * q4), value(8 * q4 + 1), value(8 * q4 + 2));
            m4[q4] = min3(m4[q4], value(8 * q4 + 3), value(8 * q4 + 4));
            m4[q4] = min3(m4[q4], value(8 * q4 + 5), value(8 * q4 + 6));
            m4[q4] = fminf(m4[q4], value(8 * q4 + 7));
          }
          const float low = fminf(min3(m4[0], m4[1], m4[2]), m4[3]);
          mask[part] = 0u;
          if (!(low > thrA)) {
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) {
              if (!(m4[q4] > thrA)) {
#pragma unroll
                for (int j = 0; j < 8; ++j) mask[part] |= !(value(8 * q4 + j) > thrA) ? 1u << (8 * q4 + j) : 0u;
              }
            }
          }
        }
        unsigned any = 0u;
#pragma unroll
        for (int part = 0; part < kParts; ++part) {
          const int left = m - i * kTcPoints - part * 32;  // records of this part
          if (left < 32) mask[part] &= left > 0 ? (1u << left) - 1u : 0u;
          any |= mask[part];
        }
        const Rec<float, D>* const tile = smR + st * S::kStagePoints + i * kTcPoints;
        if (any) {
          do {
            int part = 0;
            unsigned bits = mask[0];
#pragma unroll
            for (int x = 1; x < kParts; ++x) {
              if (bits == 0u) {
                bits = mask[x];
                part = x;
              }
            }
            const int j = __ffs(bits) - 1;
            any = 0u;
#pragma unroll
            for (int x = 0; x < kParts; ++x) {
              if (x == part) mask[x] &= mask[x] - 1;
              any |= mask[x];
            }
            offer(tile[part * 32 + j]);
          } while (any);
        }
        __syncwarp();
      }
      if (lane == 0) mbar_arrive(empty(st));
      if (++st == kTcStages) {
        st = 0;
        round ^= 1;
      }
    }
    if (!ok) failed = 1;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (failed && threadIdx.x == 128) {  // the issuing thread: nothing of the block's may outlive it
    if (multiplied) {
      tc_commit(drained());
      mbar_wait(drained(), 0, kTcDrainPolls);
    }
    for (int g = max(copiedStages - kTcStages, 0); g < copiedStages; ++g)
      mbar_wait(full(g % kTcStages), (g / kTcStages) & 1, kTcDrainPolls);
  }
  const bool plain = failed || beyond;
  if (warp < 4 && __any_sync(0xffffffffu, plain)) {
    // without the pipeline: all of the block's queries after a wait ran out,
    // otherwise those beyond the filter. 32 points at a time, a lane loading
    // each, their distances taken before the exact test.
    if (plain) {
      heap.init(a.k);
      cap = maxRadius2;
      thr = bf_threshold(heap.head(), cap);
    }
    for (int64_t base = first; base < last; base += 32) {
      Rec<float, D> mine;
      load_rec(recs, base + lane < last ? base + lane : last - 1, mine);
      unsigned near = 0u;
#pragma unroll 2
      for (int j = 0; j < 32; ++j) {
        Rec<float, D> r;
#pragma unroll
        for (int d = 0; d < D; ++d) r.p.c[d] = __shfl_sync(0xffffffffu, mine.p.c[d], j);
        near |= base + j < last && dist2_seq(q, r) <= thr ? 1u << j : 0u;
      }
      while (plain && near) {
        Rec<float, D> r;
        load_rec(recs, base + __ffs(near) - 1, r);
        near &= near - 1;
        offer(r);
      }
      __syncwarp();
    }
  }
  __syncwarp();
  if (warp == 4)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(acc), "r"(kBuffers * kTcPoints));
  if (active) {
    const int64_t part = (int64_t)blockIdx.y * partStride;
    const int f = heap.store(a.k, a.outIdx + part + qi * a.k, static_cast<float*>(a.outD2) + part + qi * a.k);
    if (a.found) a.found[qi] = f;
  }
}

}  // namespace nabo_gb300
