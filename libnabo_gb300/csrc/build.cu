// build.cu -- kd-tree construction on the device.
//
// Produces exactly the tree of the reference constructor
// KDTreeUnbalancedPtInLeavesImplicitBoundsStackOpt (nabo/kdtree_cpu.cpp:
// 109-272): sliding-midpoint split on the widest box dimension, cut clamped
// to the points' range, the two-pass in-place partition, the same leftCount
// rules, pre-order node numbering with the left child at n+1, and leaf
// buckets in the same point order. Points are stored in leaf order as
// 16-byte-aligned records, so a bucket is a contiguous run.
//
// Phases:
//   1. pack + bounds: records in cloud order, per-dimension min/max.
//   2. top levels, all segments of a level at once: the reference's rule in
//      one cooperative launch (k_top), the median rule as a stable scatter per
//      level (k_median_*), down to segments that fit in a block's shared
//      memory.
//   3. small segments: a block each (or several at once) splits its points in
//      shared memory down to leaves (k_mid).
//   4. numbering: splits and leaves are recorded by position; a count of the
//      leaves before each position gives every node its pre-order index
//      (k_leaf_ranks, k_emit).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <vector>

#include "internal.cuh"

namespace nabo_gb300 {
namespace {

constexpr int kBlock = 256;
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ int2 add2(int2 a, int2 b) { return make_int2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ uint32_t shfl_up(uint32_t v, int o) { return __shfl_up_sync(kFull, v, o); }
__device__ __forceinline__ unsigned long long shfl_up(unsigned long long v, int o) {
  return __shfl_up_sync(kFull, v, o);
}
__device__ __forceinline__ int2 shfl_up(int2 v, int o) {
  return make_int2(__shfl_up_sync(kFull, v.x, o), __shfl_up_sync(kFull, v.y, o));
}

struct MinOp {
  template <typename V>
  __device__ V operator()(V a, V b) const { return a < b ? a : b; }
};
struct MaxOp {
  template <typename V>
  __device__ V operator()(V a, V b) const { return a > b ? a : b; }
};
// Reduction over runs of equal segment id inside a warp (segments are
// contiguous position ranges, so equal ids form one run). Returns the run's
// reduction in the run's last lane (`tail`).
template <typename V, typename Op>
__device__ __forceinline__ V seg_warp_reduce(int s, V v, Op op, bool* tail) {
  const int lane = threadIdx.x & 31;
  const int prev = __shfl_up_sync(kFull, s, 1);
  const bool head = (lane == 0) || (prev != s);
  const unsigned heads = __ballot_sync(kFull, head);
  const unsigned upto = heads & (kFull >> (31 - lane));
  const int runStart = 31 - __clz(upto);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const V y = shfl_up(v, o);
    if (lane - o >= runStart) v = op(v, y);
  }
  *tail = (lane == 31) || ((heads >> (lane + 1)) & 1u);
  return v;
}

__device__ __forceinline__ int2 warp_incl_scan(int2 v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int2 y = shfl_up(v, o);
    if (lane >= o) v = add2(v, y);
  }
  return v;
}

// Exclusive scan over a block of kBlock threads.
__device__ __forceinline__ int2 block_excl_scan(int2 v, int2* total) {
  __shared__ int2 sw[kBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int2 inc = warp_incl_scan(v, lane);
  if (lane == 31) sw[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int2 w = lane < kBlock / 32 ? sw[lane] : make_int2(0, 0);
    w = warp_incl_scan(w, lane);
    if (lane < kBlock / 32) sw[lane] = w;
  }
  __syncthreads();
  const int2 wpre = warp > 0 ? sw[warp - 1] : make_int2(0, 0);
  *total = sw[kBlock / 32 - 1];
  __syncthreads();
  return add2(wpre, make_int2(inc.x - v.x, inc.y - v.y));
}

// ---------------------------------------------------------------------------
// Phase 1: packing and bounds.

template <typename T, int D>
__global__ void k_pack(const T* __restrict__ cloud, int64_t n, int64_t stride, int dim, Rec<T, D>* __restrict__ recs) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= n) return;
  Rec<T, D> r;
#pragma unroll
  for (int c = 0; c < RecSize<T, D>::chunks; ++c) r.v[c] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int d = 0; d < D; ++d) r.p.c[d] = d < dim ? cloud[p * stride + d] : T(0);
  r.p.idx = (int32_t)p;
  recs[p] = r;
}

template <typename K>
__device__ __forceinline__ K warp_min(K v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const K y = __shfl_xor_sync(kFull, v, o);
    v = y < v ? y : v;
  }
  return v;
}
template <typename K>
__device__ __forceinline__ K warp_max(K v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const K y = __shfl_xor_sync(kFull, v, o);
    v = y > v ? y : v;
  }
  return v;
}

template <typename T, int D>
__global__ void k_bounds(const Rec<T, D>* __restrict__ recs, int64_t n, int dim, typename KeyOf<T>::type* mnK,
                         typename KeyOf<T>::type* mxK, int* nonFinite) {
  using Key = typename KeyOf<T>::type;
  Key mn[D], mx[D];
  int bad = 0;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    mn[d] = ordered_key(Ar<T>::inf());
    mx[d] = ordered_key(-Ar<T>::inf());
  }
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
    Rec<T, D> r;
    load_rec(recs, p, r);
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const Key k = ordered_key(r.p.c[d]);
      mn[d] = k < mn[d] ? k : mn[d];
      mx[d] = k > mx[d] ? k : mx[d];
      bad |= (d < dim && !isfinite(r.p.c[d])) ? 1 : 0;
    }
  }
  if (__any_sync(kFull, bad) && (threadIdx.x & 31) == 0) atomicOr(nonFinite, 1);
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const Key a = warp_min(mn[d]);
    const Key b = warp_max(mx[d]);
    if ((threadIdx.x & 31) == 0 && d < dim) {
      atomicMin(mnK + d, a);
      atomicMax(mxK + d, b);
    }
  }
}

// What a packed cloud's creation reads back, in one copy: the bounds' keys, a
// flag for non-finite points, and a few points of a float cloud, evenly spread
// but at irregular positions (a scan repeats itself every so many points).
constexpr int kSamplePoints = 256;
template <typename T, int D>
struct CloudStats {
  typename KeyOf<T>::type mn[kMaxDim], mx[kMaxDim];
  int nonFinite;
  T sample[sizeof(T) == 4 ? kSamplePoints : 1][D];
};
template <typename T, int D>
__global__ void k_init_stats(CloudStats<T, D>* s, const Rec<T, D>* __restrict__ recs, int64_t n) {
  const int i = threadIdx.x;
  if (i < kMaxDim) {
    s->mn[i] = ordered_key(Ar<T>::inf());
    s->mx[i] = ordered_key(-Ar<T>::inf());
  }
  if (i == 0) s->nonFinite = 0;
  if constexpr (sizeof(T) == 4) {
    const int64_t first = n * i / kSamplePoints, width = n * (i + 1) / kSamplePoints - first;
    int64_t p = first + (width > 0 ? (int64_t)((uint32_t)i * 2654435761u) % width : 0);
    p = p < n ? p : n - 1;
#pragma unroll
    for (int d = 0; d < D; ++d) s->sample[i][d] = recs[p].p.c[d];
  }
}

__device__ __forceinline__ float next_up(float x) { return nextafterf(x, __builtin_huge_valf()); }
__device__ __forceinline__ double next_up(double x) { return nextafter(x, __builtin_huge_val()); }

// Ascending bitonic sort of 32 R keys held R per lane (element lane + 32 r),
// across the warp: partners at distance below 32 are exchanged by shuffle,
// at 32 inside the lane.
template <int R, typename Key>
__device__ __forceinline__ void warp_sort_keys(Key (&e)[R], int lane) {
#pragma unroll
  for (int k2 = 2; k2 <= 32 * R; k2 <<= 1) {
#pragma unroll
    for (int j = k2 >> 1; j > 0; j >>= 1) {
      Key o[R];
#pragma unroll
      for (int r = 0; r < R; ++r) o[r] = j >= 32 ? e[r ^ (j >> 5)] : __shfl_xor_sync(0xffffffffu, e[r], j);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int i = lane + 32 * r;
        const bool keepMin = ((i & j) == 0) == ((i & k2) == 0);
        e[r] = keepMin ? (o[r] < e[r] ? o[r] : e[r]) : (o[r] > e[r] ? o[r] : e[r]);
      }
    }
  }
}

constexpr int kMedianSamples = 31;

}  // namespace
}  // namespace nabo_gb300

#include "build_tree.cuh"

namespace nabo_gb300 {
namespace {

// ---------------------------------------------------------------------------
// Phase 2: top levels of the median rule.

template <typename T>
struct SegLevel {
  int* start;
  int* count;
  int* turns;
  T* boxLo;  // [cap * kMaxDim]
  T* boxHi;
  int* cutDim;
  T* cut;
  int* mode;  // cut above the median, at it, or by position (k_median_split)
  int* lt;
  int* leftCount;
  int* newLeft;
  int* newRight;
};

// Level bookkeeping kept on the device, so a fixed number of levels can run
// without reading anything back (graph capture) and the host-driven loop
// reads only `nseg` after each level.
struct LevelState {
  int nseg;      // segments of the current level
  int level;     // current level
};

// argMax of the box extents (nabo/kdtree_cpu.cpp:76-90): first strict
// maximum, starting from 0, so all-zero extents give dimension 0.
template <typename T>
__device__ __forceinline__ int arg_max_extent(const T* lo, const T* hi, int dim) {
  T best = T(0);
  int bd = 0;
  for (int d = 0; d < dim; ++d) {
    const T e = Ar<T>::sub(hi[d], lo[d]);
    if (e > best) {
      best = e;
      bd = d;
    }
  }
  return bd;
}

// Median-split trees (split rule 1): the cut is just above the median of the
// segment's coordinates along the cut dimension (of kMedianSamples values at
// evenly spaced positions, the segment's points being in no particular order;
// exact up to kHeld points, in k_mid). Just above (the next representable
// value): points equal to the median go left and hardly any lies on the cut.

// Single block: exclusive scan of the per-block sums. Each thread scans a contiguous run serially and one block-wide
// scan joins the runs (a loop of block-wide scans over the sums would
// serialise on its barriers: 0.2 ms per call at 22 M points).
__global__ void k_scan_block_sums(int2* sums, int nb, const LevelState* st) {
  pdl_begin();
  if (st->nseg == 0) return;
  const int per = (nb + kBlock - 1) / kBlock;
  const int b0 = threadIdx.x * per;
  const int b1 = min(b0 + per, nb);
  int2 run = make_int2(0, 0);
  for (int i = b0; i < b1; ++i) run = add2(run, sums[i]);
  int2 total;
  int2 carry = block_excl_scan(run, &total);
  for (int i = b0; i < b1; ++i) {
    const int2 v = sums[i];
    sums[i] = carry;
    carry = add2(carry, v);
  }
}

// Records the split of segment s of the current level and its two children,
// each a leaf, a small segment or a segment of the next level, with the child
// boxes cut at `cut` along `cd` (nabo/kdtree_cpu.cpp:192-223) and a next
// segment's cut dimension (each point's next cut coordinate moves along with
// the point).
template <typename T, int D>
__device__ void emit_split(const SegLevel<T>& L, const SegLevel<T>& next, int s, int leftCount, int cd, T cut,
                           const SegList<T>& small, const TreeMarks<T>& marks, int* counters, int dim, int bucket,
                           int smallMax, int segCap, int smallCap, int level) {
  const int count = L.count[s];
  const int start = L.start[s];
  const int turns = L.turns[s];
  mark_split(marks, start + leftCount, start, turns, cd, cut);
  L.leftCount[s] = leftCount;
  const T* lo = L.boxLo + (int64_t)s * kMaxDim;
  const T* hi = L.boxHi + (int64_t)s * kMaxDim;
  for (int side = 0; side < 2; ++side) {
    const int cst = side == 0 ? start : start + leftCount;
    const int ccount = side == 0 ? leftCount : count - leftCount;
    const int cturns = side == 0 ? turns + 1 : turns;
    int newSeg = -1;
    T* dLo = nullptr;
    T* dHi = nullptr;
    if (ccount <= bucket) {
      mark_leaf(marks, cst, cturns);
      atomicMax(counters + kHeight, level + 1);
    } else if (ccount > smallMax) {
      const int id = atomicAdd(counters + kNextSegs, 1);
      if (id >= segCap) {
        atomicOr(counters + kFlags, 1);
        return;
      }
      next.start[id] = cst;
      next.count[id] = ccount;
      next.turns[id] = cturns;
      dLo = next.boxLo + (int64_t)id * kMaxDim;
      dHi = next.boxHi + (int64_t)id * kMaxDim;
      newSeg = id;
    } else {
      const int sid = atomicAdd(counters + kSmallCount, 1);
      if (sid >= smallCap) {
        atomicOr(counters + kFlags, 1);
        return;
      }
      small.start[sid] = cst;
      small.count[sid] = ccount;
      small.turns[sid] = cturns;
      small.depth[sid] = level + 1;
      dLo = small.box + (int64_t)sid * 2 * D;
      dHi = dLo + D;
    }
    (side == 0 ? L.newLeft : L.newRight)[s] = newSeg;
    if (!dLo) continue;
    for (int d = 0; d < dim; ++d) {
      dLo[d] = side == 1 && d == cd ? cut : lo[d];
      dHi[d] = side == 0 && d == cd ? cut : hi[d];
    }
    if (newSeg >= 0) next.cutDim[newSeg] = arg_max_extent(dLo, dHi, dim);
  }
}

// Closes a level: makes the segments it produced the current ones.
__global__ void k_advance(LevelState* st, int* counters) {
  pdl_begin();
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  if (st->nseg > 0) {
    st->level += 1;
    counters[kLevels] = st->level;
  }
  st->nseg = counters[kNextSegs];
  counters[kNextSegs] = 0;
}

// ---- median-split top levels (split rule 1): a stable partition by scatter
//
// The median-split tree is this library's own, so its top levels need not
// reproduce the reference's in-place swaps. Each level scans two flags per
// position of a large segment, coordinate <= m and coordinate < m (m the
// segment's sampled median), keeps one of them per segment and moves every
// record to its child's range, flagged records first, each side in position
// order, into the other of two record arrays. Records whose child is a
// small segment go straight to the final array that the small-segment phase
// reads. Segment ids and cut coordinates travel with the records, so a
// level reads each position's id and coordinate twice and its record once,
// and writes its record, next id and next coordinate once: 6 launches and
// about 56 bytes per position of a large segment per level. The arrays in use
// alternate with the level's parity (LevelState::level), read on the device, so a fixed-level
// build needs no host decision.
constexpr int kItems = 4;               // consecutive positions per thread
constexpr int kTile = kBlock * kItems;  // positions per block and tile

template <typename T, int D>
struct MedianBufs {
  Rec<T, D>* rec[2];  // [n]
  int* seg[2];        // [nPad]: segment of the level, -1 outside large segments
  T* val[2];          // [nPad]: coordinate along the segment's cut dimension
  // selects rather than indexing, which would copy the struct to local memory
  __device__ Rec<T, D>* recs(int i) const { return i ? rec[1] : rec[0]; }
  __device__ int* segs(int i) const { return i ? seg[1] : seg[0]; }
  __device__ T* vals(int i) const { return i ? val[1] : val[0]; }
};

template <typename T>
__device__ __forceinline__ void load4(const T* __restrict__ p, T (&v)[kItems]) {
  if constexpr (sizeof(T) == 4) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x;
    v[1] = x.y;
    v[2] = x.z;
    v[3] = x.w;
  } else {
    const double2 a = reinterpret_cast<const double2*>(p)[0];
    const double2 b = reinterpret_cast<const double2*>(p)[1];
    v[0] = a.x;
    v[1] = a.y;
    v[2] = b.x;
    v[3] = b.y;
  }
}

// One tile's positions of a thread: segment ids, coordinates and the two
// flags (x: v <= m, y: v < m; m = L.cut[s] holds the median until the
// level's split is chosen).
template <typename T>
struct MedianItems {
  int s[kItems];
  T v[kItems];
};

template <typename T>
__device__ __forceinline__ void median_load(const int* __restrict__ seg, const T* __restrict__ val, int64_t p0,
                                            int64_t nPad, MedianItems<T>& it) {
  if (p0 < nPad) {
    const int4 s4 = *reinterpret_cast<const int4*>(seg + p0);
    it.s[0] = s4.x;
    it.s[1] = s4.y;
    it.s[2] = s4.z;
    it.s[3] = s4.w;
    load4(val + p0, it.v);
  } else {
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      it.s[i] = -1;
      it.v[i] = T(0);
    }
  }
}

template <typename T>
__device__ __forceinline__ int2 median_flag(const SegLevel<T>& L, int s, T v) {
  if (s < 0) return make_int2(0, 0);
  const T m = L.cut[s];
  return make_int2(v <= m ? 1 : 0, v < m ? 1 : 0);
}

// Each segment's sampled median, a warp each: latency-bound, one load and a
// shuffle sort. (A thread each, sorting its 31 samples in local memory, took
// 340 us of a 512-cloud, 22 M-point build; this takes 92. With the handover
// at 256 points the levels had ten times the segments and warps were slower.)
template <typename T, int D>
__global__ void k_median_cut(SegLevel<T> L, const LevelState* st, MedianBufs<T, D> B) {
  pdl_begin();
  using Key = typename KeyOf<T>::type;
  const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (s >= st->nseg) return;
  const T* val = B.vals(st->level & 1) + L.start[s];
  const int64_t count = L.count[s];
  Key e[1] = {lane < kMedianSamples ? ordered_key(val[(2 * lane + 1) * count / (2 * kMedianSamples)]) : ~Key(0)};
  warp_sort_keys<1>(e, lane);
  if (lane == kMedianSamples / 2) L.cut[s] = ordered_val(e[0], T(0));
}

// Block b scans tiles [b * tiles, (b + 1) * tiles) in position order and
// records, besides its totals, each segment's running flag counts at its
// first position (exclusive) and last position (inclusive).
// The next tile's ids and coordinates are loaded before this tile's scan.
template <typename T, int D>
__global__ void k_median_sums(MedianBufs<T, D> B, int64_t nPad, SegLevel<T> L, int tiles, int2* blockSums,
                              int2* segFirst, int2* segLast, const LevelState* st) {
  pdl_begin();
  if (st->nseg == 0) return;
  const int par = st->level & 1;
  const int* seg = B.segs(par);
  const T* val = B.vals(par);
  const int64_t first = (int64_t)blockIdx.x * tiles * kTile + threadIdx.x * kItems;
  MedianItems<T> nxt;
  median_load(seg, val, first, nPad, nxt);
  int2 carry = make_int2(0, 0);
  for (int t = 0; t < tiles; ++t) {
    const MedianItems<T> it = nxt;
    const int64_t p0 = first + (int64_t)t * kTile;
    if (t + 1 < tiles) median_load(seg, val, p0 + kTile, nPad, nxt);
    int2 f[kItems];
    int2 sum = make_int2(0, 0);
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      f[i] = median_flag(L, it.s[i], it.v[i]);
      sum = add2(sum, f[i]);
    }
    int2 total;
    int2 ex = add2(block_excl_scan(sum, &total), carry);
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      const int s = it.s[i];
      if (s >= 0) {
        const int64_t p = p0 + i;
        const int st0 = L.start[s];
        if (p == st0) segFirst[s] = ex;
        if (p == st0 + L.count[s] - 1) segLast[s] = add2(ex, f[i]);
      }
      ex = add2(ex, f[i]);
    }
    carry = add2(carry, total);
  }
  if (threadIdx.x == 0) blockSums[blockIdx.x] = carry;
}

// Chooses each segment's split from its two flag totals and writes it:
//   some point above the median  -> cut just above it, left = v <= m
//   else some point below it     -> cut at it, left = v < m
//   else (all equal)             -> cut at it, first half left by position
// L.lt keeps the chosen flag's global rank at the segment's first position.
template <typename T, int D>
__global__ void k_median_split(SegLevel<T> L, SegLevel<T> next, const LevelState* st, SegList<T> small,
                               TreeMarks<T> marks, int* counters, int dim, int bucket, int smallMax, int segCap,
                               int smallCap, const int2* __restrict__ blockPrefix, const int2* __restrict__ segFirst,
                               const int2* __restrict__ segLast, int perBlock) {
  pdl_begin();
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  const int nseg = st->nseg;
  if (s >= nseg) return;
  const int count = L.count[s];
  const int start = L.start[s];
  const int2 a = add2(blockPrefix[start / perBlock], segFirst[s]);
  const int2 b = add2(blockPrefix[(start + count - 1) / perBlock], segLast[s]);
  const int le = b.x - a.x, lt = b.y - a.y;
  const T m = L.cut[s];
  int mode, leftCount;
  T cut;
  if (le < count) {
    mode = 0;
    leftCount = le;
    cut = next_up(m);
    L.lt[s] = a.x;
  } else if (lt > 0) {
    mode = 1;
    leftCount = lt;
    cut = m;
    L.lt[s] = a.y;
  } else {
    mode = 2;
    leftCount = count / 2;
    cut = m;
  }
  leftCount = leftCount < 1 ? 1 : (leftCount > count - 1 ? count - 1 : leftCount);
  L.mode[s] = mode;
  emit_split<T, D>(L, next, s, leftCount, L.cutDim[s], cut, small, marks, counters, dim, bucket, smallMax, segCap,
                   smallCap, st->level);
}

// Moves every record of a large segment to its child's range: a record with
// r flagged records before it in its segment goes to start + r when flagged,
// to start + leftCount + (its offset - r) otherwise. Positions outside large
// segments only mark themselves outside in the next level's id array.
template <typename T, int D>
__global__ void k_median_scatter(MedianBufs<T, D> B, Rec<T, D>* __restrict__ finalRecs, int64_t nPad,
                                 SegLevel<T> L, SegLevel<T> next, int tiles, const int2* __restrict__ blockPrefix,
                                 const LevelState* st) {
  pdl_begin();
  if (st->nseg == 0) return;
  const int par = st->level & 1;
  const int* seg = B.segs(par);
  const T* val = B.vals(par);
  const Rec<T, D>* src = B.recs(par);
  Rec<T, D>* dst = B.recs(par ^ 1);
  int* segN = B.segs(par ^ 1);
  T* valN = B.vals(par ^ 1);
  const int64_t first = (int64_t)blockIdx.x * tiles * kTile + threadIdx.x * kItems;
  MedianItems<T> nxt;
  median_load(seg, val, first, nPad, nxt);
  int2 carry = blockPrefix[blockIdx.x];
  for (int t = 0; t < tiles; ++t) {
    const MedianItems<T> it = nxt;
    const int64_t p0 = first + (int64_t)t * kTile;
    if (t + 1 < tiles) median_load(seg, val, p0 + kTile, nPad, nxt);
    int2 f[kItems];
    int2 sum = make_int2(0, 0);
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      f[i] = median_flag(L, it.s[i], it.v[i]);
      sum = add2(sum, f[i]);
    }
    int2 total;
    int2 ex = add2(block_excl_scan(sum, &total), carry);
    carry = add2(carry, total);
    if (p0 >= nPad) continue;
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      const int s = it.s[i];
      const int64_t p = p0 + i;
      if (s < 0) {
        segN[p] = -1;
      } else {
        const int start = L.start[s];
        const int mode = L.mode[s];
        const int lc = L.leftCount[s];
        const int loc = (int)(p - start);
        int before;
        bool left;
        if (mode == 2) {
          before = loc < lc ? loc : lc;
          left = loc < lc;
        } else {
          before = (mode == 0 ? ex.x : ex.y) - L.lt[s];
          left = (mode == 0 ? f[i].x : f[i].y) != 0;
        }
        const int64_t dest = start + (left ? before : lc + (loc - before));
        const int child = left ? L.newLeft[s] : L.newRight[s];
        Rec<T, D> r;
        load_rec(src, p, r);
        if (child >= 0) {
          dst[dest] = r;
          segN[dest] = child;
          valN[dest] = coord_of(r, next.cutDim[child]);
        } else {
          finalRecs[dest] = r;
          segN[dest] = -1;
        }
      }
      ex = add2(ex, f[i]);
    }
  }
}

// Staging a tile (record, destination, next id and coordinate per slot)
// within 47 KB of static shared memory: float records of up to 4
// dimensions.
template <typename T, int D>
constexpr bool median_staging_fits() {
  return (size_t)kTile * (sizeof(Rec<T, D>) + 2 * sizeof(int) + sizeof(T)) <= 47 * 1024;
}

// k_median_scatter with the tile's moves staged in shared memory: each
// record, with its destination and next id and coordinate, goes to a slot
// in destination order (the tile's flagged records first, each side in
// position order, so every run of one segment and side is contiguous in
// both), then the block writes the slots out, consecutive threads to
// consecutive destinations.
template <typename T, int D>
__global__ void k_median_scatter_staged(MedianBufs<T, D> B, Rec<T, D>* __restrict__ finalRecs, int64_t nPad,
                                        SegLevel<T> L, SegLevel<T> next, int tiles,
                                        const int2* __restrict__ blockPrefix, const LevelState* st) {
  // (instantiated only where the staging fits; see median_scatter)
  constexpr int kStage = median_staging_fits<T, D>() ? kTile : 1;
  __shared__ Rec<T, D> sRec[kStage];
  __shared__ int sDest[kStage];
  __shared__ int sChild[kStage];
  __shared__ T sVal[kStage];
  pdl_begin();
  if (st->nseg == 0) return;
  const int par = st->level & 1;
  const int* seg = B.segs(par);
  const T* val = B.vals(par);
  const Rec<T, D>* src = B.recs(par);
  Rec<T, D>* dst = B.recs(par ^ 1);
  int* segN = B.segs(par ^ 1);
  T* valN = B.vals(par ^ 1);
  const int64_t first = (int64_t)blockIdx.x * tiles * kTile + threadIdx.x * kItems;
  MedianItems<T> nxt;
  median_load(seg, val, first, nPad, nxt);
  int2 carry = blockPrefix[blockIdx.x];
  for (int t = 0; t < tiles; ++t) {
    const MedianItems<T> it = nxt;
    const int64_t p0 = first + (int64_t)t * kTile;
    if (t + 1 < tiles) median_load(seg, val, p0 + kTile, nPad, nxt);
    int2 f[kItems];
    int2 sum = make_int2(0, 0);
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      f[i] = median_flag(L, it.s[i], it.v[i]);
      sum = add2(sum, f[i]);
    }
    int2 total;
    int2 ex = add2(block_excl_scan(sum, &total), carry);
    carry = add2(carry, total);
    // destination of each held record and its side
    int dest[kItems];
    bool left[kItems];
    int2 side = make_int2(0, 0);  // (left, right) records this thread moves
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      const int s = it.s[i];
      dest[i] = -1;
      left[i] = false;
      if (s >= 0) {
        const int64_t p = p0 + i;
        const int start = L.start[s];
        const int mode = L.mode[s];
        const int lc = L.leftCount[s];
        const int loc = (int)(p - start);
        int before;
        if (mode == 2) {
          before = loc < lc ? loc : lc;
          left[i] = loc < lc;
        } else {
          before = (mode == 0 ? ex.x : ex.y) - L.lt[s];
          left[i] = (mode == 0 ? f[i].x : f[i].y) != 0;
        }
        dest[i] = start + (left[i] ? before : lc + (loc - before));
        side = add2(side, make_int2(left[i] ? 1 : 0, left[i] ? 0 : 1));
      } else if (p0 < nPad) {
        segN[p0 + i] = -1;
      }
      ex = add2(ex, f[i]);
    }
    int2 sideTotal;
    int2 slot = block_excl_scan(side, &sideTotal);
    slot.y += sideTotal.x;  // rights after all lefts
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      if (dest[i] < 0) continue;
      const int s = it.s[i];
      const int j = left[i] ? slot.x++ : slot.y++;
      const int child = left[i] ? L.newLeft[s] : L.newRight[s];
      Rec<T, D> r;
      load_rec(src, p0 + i, r);
      sRec[j] = r;
      sChild[j] = child;
      sDest[j] = dest[i];
      if (child >= 0) sVal[j] = coord_of(r, next.cutDim[child]);
    }
    __syncthreads();
    const int moved = sideTotal.x + sideTotal.y;
    for (int j = threadIdx.x; j < moved; j += blockDim.x) {
      const int d = sDest[j];
      const int child = sChild[j];
      if (child >= 0) {
        dst[d] = sRec[j];
        segN[d] = child;
        valN[d] = sVal[j];
      } else {
        finalRecs[d] = sRec[j];
        segN[d] = -1;
      }
    }
    __syncthreads();
  }
}

// The scatter kernel for this record size.
template <typename T, int D>
constexpr auto median_scatter() {
  if constexpr (median_staging_fits<T, D>())
    return k_median_scatter_staged<T, D>;
  else
    return k_median_scatter<T, D>;
}

// A fixed-level build that ran out of levels leaves records of unfinished
// segments in the working arrays; they go to the final array, whose cloud
// ranges then hold every point (the one-leaf-per-cloud fallback reads them).
template <typename T, int D>
__global__ void k_median_flush(MedianBufs<T, D> B, Rec<T, D>* finalRecs, int64_t n, const LevelState* st) {
  if (st->nseg == 0) return;
  const int par = st->level & 1;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x)
    if (B.segs(par)[p] >= 0) finalRecs[p] = B.recs(par)[p];
}

// ---- forest set-up: clouds are contiguous point ranges [off[c], off[c+1])

// Packs the clouds into records (index within the cloud) and reduces each
// cloud's per-dimension min/max (ordered keys) and a non-finite flag, in
// one pass. Block b takes the contiguous positions [b * chunk, (b + 1) *
// chunk) a tile of kBlock at a time, following the clouds with a cursor (a
// binary search once per thread); each lane keeps the running min/max of
// its current cloud, and the warp flushes them (reduced across the lanes
// of each cloud, one atomic per cloud and dimension) only when some lane's
// cloud changes, and at the end. With `smallRoots`, points of clouds whose
// root is a leaf or a small segment (at most rootMax points) are also written
// there.
template <typename T, int D>
__global__ void k_pack_bounds(const T* __restrict__ cloud, int64_t n, int64_t stride, int dim,
                              const int64_t* __restrict__ off, int nClouds, int64_t chunk,
                              Rec<T, D>* __restrict__ recs, Rec<T, D>* __restrict__ smallRoots, int rootMax,
                              typename KeyOf<T>::type* mnK, typename KeyOf<T>::type* mxK, int* nonFinite) {
  using Key = typename KeyOf<T>::type;
  const int64_t begin = blockIdx.x * chunk;
  const int64_t end = begin + chunk < n ? begin + chunk : n;
  if (begin >= end) return;
  int c = cloud_of(off, nClouds, begin + threadIdx.x < end ? begin + threadIdx.x : begin);
  int cur = -1;  // cloud of the running min/max
  Key kmin[D], kmax[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    kmin[d] = ~Key(0);
    kmax[d] = 0;
  }
  int bad = 0;
  auto flush = [&]() {
#pragma unroll
    for (int d = 0; d < D; ++d) {
      bool tail;
      const Key a = seg_warp_reduce(cur, kmin[d], MinOp(), &tail);
      const Key b = seg_warp_reduce(cur, kmax[d], MaxOp(), &tail);
      if (tail && cur >= 0 && d < dim) {
        atomicMin(mnK + (int64_t)cur * kMaxDim + d, a);
        atomicMax(mxK + (int64_t)cur * kMaxDim + d, b);
      }
      kmin[d] = ~Key(0);
      kmax[d] = 0;
    }
  };
  for (int64_t p0 = begin; p0 < end; p0 += kBlock) {
    const int64_t p = p0 + threadIdx.x;
    int cp = -1;
    Rec<T, D> r;
    if (p < end) {
      while (off[c + 1] <= p) ++c;
      cp = c;
#pragma unroll
      for (int q = 0; q < RecSize<T, D>::chunks; ++q) r.v[q] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int d = 0; d < D; ++d) r.p.c[d] = d < dim ? cloud[p * stride + d] : T(0);
      r.p.idx = (int32_t)(p - off[c]);
      recs[p] = r;
      if (smallRoots && off[c + 1] - off[c] <= rootMax) smallRoots[p] = r;
    }
    if (__any_sync(kFull, cp != cur)) {
      flush();
      cur = cp;
    }
    if (cp >= 0) {
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const Key k = ordered_key(r.p.c[d]);
        kmin[d] = k < kmin[d] ? k : kmin[d];
        kmax[d] = k > kmax[d] ? k : kmax[d];
        bad |= (d < dim && !isfinite(r.p.c[d])) ? 1 : 0;
      }
    }
  }
  flush();
  if (__any_sync(kFull, bad) && (threadIdx.x & 31) == 0) atomicOr(nonFinite, 1);
}

template <typename T>
__global__ void k_init_keys_forest(typename KeyOf<T>::type* mnK, typename KeyOf<T>::type* mxK, int nClouds) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nClouds * kMaxDim) return;
  mnK[i] = ordered_key(Ar<T>::inf());
  mxK[i] = ordered_key(-Ar<T>::inf());
}

// One root per cloud: a leaf, a small segment, or a segment of level 0 (of the
// median rule; k_top's blocks find their own). Root box = (min,
// max(numeric_limits<T>::min(), max)), as the reference's constructor sets it
// (nabo/nabo.cpp:73-74, nabo/kdtree_cpu.cpp:256-267).
template <typename T, int D>
__global__ void k_forest_roots(const int64_t* __restrict__ off, int nClouds, const typename KeyOf<T>::type* mnK,
                               const typename KeyOf<T>::type* mxK, int dim, int bucket, int smallMax, int median,
                               SegLevel<T> L, SegList<T> small,
                               TreeMarks<T> marks, LevelState* st, int* counters, int* rootSeg, T* rootLo,
                               T* rootHi) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nClouds) return;
  const int start = (int)off[c];
  const int count = (int)(off[c + 1] - start);
  T lo[D], hi[D];
#pragma unroll
  for (int d = 0; d < D; ++d) {
    lo[d] = hi[d] = T(0);
    if (d < dim) {
      lo[d] = ordered_val(mnK[(int64_t)c * kMaxDim + d], T(0));
      const T mx = ordered_val(mxK[(int64_t)c * kMaxDim + d], T(0));
      const T tiny = std::numeric_limits<T>::min();
      hi[d] = mx > tiny ? mx : tiny;
      rootLo[(int64_t)c * kMaxDim + d] = lo[d];
      rootHi[(int64_t)c * kMaxDim + d] = hi[d];
    }
  }
  Split<T> first{};
  first.start = -1;
  first.turnsDim = (uint32_t)c;
  marks.split[start] = first;
  int seg = -1;
  if (count <= bucket) {
    mark_leaf(marks, start, -c);
  } else if (count <= smallMax) {
    const int id = atomicAdd(counters + kSmallCount, 1);
    small.start[id] = start;
    small.count[id] = count;
    small.turns[id] = -c;
    small.depth[id] = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      small.box[(int64_t)id * 2 * D + d] = lo[d];
      small.box[(int64_t)id * 2 * D + D + d] = hi[d];
    }
  } else if (median) {
    seg = atomicAdd(&st->nseg, 1);
    L.start[seg] = start;
    L.count[seg] = count;
    L.turns[seg] = -c;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      if (d < dim) {
        L.boxLo[(int64_t)seg * kMaxDim + d] = lo[d];
        L.boxHi[(int64_t)seg * kMaxDim + d] = hi[d];
      }
    }
    // read before any level kernel runs
    T mid;
    L.cutDim[seg] = widest_dim<T, D>(lo, hi, dim, &mid);
  }
  if (rootSeg) rootSeg[c] = seg;
}

// The median rule's root segment of each position (-1 for a leaf or small
// root, and for the padding [n, nPad)) and the position's coordinate along
// that segment's cut dimension, by contiguous block ranges with a cloud
// cursor as in k_pack_bounds.
template <typename T, int D>
__global__ void k_init_segof(int* segOf, int64_t n, int64_t nPad, int64_t chunk, const int64_t* __restrict__ off,
                             int nClouds, const int* __restrict__ rootSeg, const Rec<T, D>* __restrict__ recs,
                             const int* __restrict__ cutDim, T* val) {
  const int64_t begin = blockIdx.x * chunk;
  const int64_t end = begin + chunk < nPad ? begin + chunk : nPad;
  if (begin >= end) return;
  int c = begin < n ? cloud_of(off, nClouds, begin + threadIdx.x < n ? begin + threadIdx.x : begin) : 0;
  for (int64_t p = begin + threadIdx.x; p < end; p += kBlock) {
    int s = -1;
    if (p < n) {
      while (off[c + 1] <= p) ++c;
      s = rootSeg[c];
      if (s >= 0) val[p] = recs[p].p.c[cutDim[s]];
    }
    segOf[p] = s;
  }
}

// ---------------------------------------------------------------------------
// Host side.

// Stream-ordered scratch that is released when the owner goes out of scope.
struct Scratch {
  cudaStream_t stream;
  std::vector<void*> ptrs;
  explicit Scratch(cudaStream_t s) : stream(s) {}
  ~Scratch() {
    for (void* p : ptrs) scratch_free(p, stream);
  }
  template <typename V>
  cudaError_t get(V** out, int64_t count) {
    void* p = nullptr;
    const size_t bytes = (size_t)std::max<int64_t>(count, 1) * sizeof(V);
    cudaError_t e = scratch_alloc(&p, bytes, stream);
    if (e == cudaSuccess) ptrs.push_back(p);
    *out = static_cast<V*>(p);
    return e;
  }
};

// One block of stream-ordered scratch, laid out in two walks of the same
// list of arrays (a build took about 60 allocations, 1-2 us of host time
// each).
struct Arena {
  char* base = nullptr;
  size_t bytes = 0;
  template <typename V>
  void take(V*& p, int64_t count) {
    p = base ? reinterpret_cast<V*>(base + bytes) : nullptr;
    bytes += ((size_t)std::max<int64_t>(count, 1) * sizeof(V) + 255) & ~size_t(255);
  }
};

template <typename T>
void take_level(Arena& A, SegLevel<T>& L, int64_t cap) {
  A.take(L.start, cap);
  A.take(L.count, cap);
  A.take(L.turns, cap);
  A.take(L.boxLo, cap * kMaxDim);
  A.take(L.boxHi, cap * kMaxDim);
  A.take(L.cutDim, cap);
  A.take(L.cut, cap);
  A.take(L.mode, cap);
  A.take(L.lt, cap);
  A.take(L.leftCount, cap);
  A.take(L.newLeft, cap);
  A.take(L.newRight, cap);
}

template <typename T>
double host_key_to_double(typename KeyOf<T>::type k);
template <>
double host_key_to_double<float>(uint32_t k) {
  const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  float f;
  std::memcpy(&f, &u, 4);
  return (double)f;
}
template <>
double host_key_to_double<double>(unsigned long long k) {
  const unsigned long long u = (k & 0x8000000000000000ull) ? (k & 0x7fffffffffffffffull) : ~k;
  double f;
  std::memcpy(&f, &u, 8);
  return f;
}

// Centre and scale of the tensor-core filter's coordinates: the sample's medians,
// and the power of 2 that brings all but its few farthest points to between 4
// and 8 from there. Left at scale 0 when the cloud's range does not suit it.
template <int D>
void tc_scale(const CloudStats<float, D>& st, int dim, const double* lo, const double* hi, TcScale* s) {
  constexpr int kFar = kSamplePoints / 32;
  double widest = 0.0;
  for (int d = 0; d < dim; ++d) {
    if (!(std::fabs(lo[d]) < 1e15 && std::fabs(hi[d]) < 1e15)) return;
    widest = std::max(widest, hi[d] - lo[d]);
  }
  if (!(widest > 1e-15)) return;
  float v[kSamplePoints], reach[kSamplePoints] = {};
  for (int d = 0; d < dim; ++d) {
    for (int i = 0; i < kSamplePoints; ++i) v[i] = st.sample[i][d];
    std::nth_element(v, v + kSamplePoints / 2, v + kSamplePoints);
    s->centre[d] = v[kSamplePoints / 2];
    for (int i = 0; i < kSamplePoints; ++i)
      reach[i] = std::max(reach[i], std::fabs(st.sample[i][d] - s->centre[d]));
  }
  std::nth_element(reach, reach + kSamplePoints - 1 - kFar, reach + kSamplePoints);
  double r = reach[kSamplePoints - 1 - kFar];
  if (!(r > 1e-15)) r = widest;  // (nearly all points are one)
  int e = 0;
  std::frexp(r, &e);  // r <= 2^e
  s->scale = (float)std::ldexp(1.0, 3 - e);
  s->scale2 = s->scale * s->scale;
}

// Per-dimension bounds; fails on NaN or infinite coordinates, for which
// the reference's split loop does not terminate (idealCutVal becomes NaN
// and leftCount 0, nabo/kdtree_cpu.cpp:180-190).
template <typename T, int D>
int compute_bounds(const Rec<T, D>* recs, int64_t n, int dim, cudaStream_t stream, Scratch& sc, double* lo,
                   double* hi, TcScale* tc) {
  CloudStats<T, D>* st;
  NABO_CUDA_TRY(sc.get(&st, 1));
  k_init_stats<T, D><<<1, kSamplePoints, 0, stream>>>(st, recs, n);
  const int grid = (int)std::min<int64_t>(ceil_div(n, kBlock), 152 * 8);
  k_bounds<T, D><<<grid, kBlock, 0, stream>>>(recs, n, dim, st->mn, st->mx, &st->nonFinite);
  NABO_CUDA_TRY(cudaGetLastError());
  CloudStats<T, D> h;
  NABO_CUDA_TRY(cudaMemcpyAsync(&h, st, sizeof(h), cudaMemcpyDeviceToHost, stream));
  NABO_CUDA_TRY(cudaStreamSynchronize(stream));
  if (h.nonFinite) return set_error(kErrArgument, "Cloud has non-finite (NaN or infinite) coordinates");
  for (int d = 0; d < kMaxDim; ++d) {
    lo[d] = d < dim ? host_key_to_double<T>(h.mn[d]) : 0.0;
    hi[d] = d < dim ? host_key_to_double<T>(h.mx[d]) : 0.0;
  }
  if constexpr (sizeof(T) == 4) tc_scale<D>(h, dim, lo, hi, tc);
  return kOk;
}

}  // namespace

template <typename T, int D>
int pack_cloud(const T* dCloud, int64_t n, int64_t stride, int dim, cudaStream_t stream, DeviceCloud* out) {
  Rec<T, D>* recs = nullptr;
  NABO_CUDA_TRY(object_alloc((void**)&recs, (size_t)n * sizeof(Rec<T, D>), stream));
  out->recs = recs;
  k_pack<T, D><<<ceil_div(n, kBlock), kBlock, 0, stream>>>(dCloud, n, stride, dim, recs);
  NABO_CUDA_TRY(cudaGetLastError());
  Scratch sc(stream);
  const int rc = compute_bounds<T, D>(recs, n, dim, stream, sc, out->lo, out->hi, &out->tc);
  if (rc != kOk) return rc;
  return kOk;
}

// Builds the trees of `nClouds` clouds stored back to back (cloud c =
// points [off[c], off[c+1]) of dCloud) into one record array and one node
// array: cloud c's tree is the pre-order range [nodeOffset[c],
// nodeOffset[c+1]), its points keep their index within the cloud.
// maxLevels < 0: as many top levels as the trees need (the median rule's
// host loop reads one int per level; the reference's rule runs them in one
// launch); a cloud with non-finite coordinates stops the build, reported in
// f->status. maxLevels >= 0: at most that many, with no host
// synchronisation, so the whole build can be captured in a CUDA graph; a
// tree needing more sets the overflow flag (f->status).
template <typename T, int D>
int build_forest(const T* dCloud, int64_t n, int64_t stride, int dim, unsigned bucketSize, const int64_t* dOff,
                 int nClouds, int maxLevels, cudaStream_t stream, ForestOut* f, int splitRule) {
  using Key = typename KeyOf<T>::type;
  using Mid = MidShape<T, D>;
  const int N = (int)n;
  const bool hostDriven = maxLevels < 0;
  const bool median = splitRule == 1;
  const int bucket = (int)std::min<int64_t>(bucketSize, std::numeric_limits<int>::max());
  int device = 0, sms = 0;
  NABO_CUDA_TRY(cudaGetDevice(&device));
  NABO_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  sms = std::max(sms, 1);

  // The median split works in two record arrays of its own (positions padded
  // to whole tiles) and leaves the final array to its scatter.
  const int64_t nPad = median ? (std::max<int64_t>(n, 1) + kTile - 1) / kTile * kTile : n;
  // per-position passes over contiguous block ranges: 8 blocks per SM
  const int rangeBlocks = std::max(1, std::min(ceil_div(std::max<int64_t>(n, 1), kBlock), 8 * sms));
  const int64_t rangeChunk = (int64_t)ceil_div(ceil_div(std::max<int64_t>(n, 1), rangeBlocks), kBlock) * kBlock;

  // Small segments: what a block of k_mid holds in shared memory. (Median
  // rule, 512 clouds of 21 M points, built and searched: handed over at 256
  // points 18.8 ms, 1024 18.3, 2048 18.1, 4096 17.9.)
  const int smallMax = Mid::kMax;
  const size_t midSmem = Mid::smem(smallMax, bucket);
  // The limit is the kernel's, shared by all threads that build: always set to
  // the most any build asks for (the smallest bucket's), never to this one's
  // own need, which could refuse another thread's launch.
  constexpr int kMidSmemMax = (int)Mid::smem(Mid::kMax, 2);
  NABO_CUDA_TRY(cudaFuncSetAttribute(k_mid<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMidSmemMax));
  int midOcc = 0;
  NABO_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&midOcc, k_mid<T, D>, Mid::kThreads, midSmem));

  const bool top = !median && n > smallMax;

  const int64_t segCap = n / (smallMax + 1) + 2;
  const int64_t smallCap = n / ((int64_t)bucket + 1) + nClouds + 2;
  const int64_t words = n / 32 + 1;
  const int rankBlocks = ceil_div(words, kRankBlock);
  const int nb = ceil_div(n, kBlock);

  int* counters;
  LevelState* st;
  TreeMarks<T> marks;
  uint32_t *rank, *rankSums;
  Key* keys;
  SegList<T> small;
  MedianBufs<T, D> mb = {};
  int* rootSeg = nullptr;
  int2 *blockSums, *segFirst, *segLast;
  SegLevel<T> cur = {}, nxt = {};
  TopArgs<T, D> ta = {};
  size_t zeroed = 0;
  const auto layout = [&](Arena& A) {
    A.take(counters, kBuildCounters);
    A.take(st, 1);
    A.take(ta.st, 1);
    A.take(marks.leafBits, words);
    zeroed = A.bytes;
    A.take(marks.split, n);
    A.take(marks.leafTurns, n);
    A.take(rank, words);
    A.take(rankSums, rankBlocks + 1);
    A.take(keys, 2 * (int64_t)nClouds * kMaxDim);
    A.take(small.start, smallCap);
    A.take(small.count, smallCap);
    A.take(small.turns, smallCap);
    A.take(small.depth, smallCap);
    A.take(small.box, smallCap * 2 * D);
    if (median) {
      for (int i = 0; i < 2; ++i) {
        A.take(mb.rec[i], n);
        A.take(mb.seg[i], nPad);
        A.take(mb.val[i], nPad);
      }
      A.take(rootSeg, nClouds);
      A.take(blockSums, nb);
      A.take(segFirst, segCap);
      A.take(segLast, segCap);
      take_level(A, cur, segCap);
      take_level(A, nxt, segCap);
    } else if (top) {
      A.take(ta.exch, n);
      A.take(ta.head, sms);
      A.take(ta.tail, sms);
      A.take(ta.head2, sms);
      A.take(ta.tail2, sms);
    }
  };
  Arena A;
  layout(A);
  Scratch sc(stream);
  NABO_CUDA_TRY(sc.get(&A.base, (int64_t)A.bytes));
  A.bytes = 0;
  layout(A);
  NABO_CUDA_TRY(cudaMemsetAsync(A.base, 0, zeroed, stream));
  NABO_CUDA_TRY(cudaMemsetAsync(f->status, 0, 4 * sizeof(int), stream));

  // records and per-cloud bounds in one pass
  Rec<T, D>* recs = static_cast<Rec<T, D>*>(f->recs);
  Rec<T, D>* packed = median ? mb.rec[0] : recs;
  k_init_keys_forest<T><<<ceil_div(nClouds * kMaxDim, 256), 256, 0, stream>>>(keys, keys + nClouds * kMaxDim,
                                                                              nClouds);
  if (n > 0)
    k_pack_bounds<T, D><<<rangeBlocks, kBlock, 0, stream>>>(dCloud, n, stride, dim, dOff, nClouds, rangeChunk, packed,
                                                            median ? recs : nullptr, std::max(smallMax, bucket), keys,
                                                            keys + nClouds * kMaxDim, f->status + 0);
  NABO_CUDA_TRY(cudaGetLastError());
  const int* nonFinite = hostDriven ? f->status + 0 : nullptr;
  if (hostDriven && median) {
    int bad = 0;
    NABO_CUDA_TRY(cudaMemcpyAsync(&bad, f->status + 0, sizeof(int), cudaMemcpyDeviceToHost, stream));
    NABO_CUDA_TRY(cudaStreamSynchronize(stream));
    if (bad) return set_error(kErrArgument, "Cloud has non-finite (NaN or infinite) coordinates");
  }
  k_forest_roots<T, D><<<ceil_div(nClouds, 128), 128, 0, stream>>>(
      dOff, nClouds, keys, keys + nClouds * kMaxDim, dim, bucket, smallMax, median ? 1 : 0, cur, small, marks, st,
      counters, rootSeg, static_cast<T*>(f->rootLo), static_cast<T*>(f->rootHi));
  NABO_CUDA_TRY(cudaGetLastError());

  if (top) {
    ta.recs = recs;
    ta.off = dOff;
    ta.rootLo = static_cast<const T*>(f->rootLo);
    ta.rootHi = static_cast<const T*>(f->rootHi);
    ta.small = small;
    ta.marks = marks;
    ta.counters = counters;
    ta.nonFinite = nonFinite;
    ta.n = N;
    ta.nClouds = nClouds;
    ta.dim = dim;
    ta.smallMax = smallMax;
    ta.bucket = bucket;
    ta.maxLevels = maxLevels;
    ta.smallCap = (int)smallCap;
    ta.barrierPolls = f->barrierPolls;
    // One block per SM, each with its share of the positions. All of them have
    // to be resident at once: where the launch may use fewer SMs than the
    // device has (a stream or context with a part of them) it is refused, and
    // fewer blocks take more positions each.
    for (int most = sms;;) {
      const int chunk = (int)std::max<int64_t>(kTopMinChunk, ((n + most - 1) / most + 31) / 32 * 32);
      const int topBlocks = ceil_div(n, chunk);
      // the segments overlapping a chunk hold more than smallMax points each
      const int pieces = chunk / smallMax + 2;
      const size_t withRecs = TopShape<T, D>::bytes(chunk, pieces, true);
      const size_t withLists = TopShape<T, D>::bytes(chunk, pieces, false);
      const int topMode = withRecs <= kTopSmemMax ? kTopResident : (withLists <= kTopSmemMax ? kTopLists : kTopGlobal);
      ta.chunk = chunk;
      ta.pieces = pieces;
      ta.workBytes = (int64_t)withLists;
      if (topMode == kTopGlobal) NABO_CUDA_TRY(sc.get(&ta.work, (int64_t)withLists * topBlocks));
      const void* kernel = topMode == kTopResident ? (const void*)k_top<T, D, kTopResident>
                           : topMode == kTopLists  ? (const void*)k_top<T, D, kTopLists>
                                                   : (const void*)k_top<T, D, kTopGlobal>;
      const size_t topSmem = topMode == kTopResident ? withRecs : (topMode == kTopLists ? withLists : 0);
      // the most any build asks for, as k_mid's
      if (topSmem > 0)
        NABO_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTopSmemMax));
      void* args[] = {&ta};
      const cudaError_t e =
          cudaLaunchCooperativeKernel(kernel, dim3(topBlocks), dim3(kTopThreads), args, topSmem, stream);
      if (e != cudaErrorCooperativeLaunchTooLarge || topBlocks == 1) {
        NABO_CUDA_TRY(e);
        break;
      }
      cudaGetLastError();
      most = topBlocks / 2;
    }
  }
  if (median) {
    if (nPad > 0) {
      const int64_t segChunk = rangeChunk * ceil_div(nPad, rangeChunk * rangeBlocks);
      k_init_segof<T, D><<<ceil_div(nPad, segChunk), kBlock, 0, stream>>>(mb.seg[0], n, nPad, segChunk, dOff, nClouds,
                                                                          rootSeg, packed, cur.cutDim, mb.val[0]);
      NABO_CUDA_TRY(cudaGetLastError());
    }
    const int sg = ceil_div(segCap, 128);
    // as many blocks as are resident at once, each scanning a contiguous run
    // of mTiles tiles of kTile positions
    const int mTilesTotal = (int)(nPad / kTile);
    int mOcc = 0;
    NABO_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&mOcc, median_scatter<T, D>(), kBlock, 0));
    const int mGrid = std::max(1, std::min(mTilesTotal, std::max(mOcc, 1) * sms));
    const int mTiles = ceil_div(mTilesTotal, mGrid);
    const int mBlocks = ceil_div(mTilesTotal, mTiles);
    for (int level = 0; hostDriven || level < maxLevels; ++level) {
      if (hostDriven) {
        int nseg = 0;
        NABO_CUDA_TRY(cudaMemcpyAsync(&nseg, &st->nseg, sizeof(int), cudaMemcpyDeviceToHost, stream));
        NABO_CUDA_TRY(cudaStreamSynchronize(stream));
        if (nseg == 0) break;
        if (level >= N) return set_error(kErrInternal, "kd-tree build: more levels than points");
      }
      NABO_CUDA_TRY(launch_pdl(k_median_cut<T, D>, ceil_div(segCap, 4), 128, 0, stream, cur, st, mb));
      NABO_CUDA_TRY(launch_pdl(k_median_sums<T, D>, mBlocks, kBlock, 0, stream, mb, nPad, cur, mTiles, blockSums,
                               segFirst, segLast, st));
      NABO_CUDA_TRY(launch_pdl(k_scan_block_sums, 1, kBlock, 0, stream, blockSums, mBlocks, st));
      NABO_CUDA_TRY(launch_pdl(k_median_split<T, D>, sg, 128, 0, stream, cur, nxt, st, small, marks, counters, dim,
                               bucket, smallMax, (int)segCap, (int)smallCap, (const int2*)blockSums, (const int2*)segFirst,
                               (const int2*)segLast, mTiles * kTile));
      NABO_CUDA_TRY(launch_pdl(median_scatter<T, D>(), mBlocks, kBlock, 0, stream, mb, recs, nPad, cur, nxt, mTiles,
                               (const int2*)blockSums, st));
      NABO_CUDA_TRY(launch_pdl(k_advance, 1, 1, 0, stream, st, counters));
      std::swap(cur, nxt);
    }
    k_median_flush<T, D><<<std::max(1, std::min(nb, 8 * sms)), kBlock, 0, stream>>>(mb, recs, n, st);
  }

  // small segments (their count is known on the device only): one wave of
  // resident blocks taking them from a counter
  MidArgs<T, D> ma = {};
  ma.recs = recs;
  ma.small = small;
  ma.marks = marks;
  ma.counters = counters;
  ma.nonFinite = nonFinite;
  ma.dim = dim;
  ma.bucket = bucket;
  ma.cap = smallMax;
  ma.claim = 16;
  ma.maxLevels = maxLevels;
  ma.splitRule = splitRule;
  const int midGrid = (int)std::min<int64_t>(smallCap, (int64_t)std::max(midOcc, 1) * sms);
  k_mid<T, D><<<midGrid, Mid::kThreads, midSmem, stream>>>(ma);
  NABO_CUDA_TRY(cudaGetLastError());

  k_leaf_ranks<<<rankBlocks, kRankBlock, 0, stream>>>(marks.leafBits, words, rank, rankSums);
  k_leaf_rank_sums<<<1, kRankBlock, 0, stream>>>(rankSums, rankBlocks, &st->nseg, counters, f->status);
  k_emit<T><<<ceil_div(std::max<int64_t>(n, 1), kBlock), kBlock, 0, stream>>>(
      marks, rank, rankSums, N, rankBlocks, dOff, nClouds, f->status, static_cast<Node<T>*>(f->nodes), f->nodeCap,
      f->nodeOffset);
  NABO_CUDA_TRY(cudaGetLastError());
  return kOk;
}

namespace {
// What a single-cloud build reads back, in one copy.
template <typename T>
struct BuildResult {
  int64_t off[2];
  int64_t nodeOffset[2];
  int status[4];
  T box[2 * kMaxDim];
};
template <typename T>
__global__ void k_one_cloud(BuildResult<T>* r, int64_t n) {
  r->off[0] = 0;
  r->off[1] = n;
}
}  // namespace

template <typename T, int D>
int build_kdtree(const T* dCloud, int64_t n, int64_t stride, int dim, unsigned bucketSize, cudaStream_t stream,
                 DeviceCloud* out, double* rootMin, double* rootMax, int splitRule) {
  Scratch sc(stream);
  ForestOut f;
  Rec<T, D>* recs = nullptr;
  Node<T>* nodes = nullptr;
  NABO_CUDA_TRY(object_alloc((void**)&recs, (size_t)n * sizeof(Rec<T, D>), stream));
  out->recs = recs;  // owned by the caller from here on
  // Upper bound on the node count: every leaf holds at least one point.
  const int64_t nodeCap = 2 * n;
  NABO_CUDA_TRY(object_alloc((void**)&nodes, (size_t)nodeCap * sizeof(Node<T>), stream));
  out->nodes = nodes;
  BuildResult<T>* res;
  NABO_CUDA_TRY(sc.get(&res, 1));
  k_one_cloud<T><<<1, 1, 0, stream>>>(res, n);
  NABO_CUDA_TRY(cudaGetLastError());
  f.recs = recs;
  f.nodes = nodes;
  f.nodeCap = nodeCap;
  f.nodeOffset = res->nodeOffset;
  f.status = res->status;
  f.rootLo = res->box;
  f.rootHi = res->box + kMaxDim;
  const int rc = build_forest<T, D>(dCloud, n, stride, dim, bucketSize, res->off, 1, -1, stream, &f, splitRule);
  if (rc != kOk) return rc;
  BuildResult<T> h;
  NABO_CUDA_TRY(cudaMemcpyAsync(&h, res, sizeof(h), cudaMemcpyDeviceToHost, stream));
  NABO_CUDA_TRY(cudaStreamSynchronize(stream));
  const int* hs = h.status;
  const T* hbox = h.box;
  const int64_t total = h.nodeOffset[1];
  if (hs[0]) return set_error(kErrArgument, "Cloud has non-finite (NaN or infinite) coordinates");
  if (hs[1]) return set_error(kErrInternal, "kd-tree build: internal check failed (capacity or pairing)");
  if (total <= 0 || total > nodeCap) return set_error(kErrInternal, "kd-tree build: inconsistent node count");
  if (total - 1 > (int64_t)kMaxNodeIndex)
    return set_error(kErrUnsupported, "kd-tree build: the tree has more nodes than the device layout indexes");
  out->nodeCount = total;
  out->height = hs[2];
  for (int d = 0; d < kMaxDim; ++d) {
    rootMin[d] = d < dim ? (double)hbox[d] : 0.0;
    rootMax[d] = d < dim ? (double)hbox[kMaxDim + d] : 0.0;
    // true bounds for query ordering: the root box's max is the true max
    // unless the quirk lifted it to numeric_limits<T>::min()
    out->lo[d] = rootMin[d];
    out->hi[d] = rootMax[d];
  }
  return kOk;
}

namespace {

// Float copies of double records (same order), for the search's float
// pre-filter of leaf points, and the largest coordinate magnitude over the
// searched dimensions (as float bits, atomicMax: non-negative floats order
// like their bit patterns). Coordinates beyond the float range become inf,
// which switches the pre-filter off.
template <int D>
__global__ void k_narrow(const Rec<double, D>* __restrict__ recs, int64_t n, int dim, Rec<float, D>* out,
                         unsigned* coordMaxBits) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  float m = 0.0f;
  if (p < n) {
    Rec<double, D> r;
    load_rec(recs, p, r);
    Rec<float, D> f;
#pragma unroll
    for (int c = 0; c < RecSize<float, D>::chunks; ++c) f.v[c] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int d = 0; d < D; ++d) {
      f.p.c[d] = (float)r.p.c[d];
      if (d < dim) m = fmaxf(m, fabsf(f.p.c[d]));
    }
    f.p.idx = r.p.idx;
    out[p] = f;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(kFull, m, o));
  if ((threadIdx.x & 31) == 0 && m > 0.0f) atomicMax(coordMaxBits, __float_as_uint(m));
}

}  // namespace

template <int D>
int narrow_records(const void* recs, int64_t n, int dim, void* recs32, float* coordMax, cudaStream_t stream) {
  NABO_CUDA_TRY(cudaMemsetAsync(coordMax, 0, sizeof(float), stream));
  if (n > 0)
    k_narrow<D><<<ceil_div(n, kBlock), kBlock, 0, stream>>>(static_cast<const Rec<double, D>*>(recs), n, dim,
                                                            static_cast<Rec<float, D>*>(recs32),
                                                            reinterpret_cast<unsigned*>(coordMax));
  NABO_CUDA_TRY(cudaGetLastError());
  return kOk;
}
template int narrow_records<2>(const void*, int64_t, int, void*, float*, cudaStream_t);
template int narrow_records<3>(const void*, int64_t, int, void*, float*, cudaStream_t);
template int narrow_records<4>(const void*, int64_t, int, void*, float*, cudaStream_t);
template int narrow_records<8>(const void*, int64_t, int, void*, float*, cudaStream_t);
template int narrow_records<16>(const void*, int64_t, int, void*, float*, cudaStream_t);

#define NABO_BUILD_INSTANTIATE(T, D)                                                                          \
  template int build_kdtree<T, D>(const T*, int64_t, int64_t, int, unsigned, cudaStream_t, DeviceCloud*,      \
                                  double*, double*, int);                                                      \
  template int build_forest<T, D>(const T*, int64_t, int64_t, int, unsigned, const int64_t*, int, int,        \
                                  cudaStream_t, ForestOut*, int);                                             \
  template int pack_cloud<T, D>(const T*, int64_t, int64_t, int, cudaStream_t, DeviceCloud*);

NABO_BUILD_INSTANTIATE(float, 2)
NABO_BUILD_INSTANTIATE(float, 3)
NABO_BUILD_INSTANTIATE(float, 4)
NABO_BUILD_INSTANTIATE(float, 8)
NABO_BUILD_INSTANTIATE(float, 16)
NABO_BUILD_INSTANTIATE(double, 2)
NABO_BUILD_INSTANTIATE(double, 3)
NABO_BUILD_INSTANTIATE(double, 4)
NABO_BUILD_INSTANTIATE(double, 8)
NABO_BUILD_INSTANTIATE(double, 16)

}  // namespace nabo_gb300
