// build_tree.cuh -- splitting, numbering and writing the trees of a forest
// build (included by build.cu only).
//
// Every split is recorded at its split position, the position p where the
// right child's points begin: exactly one inner node of the forest splits at
// a given p, and every p that is not a cloud's first point and begins a leaf
// is one. A leaf is recorded at its first position (a bit and its count of
// left turns). In pre-order, with every left child next to its parent, a
// node that begins at position a has the index
//     2 * (leaves that begin before a) + (left turns on its path) - cloud
// (each leaf before it closes two nodes but for the turns still open; cloud
// c's tree starts c nodes earlier than twice the leaves before it because c
// trees have one inner node fewer than leaves). So one count of leaf bits
// numbers all nodes of all trees at once, in any order, and no node is
// written before its final place is known.
#pragma once

#include "internal.cuh"

namespace nabo_gb300 {
namespace {

// An inner node at its split position: where its points begin, its left turns
// (minus its cloud's number) * 16 + cut dimension, its cut. A cloud's first
// position holds start = -1 and the cloud's number.
template <typename T>
struct Split;
template <>
struct alignas(16) Split<float> {
  int start;
  uint32_t turnsDim;
  float cut;
  int pad;
};
template <>
struct alignas(16) Split<double> {
  int start;
  uint32_t turnsDim;
  double cut;
};

template <typename T>
struct TreeMarks {
  Split<T>* split;     // [n]
  int* leafTurns;      // [n], valid where a leaf begins
  uint32_t* leafBits;  // [n / 32 + 1], zeroed
};

template <typename T>
__device__ __forceinline__ void mark_leaf(const TreeMarks<T>& m, int p, int turns) {
  m.leafTurns[p] = turns;
  atomicOr(m.leafBits + (p >> 5), 1u << (p & 31));
}
template <typename T>
__device__ __forceinline__ void mark_split(const TreeMarks<T>& m, int p, int start, int turns, int cd, T cut) {
  Split<T> s{};
  s.start = start;
  s.turnsDim = ((uint32_t)turns << 4) | (uint32_t)cd;
  s.cut = cut;
  m.split[p] = s;
}

// Segments small enough for k_mid: more than a bucket, at most its smallMax
// points. Boxes: 2 * D values each, lows then highs.
template <typename T>
struct SegList {
  int* start;
  int* count;
  int* turns;
  int* depth;
  T* box;
};

// Device counters of a build.
enum BuildCounter { kNextSegs = 0, kSmallCount = 1, kHeight = 2, kFlags = 3, kLevels = 4, kNextSmall = 5, kBuildCounters = 8 };

// The reference's split of a node (nabo/kdtree_cpu.cpp:126-190): the box
// midpoint along its widest dimension, clamped to the points' range.
enum SplitMode { kInside = 0, kBelowMin = 1, kAboveMax = 2 };

template <typename T, int D>
__device__ __forceinline__ int widest_dim(const T (&lo)[D], const T (&hi)[D], int dim, T* mid) {
  // first strict maximum, starting from 0 (nabo/kdtree_cpu.cpp:76-90)
  T best = T(0), l = lo[0], h = hi[0];
  int cd = 0;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const T ext = Ar<T>::sub(hi[d], lo[d]);
    if (d < dim && ext > best) {
      best = ext;
      cd = d;
      l = lo[d];
      h = hi[d];
    }
  }
  // (max + min) / 2 (nabo/kdtree_cpu.cpp:135); halving is exact
  *mid = Ar<T>::mul(Ar<T>::add(h, l), T(0.5));
  return cd;
}

// nabo/kdtree_cpu.cpp:180-190, with lt points below the cut and eq on it.
__device__ __forceinline__ int left_count(int mode, int count, int lt, int eq) {
  int l;
  if (mode == kBelowMin)
    l = 1;
  else if (mode == kAboveMax)
    l = count - 1;
  else if (lt > count / 2)
    l = lt;
  else if (lt + eq < count / 2)
    l = lt + eq;
  else
    l = count / 2;
  // finite coordinates guarantee 1 <= l < count; keep the split productive
  // whatever happens
  return l < 1 ? 1 : (l > count - 1 ? count - 1 : l);
}

template <typename T, int D>
__device__ __forceinline__ T coord_of(const Rec<T, D>& r, int cd) {
  T v = r.p.c[0];
#pragma unroll
  for (int d = 1; d < D; ++d) v = d == cd ? r.p.c[d] : v;
  return v;
}

// ---------------------------------------------------------------------------
// Top levels of the reference's rule: k_top.
//
// One cooperative launch runs all levels of all segments above smallMax
// points, however many (launches per level and pass, with a host read in
// between, cost 55-125 us a level). Each block owns `chunk` consecutive
// positions for the whole build, their records in shared memory when they
// fit, and keeps the segments that overlap them as its own list: every block
// of a segment takes the same decisions from the same numbers, so no segment
// table is shared. A level is
//   stats  each piece's coordinates along its segment's cut dimension: how
//          many lie below / on the box midpoint, the extremes and how many
//          lie there (enough for any of the three clamped cuts). A segment
//          that crosses chunks leaves each block's part where the others
//          find it by position: the piece that began in an earlier chunk is
//          the chunk's head, the one that goes on into the next its tail.
//   send   the segment's totals and the counts before this chunk, then the
//          reference's partition (nabo/kdtree_cpu.cpp:149-177): with C(p)
//          elements passing the test before position p of the segment and
//          `mid` in all, a failing element at p < mid is the (p - C)-th
//          misplaced from the left, a passing one at p >= mid the
//          (mid - 1 - C)-th from the right; each writes its record to that
//          slot of its side in the segment's part of the exchange buffer
//   take   each misplaced position reads the record of the same slot of the
//          other side; the split is recorded and the children become leaves,
//          small segments or the pieces of the next level
// with a grid barrier after `send` and after the next `stats`: a level is
// bound by these and a few dependent L2 reads, not by its data: 10 us a level
// at 83 k lidar points (13 levels), 18 us at 1.15 M (18 levels, 7,560 records
// a block).
// The reference partitions twice, by v < cut and then [lt, count) by v <= cut.
// A clamped cut needs one of the two only: below the minimum nothing is
// smaller than the cut, above the maximum nothing is greater. The second
// pass (count, send and take once more) runs on levels where some unclamped
// cut has points on it.
constexpr int kTopThreads = 1024;
constexpr int kTopWarps = kTopThreads / 32;
constexpr int kTopMinChunk = 1024;
constexpr size_t kTopSmemMax = 200 * 1024;

template <typename T, int D>
struct TopSeg {
  int start, count, turns, depth;
  T lo[D], hi[D];
};
template <typename T>
struct TopTask {
  T mn, mx;
  int nmn, nmx, lt, eq;
};
template <typename T>
struct TopInfo {
  T cut;
  int cd, mode, mid, lt, eq, before, votesAt;
};
struct TopState {
  int active[4];  // blocks with pieces at level l in [l & 3]
  int second[4];  // level l has a second pass
  unsigned barrier;
  int pad[7];
};
template <typename T, int D>
struct TopArgs {
  Rec<T, D>* recs;
  Rec<T, D>* exch;  // [n]
  unsigned char* work;  // kTopGlobal: workBytes per block
  int64_t workBytes;
  TopTask<T>* head;  // [blocks]
  TopTask<T>* tail;
  int* head2;
  int* tail2;
  const int64_t* off;
  const T* rootLo;
  const T* rootHi;
  SegList<T> small;
  TreeMarks<T> marks;
  TopState* st;
  int* counters;
  const int* nonFinite;  // stop at once if set (null: never)
  int n, nClouds, dim, chunk, pieces, smallMax, bucket, maxLevels, smallCap, barrierPolls;
};

// A block's working memory: the chunk's records (when resident), two lists of
// pieces, their split, statistics and per-warp counts, the partition votes.
// With the records and the lists in shared memory, only the lists there
// (chunks of many records), or nothing (hundreds of millions of points).
enum TopMode { kTopResident = 0, kTopLists = 1, kTopGlobal = 2 };
template <typename T, int D>
struct TopShape {
  static constexpr size_t bytes(int64_t chunk, int64_t pieces, bool resident) {
    return ((resident ? (size_t)chunk * sizeof(Rec<T, D>) : 0) +
            (size_t)pieces * (2 * sizeof(TopSeg<T, D>) + sizeof(TopInfo<T>) + sizeof(TopTask<T>) +
                              kTopWarps * sizeof(int)) +
            (size_t)(chunk / 32 + 1 + pieces) * sizeof(uint32_t) + 63) / 64 * 64;
  }
};

// Waits until every block has arrived as often as this one (all blocks are
// resident: cooperative launch). False after that many polls, and then in
// every block: one that gives up takes its arrival back, unless all have
// arrived by then, so that no other passes. The blocks then leave one after
// another, every record still in one place, and the build reports that it did
// not finish.
__device__ __forceinline__ bool grid_barrier(unsigned* count, unsigned target, int polls) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(count, 1u);
    int good = 0;
    for (int i = 0; i < polls && !good; ++i) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
      good = (int)(v - target) >= 0;
    }
    if (!good) {
      for (unsigned v = atomicAdd(count, 0u); !(good = (int)(v - target) >= 0);) {
        const unsigned old = atomicCAS(count, v, v - 1u);
        if (old == v) break;
        v = old;
      }
    }
    __threadfence();
    ok = good;
  }
  __syncthreads();
  return ok;
}

template <typename T>
__device__ __forceinline__ void merge_min(T& a, int& na, T b, int nb) {
  na = b < a ? nb : (b == a ? na + nb : na);
  a = b < a ? b : a;
}
template <typename T>
__device__ __forceinline__ void merge_max(T& a, int& na, T b, int nb) {
  na = b > a ? nb : (b == a ? na + nb : na);
  a = b > a ? b : a;
}
template <typename T>
__device__ __forceinline__ void merge_task(TopTask<T>& a, const TopTask<T>& b) {
  merge_min(a.mn, a.nmn, b.mn, b.nmn);
  merge_max(a.mx, a.nmx, b.mx, b.nmx);
  a.lt += b.lt;
  a.eq += b.eq;
}
template <typename T>
__device__ __forceinline__ TopTask<T> empty_task() {
  return {std::numeric_limits<T>::max(), std::numeric_limits<T>::lowest(), 0, 0, 0, 0};
}
template <typename T>
__device__ __forceinline__ TopTask<T> warp_merge(TopTask<T> a) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    TopTask<T> b;
    b.mn = __shfl_xor_sync(kFull, a.mn, o);
    b.mx = __shfl_xor_sync(kFull, a.mx, o);
    b.nmn = __shfl_xor_sync(kFull, a.nmn, o);
    b.nmx = __shfl_xor_sync(kFull, a.nmx, o);
    b.lt = __shfl_xor_sync(kFull, a.lt, o);
    b.eq = __shfl_xor_sync(kFull, a.eq, o);
    merge_task(a, b);
  }
  return a;
}

// Appends a segment to k_mid's list.
template <typename T, int D>
__device__ __forceinline__ void list_small(const TopArgs<T, D>& a, const TopSeg<T, D>& c) {
  const int id = atomicAdd(a.counters + kSmallCount, 1);
  if (id >= a.smallCap) {
    atomicOr(a.counters + kFlags, 1);
    return;
  }
  a.small.start[id] = c.start;
  a.small.count[id] = c.count;
  a.small.turns[id] = c.turns;
  a.small.depth[id] = c.depth;
  T* box = a.small.box + (int64_t)id * 2 * D;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    box[d] = c.lo[d];
    box[D + d] = c.hi[d];
  }
}

template <typename T, int D, int MODE>
__global__ void __launch_bounds__(kTopThreads, 1) k_top(const TopArgs<T, D> a) {
  using Seg = TopSeg<T, D>;
  constexpr bool RESIDENT = MODE == kTopResident;
  extern __shared__ __align__(16) unsigned char topSmem[];
  __shared__ int listCount[2];
  __shared__ TopTask<T> part[kTopWarps];
  if (a.nonFinite && *a.nonFinite) return;  // uniform over the grid
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t below = (1u << lane) - 1u;
  const int me = blockIdx.x;
  const int c0 = me * a.chunk, c1 = (int)min((int64_t)a.n, (int64_t)c0 + a.chunk);
  unsigned char* const base = MODE == kTopGlobal ? a.work + a.workBytes * blockIdx.x : topSmem;
  Rec<T, D>* const own = reinterpret_cast<Rec<T, D>*>(base);
  // position p's record: data[p - c0]
  Rec<T, D>* const data = RESIDENT ? own : a.recs + c0;
  Seg* const list0 = reinterpret_cast<Seg*>(own + (RESIDENT ? a.chunk : 0));
  Seg* const list1 = list0 + a.pieces;
  TopInfo<T>* const info = reinterpret_cast<TopInfo<T>*>(list1 + a.pieces);
  TopTask<T>* const stat = reinterpret_cast<TopTask<T>*>(info + a.pieces);
  int* const warpBefore = reinterpret_cast<int*>(stat + a.pieces);  // [piece][warp]
  uint32_t* const votes = reinterpret_cast<uint32_t*>(warpBefore + a.pieces * kTopWarps);
  unsigned arrive = 0;
  const auto barrier = [&]() {
    arrive += gridDim.x;
    if (grid_barrier(&a.st->barrier, arrive, a.barrierPolls)) return true;
    if (threadIdx.x == 0) atomicOr(a.counters + kFlags, 1);
    return false;
  };
  const auto crosses = [&](const Seg& S) { return S.start < c0 || S.start + S.count > c1; };

  if (RESIDENT)
    for (int i = threadIdx.x; i < c1 - c0; i += kTopThreads) own[i] = a.recs[c0 + i];
  // the clouds that overlap the chunk and are no leaf or small segment
  if (threadIdx.x < 2) listCount[threadIdx.x] = 0;
  __syncthreads();
  for (int c = cloud_of(a.off, a.nClouds, c0) + threadIdx.x; c < a.nClouds && a.off[c] < c1; c += kTopThreads) {
    const int64_t count = a.off[c + 1] - a.off[c];
    if (count <= a.smallMax || count <= a.bucket) continue;
    Seg S;
    S.start = (int)a.off[c];
    S.count = (int)count;
    S.turns = -c;
    S.depth = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      S.lo[d] = d < a.dim ? a.rootLo[(int64_t)c * kMaxDim + d] : T(0);
      S.hi[d] = d < a.dim ? a.rootHi[(int64_t)c * kMaxDim + d] : T(0);
    }
    const int i = atomicAdd(&listCount[0], 1);
    if (i < a.pieces) list0[i] = S;
  }
  __syncthreads();

  // One pass's votes (`first`) and ranks over this chunk's part of a segment,
  // from its position o on (start, or start + lt for the second pass); `f` is
  // called with (local index, misplaced on the left, slot of its side, slot
  // of the other side) for every misplaced position.
  const auto walk = [&](int i, const Seg& S, int o, int mid, bool lessEq, bool first, auto&& f) {
    const TopInfo<T>& I = info[i];
    const int lo = max(o, c0), hi = min(S.start + S.count, c1);
    const int len = hi - lo;
    if (len <= 0) return;  // uniform over the block
    const int rounds = (len + kTopThreads - 1) / kTopThreads;
    uint32_t* const mine = votes + I.votesAt + warp * rounds;
    const int run = lo - c0 + warp * rounds * 32;  // this warp's positions
    const int at = run + lane;
    if (first) {
      const T cut = I.cut;
      const int cd = I.cd;
      int sum = 0;
      for (int r = 0; r < rounds && run + r * 32 < hi - c0; ++r) {
        const int x = at + r * 32;
        bool pass = false;
        if (x < hi - c0) {
          const T v = data[x].p.c[cd];
          pass = lessEq ? v <= cut : v < cut;
        }
        const uint32_t b = __ballot_sync(kFull, pass);
        if (lane == 0) mine[r] = b;
        sum += __popc(b);
      }
      if (lane == 0) warpBefore[i * kTopWarps + warp] = sum;
      __syncthreads();
      if (warp == 0) {
        const int s = warpBefore[i * kTopWarps + lane];
        int inc = s;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int y = __shfl_up_sync(kFull, inc, d);
          if (lane >= d) inc += y;
        }
        warpBefore[i * kTopWarps + lane] = I.before + inc - s;
      }
      __syncthreads();
    }
    const int half = (S.start + S.count - o) / 2;
    int c = warpBefore[i * kTopWarps + warp];
    if (first) __syncwarp();
    for (int r = 0; r < rounds && run + r * 32 < hi - c0; ++r) {
      const int x = at + r * 32;
      const uint32_t b = mine[r];
      const int ci = c + __popc(b & below);
      const int p = x + c0 - o;
      const bool pass = (b >> lane) & 1u;
      if (x < hi - c0) {
        if (p < mid && !pass) f(x, o + p - ci, o + half + p - ci);
        if (p >= mid && pass) f(x, o + half + mid - 1 - ci, o + mid - 1 - ci);
      }
      c += __popc(b);
    }
  };
  const auto send = [&](int x, int slot, int) { a.exch[slot] = data[x]; };
  const auto take = [&](int x, int, int slot) { data[x] = a.exch[slot]; };

  int level = 0;
  for (;; ++level) {
    Seg* const list = (level & 1) ? list1 : list0;
    Seg* const nextList = (level & 1) ? list0 : list1;
    const int np = min(listCount[level & 1], a.pieces);
    // stats
    for (int i = 0; i < np; ++i) {
      const Seg& S = list[i];
      T ideal;
      const int cd = widest_dim<T, D>(S.lo, S.hi, a.dim, &ideal);
      TopTask<T> m = empty_task<T>();
      const int hi = min(S.start + S.count, c1) - c0;
      for (int x = max(S.start, c0) - c0 + (int)threadIdx.x; x < hi; x += kTopThreads) {
        const T v = data[x].p.c[cd];
        merge_min(m.mn, m.nmn, v, 1);
        merge_max(m.mx, m.nmx, v, 1);
        m.lt += v < ideal ? 1 : 0;
        m.eq += v == ideal ? 1 : 0;
      }
      m = warp_merge(m);
      if (lane == 0) part[warp] = m;
      __syncthreads();
      if (warp == 0) {
        m = warp_merge(part[lane]);
        if (lane == 0) {
          stat[i] = m;
          if (crosses(S)) (S.start < c0 ? a.head : a.tail)[me] = m;
        }
      }
      __syncthreads();
    }
    if (threadIdx.x == 0 && np > 0) atomicAdd(&a.st->active[level & 3], 1);
    if (!barrier()) return;
    if (a.st->active[level & 3] == 0) break;
    if (a.maxLevels >= 0 && level >= a.maxLevels) {
      if (me == 0 && threadIdx.x == 0) atomicOr(a.counters + kFlags, 1);
      break;
    }
    if (me == 0 && threadIdx.x == 0) {  // read last two levels ago, next written in the next one
      a.st->active[(level + 2) & 3] = 0;
      a.st->second[(level + 2) & 3] = 0;
    }
    // the segments' totals, a warp each
    for (int i = warp; i < np; i += kTopWarps) {
      const Seg& S = list[i];
      T ideal;
      const int cd = widest_dim<T, D>(S.lo, S.hi, a.dim, &ideal);
      TopTask<T> all = empty_task<T>(), pre = empty_task<T>();
      if (crosses(S)) {
        const int ks = S.start / a.chunk, ke = (S.start + S.count - 1) / a.chunk;
        for (int k = ks + lane; k <= ke; k += 32) {
          const TopTask<T> e = k == ks ? a.tail[k] : a.head[k];
          merge_task(all, e);
          if (k < me) merge_task(pre, e);
        }
        all = warp_merge(all);
        pre = warp_merge(pre);
      } else {
        all = stat[i];
      }
      // the piece's votes: a word per 32 positions, the pieces in order, one
      // word more for each earlier one
      int rank = 0;
      for (int j = lane; j < np; j += 32) rank += list[j].start < S.start ? 1 : 0;
      rank = __reduce_add_sync(kFull, rank);
      if (lane == 0) {
        TopInfo<T> I;
        I.votesAt = ((max(S.start, c0) - c0) >> 5) + rank;
        I.cd = cd;
        I.mode = ideal < all.mn ? kBelowMin : (ideal > all.mx ? kAboveMax : kInside);
        I.cut = I.mode == kBelowMin ? all.mn : (I.mode == kAboveMax ? all.mx : ideal);
        I.lt = I.mode == kBelowMin ? 0 : all.lt - (I.mode == kAboveMax ? all.nmx : 0);
        I.eq = I.mode == kBelowMin ? all.nmn : (I.mode == kAboveMax ? all.nmx : all.eq);
        I.mid = I.mode == kBelowMin ? I.eq : I.lt;
        I.before = I.mode == kBelowMin ? (pre.mn == I.cut ? pre.nmn : 0)
                                       : pre.lt - (I.mode == kAboveMax && pre.mx == I.cut ? pre.nmx : 0);
        info[i] = I;
        if (I.mode == kInside && I.eq > 0) a.st->second[level & 3] = 1;
      }
    }
    __syncthreads();
    for (int i = 0; i < np; ++i) walk(i, list[i], list[i].start, info[i].mid, info[i].mode == kBelowMin, true, send);
    if (!barrier()) return;
    const bool second = a.st->second[level & 3] != 0;
    for (int i = 0; i < np; ++i) walk(i, list[i], list[i].start, info[i].mid, info[i].mode == kBelowMin, false, take);
    __syncthreads();
    if (second) {  // the segments with points on an unclamped cut: [lt, count) by v <= cut
      const auto again = [&](int i) { return info[i].mode == kInside && info[i].eq > 0; };
      for (int i = 0; i < np; ++i) {
        if (!again(i)) continue;  // uniform over the block
        const Seg& S = list[i];
        const TopInfo<T>& I = info[i];
        const int hi = min(S.start + S.count, c1) - c0;
        int c = 0;
        for (int x = max(S.start + I.lt, c0) - c0 + (int)threadIdx.x; x < hi; x += kTopThreads)
          c += data[x].p.c[I.cd] <= I.cut ? 1 : 0;
        c = __reduce_add_sync(kFull, c);
        if (lane == 0) part[warp].eq = c;
        __syncthreads();
        if (warp == 0) {
          c = __reduce_add_sync(kFull, part[lane].eq);
          if (lane == 0 && crosses(S)) (S.start < c0 ? a.head2 : a.tail2)[me] = c;
        }
        __syncthreads();
      }
      if (!barrier()) return;
      for (int i = warp; i < np; i += kTopWarps) {
        if (!again(i)) continue;
        const Seg& S = list[i];
        int pre = 0;
        if (crosses(S)) {
          const int ks = S.start / a.chunk;
          for (int k = ks + lane; k < me; k += 32) pre += k == ks ? a.tail2[k] : a.head2[k];
          pre = __reduce_add_sync(kFull, pre);
        }
        if (lane == 0) info[i].before = pre;
      }
      __syncthreads();
      for (int i = 0; i < np; ++i)
        if (again(i)) walk(i, list[i], list[i].start + info[i].lt, info[i].eq, true, true, send);
      if (!barrier()) return;
      for (int i = 0; i < np; ++i)
        if (again(i)) walk(i, list[i], list[i].start + info[i].lt, info[i].eq, true, false, take);
      __syncthreads();
    }
    // the splits, recorded by the block that holds the position concerned
    if (threadIdx.x == 0) listCount[level & 1] = 0;
    for (int i = threadIdx.x; i < np; i += kTopThreads) {
      const Seg S = list[i];
      const TopInfo<T> I = info[i];
      const int leftCount = left_count(I.mode, S.count, I.lt, I.eq);
      const int split = S.start + leftCount;
      if (split >= c0 && split < c1) mark_split(a.marks, split, S.start, S.turns, I.cd, I.cut);
      for (int side = 0; side < 2; ++side) {
        Seg c = S;
        c.start = side ? split : S.start;
        c.count = side ? S.count - leftCount : leftCount;
        c.turns = side ? S.turns : S.turns + 1;
        c.depth = S.depth + 1;
#pragma unroll
        for (int d = 0; d < D; ++d) {
          c.lo[d] = side && d == I.cd ? I.cut : S.lo[d];
          c.hi[d] = !side && d == I.cd ? I.cut : S.hi[d];
        }
        const bool begins = c.start >= c0 && c.start < c1;
        if (c.count <= a.bucket) {
          if (begins) {
            mark_leaf(a.marks, c.start, c.turns);
            atomicMax(a.counters + kHeight, c.depth);
          }
        } else if (c.count <= a.smallMax) {
          if (begins) list_small(a, c);
        } else if (c.start < c1 && c.start + c.count > c0) {
          const int j = atomicAdd(&listCount[(level + 1) & 1], 1);
          if (j < a.pieces)
            nextList[j] = c;
          else
            atomicOr(a.counters + kFlags, 1);  // unreachable
        }
      }
    }
    __syncthreads();
  }
  if (RESIDENT)
    for (int i = threadIdx.x; i < c1 - c0; i += kTopThreads) a.recs[c0 + i] = own[i];
  if (me == 0 && threadIdx.x == 0) atomicMax(a.counters + kLevels, level);
}

// ---------------------------------------------------------------------------
// Small segments: k_mid.
//
// A block stages segments in shared memory and splits them down to leaves.
// Nodes of more than 32 points are split by a warp each, a generation of
// nodes at a time (the warps take the nodes of a list and append the children
// to the next one). Nodes of 9 to 32 points (above the bucket size, in
// general) are packed into windows of 32 consecutive positions, one point per
// lane, and split all at once, level by level, with ballots, shuffles and
// segmented scans: a warp does for a whole window what one node at a time
// took it, and no stack is kept. The splits are the reference's recursion
// (nabo/kdtree_cpu.cpp:110-225), or the median rule's. Bound by the latency of
// its dependent shared-memory and shuffle steps. (Search-ready tree from a
// device cloud, level launches and a warp per 256-point segment -> k_top,
// k_mid and k_emit: 83 k lidar points 1.31 -> 0.26 ms of kernels, 1.15 M
// points 2.9 -> 0.55 ms. Segments of 4096, 3072 and 2048 points, 256 to 1024
// threads: the whole build within 3 % at 83 k points, 4096 and 512 the
// fastest at 1.15 M.)
template <typename T, int D>
struct MidNode {
  int st, count, turns, depth;
  int delta;  // global position - slot position
  T lo[D], hi[D];
};

template <typename T, int D>
struct MidShape {
  static constexpr int kThreads = sizeof(Rec<T, D>) <= 32 ? 512 : 256;
  static constexpr int kBlocks = sizeof(Rec<T, D>) <= 16 ? 2 : 1;  // per SM at least
  // largest segment of the reference's rule
  static constexpr int kMax = sizeof(Rec<T, D>) <= 16   ? 4096
                              : sizeof(Rec<T, D>) <= 48 ? 2048
                              : sizeof(Rec<T, D>) <= 80 ? 1024
                                                        : 512;
  static constexpr int nodes(int cap) { return cap / 33 + 2; }
  static constexpr int jobs(int cap, int bucket) { return bucket < 32 ? cap / (bucket + 1) + 2 : 1; }
  static constexpr size_t smem(int cap, int bucket) {
    return (size_t)cap * sizeof(Rec<T, D>) + (size_t)(2 * nodes(cap) + jobs(cap, bucket)) * sizeof(MidNode<T, D>) +
           (size_t)cap * 2 * sizeof(uint16_t);
  }
};

template <typename T, int D>
struct MidArgs {
  Rec<T, D>* recs;
  SegList<T> small;
  TreeMarks<T> marks;
  int* counters;
  const int* nonFinite;
  int dim, bucket, cap, claim, maxLevels, splitRule;
};

// The i-th misplaced element from the left of a node trades with the i-th
// from the right (see k_top), by a warp on pts[lo, hi): `mid` elements pass.
// tab: hi - lo entries.
template <typename T, int D>
__device__ __forceinline__ void warp_partition(Rec<T, D>* pts, int count, int mid, int cd, T cut, bool lessEq,
                                               uint16_t* tab, int lane) {
  if (mid == 0 || mid == count) return;
  const unsigned below = (1u << lane) - 1u;
  uint16_t* tabB = tab + count / 2;
  int c = 0, moved = 0;
  for (int c0 = 0; c0 < count; c0 += 32) {
    const int i = c0 + lane;
    bool pass = false;
    if (i < count) {
      const T v = pts[i].p.c[cd];
      pass = lessEq ? v <= cut : v < cut;
    }
    const unsigned b = __ballot_sync(kFull, pass);
    const int ci = c + __popc(b & below);
    if (i < mid && !pass) tab[i - ci] = (uint16_t)i;
    if (i >= mid && i < count && pass) tabB[mid - 1 - ci] = (uint16_t)i;
    if (c0 <= mid && mid < c0 + 32) moved = mid - (c + __popc(b & ((1u << (mid - c0)) - 1u)));
    c += __popc(b);
  }
  __syncwarp();
  for (int j = lane; j < moved; j += 32) {
    const int x = tab[j], y = tabB[j];
    const Rec<T, D> r = pts[x];
    pts[x] = pts[y];
    pts[y] = r;
  }
  __syncwarp();
}

__device__ __forceinline__ float warp_min_val(float v) { return ordered_val(__reduce_min_sync(kFull, ordered_key(v)), 0.0f); }
__device__ __forceinline__ float warp_max_val(float v) { return ordered_val(__reduce_max_sync(kFull, ordered_key(v)), 0.0f); }
__device__ __forceinline__ double warp_min_val(double v) { return warp_min(v); }
__device__ __forceinline__ double warp_max_val(double v) { return warp_max(v); }

__device__ __forceinline__ uint32_t warp_or(uint32_t v) { return __reduce_or_sync(kFull, v); }
__device__ __forceinline__ uint32_t warp_and(uint32_t v) { return __reduce_and_sync(kFull, v); }
__device__ __forceinline__ unsigned long long warp_or(unsigned long long v) {
  return (unsigned long long)warp_or((uint32_t)(v >> 32)) << 32 | warp_or((uint32_t)v);
}
__device__ __forceinline__ unsigned long long warp_and(unsigned long long v) {
  return (unsigned long long)warp_and((uint32_t)(v >> 32)) << 32 | warp_and((uint32_t)v);
}

// The middle one of 31 values sampled evenly, as the median rule's top levels
// take it.
template <typename T, int D>
__device__ __forceinline__ T warp_sampled_median(const Rec<T, D>* node, int count, int cd, int lane) {
  using Key = typename KeyOf<T>::type;
  Key e[1] = {lane < kMedianSamples ? ordered_key(node[(int)((int64_t)(2 * lane + 1) * count / (2 * kMedianSamples))].p.c[cd])
                                    : ~Key(0)};
  warp_sort_keys<1>(e, lane);
  return ordered_val(__shfl_sync(kFull, e[0], kMedianSamples / 2), T(0));
}

// The lower median (rank count / 2) of up to kHeld values, by a warp holding
// every 32nd of them in each lane: bit by bit below the bits that all keys
// share, until one candidate is left (about 11 rounds instead of a bit each).
// Instantiated for 64, 128 and 256 values: most nodes have far fewer than 256
// (k_mid of a 512-cloud, 22 M-point build: 2.75 -> 2.64 ms).
constexpr int kHeld = 256;
template <int kPer, typename T, int D>
__device__ __forceinline__ T warp_median_of(const Rec<T, D>* node, int count, int cd, int lane) {
  using Key = typename KeyOf<T>::type;
  Key k[kPer];
  Key any = 0, all = ~Key(0);
  unsigned alive = 0;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    k[j] = 0;
    if (lane + 32 * j < count) {
      k[j] = ordered_key(node[lane + 32 * j].p.c[cd]);
      any |= k[j];
      all &= k[j];
      alive |= 1u << j;
    }
  }
  any = warp_or(any);
  const Key diff = any & ~warp_and(all);  // bits in which some keys differ
  int left = count, want = count / 2;
  for (int b = 8 * (int)sizeof(Key) - 1; b >= 0 && left > 1; --b) {
    if (!((diff >> b) & 1)) continue;
    unsigned zeros = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) zeros |= ((k[j] >> b) & 1) ? 0u : 1u << j;
    zeros &= alive;
    const int c = __reduce_add_sync(kFull, __popc(zeros));
    if (want < c) {
      alive = zeros;
      left = c;
    } else {
      want -= c;
      alive &= ~zeros;
      left -= c;
    }
  }
  Key m = k[0];
#pragma unroll
  for (int j = 1; j < kPer; ++j)
    if ((alive & ((1u << j) - 1u)) == 0u) m = k[j];
  const int src = __ffs(__ballot_sync(kFull, alive != 0u)) - 1;
  return ordered_val(__shfl_sync(kFull, m, src), T(0));
}
template <typename T, int D>
__device__ __forceinline__ T warp_median(const Rec<T, D>* node, int count, int cd, int lane) {
  if (count <= 64) return warp_median_of<2>(node, count, cd, lane);
  if (count <= 128) return warp_median_of<4>(node, count, cd, lane);
  return warp_median_of<kHeld / 32>(node, count, cd, lane);
}

// Splits a node, by a warp, at `ideal` (the median rule: just above it, so
// that points equal to it go left and hardly any lies on the cut) and
// partitions by v < cut, or v <= cut below the minimum. Returns the mode.
// `sampled`: a sampled median with nothing above it divides the points on it
// by position.
template <typename T, int D>
__device__ __forceinline__ int split_node(Rec<T, D>* pts, int count, int cd, T ideal, bool sampled, uint16_t* tab,
                                          int lane, T* cutOut, int* ltOut, int* eqOut) {
  T mn = std::numeric_limits<T>::max(), mx = std::numeric_limits<T>::lowest();
  int lt = 0, eq = 0;
#pragma unroll 4
  for (int j = lane; j < count; j += 32) {
    const T v = pts[j].p.c[cd];
    mn = v < mn ? v : mn;
    mx = v > mx ? v : mx;
    lt += v < ideal ? 1 : 0;
    eq += v == ideal ? 1 : 0;
  }
  mn = warp_min_val(mn);
  mx = warp_max_val(mx);
  lt = __reduce_add_sync(kFull, lt);
  eq = __reduce_add_sync(kFull, eq);
  int mode = kInside;
  T cut = ideal;
  if (ideal < mn || ideal > mx) {  // the points on a clamped cut
    mode = ideal < mn ? kBelowMin : kAboveMax;
    cut = ideal < mn ? mn : mx;
    eq = 0;
    for (int j = lane; j < count; j += 32) eq += pts[j].p.c[cd] == cut ? 1 : 0;
    eq = __reduce_add_sync(kFull, eq);
    lt = mode == kBelowMin ? 0 : lt - eq;  // above the maximum, lt counted every point
    if (sampled) mode = kInside;
  }
  *cutOut = cut;
  *ltOut = lt;
  *eqOut = eq;
  const bool lessEq = mode == kBelowMin;
  warp_partition<T, D>(pts, count, lessEq ? eq : lt, cd, cut, lessEq, tab, lane);
  return mode;
}

// A record from another lane.
template <typename T, int D>
__device__ __forceinline__ Rec<T, D> shfl_rec(const Rec<T, D>& r, int src) {
  Rec<T, D> o;
#pragma unroll
  for (int c = 0; c < RecSize<T, D>::chunks; ++c) {
    o.v[c].x = __shfl_sync(kFull, r.v[c].x, src);
    o.v[c].y = __shfl_sync(kFull, r.v[c].y, src);
    o.v[c].z = __shfl_sync(kFull, r.v[c].z, src);
    o.v[c].w = __shfl_sync(kFull, r.v[c].w, src);
  }
  return o;
}

template <typename T, int D>
__global__ void __launch_bounds__(MidShape<T, D>::kThreads, MidShape<T, D>::kBlocks) k_mid(const MidArgs<T, D> a) {
  using Node = MidNode<T, D>;
  extern __shared__ __align__(16) unsigned char midSmem[];
  __shared__ int listCount[2], jobCount, claimAt, take, total;
  __shared__ int slotOf[32], startOf[32], countOf[32];
  if (a.nonFinite && *a.nonFinite) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int nodeCap = MidShape<T, D>::nodes(a.cap);
  Rec<T, D>* const pts = reinterpret_cast<Rec<T, D>*>(midSmem);
  Node* const list0 = reinterpret_cast<Node*>(pts + a.cap);
  Node* const list1 = list0 + nodeCap;
  Node* const jobs = list1 + nodeCap;
  uint16_t* const tab = reinterpret_cast<uint16_t*>(jobs + MidShape<T, D>::jobs(a.cap, a.bucket));
  uint16_t* const jobAt = tab + a.cap;
  const int nS = a.counters[kSmallCount];
  // segments a block claims at once: many when there are enough for every
  // block, one when there are few
  const int claim = max(1, min(a.claim, nS / (2 * (int)gridDim.x)));
  const unsigned below = (1u << lane) - 1u;
  int hmax = 0, levels = 0;

  // A child (or a segment itself): a leaf, a window's node, or a node of `next`.
  const auto add = [&](const Node& c, int next) {
    if (c.count <= a.bucket) {
      mark_leaf(a.marks, c.st + c.delta, c.turns);
      hmax = max(hmax, c.depth);
    } else if (c.count <= 32) {
      const int j = atomicAdd(&jobCount, 1);
      jobs[j] = c;
      jobAt[c.st] = (uint16_t)j;
    } else {
      const int i = atomicAdd(&listCount[next], 1);
      (next ? list1 : list0)[i] = c;
    }
  };

  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) claimAt = atomicAdd(a.counters + kNextSmall, claim);
    __syncthreads();
    const int c0 = claimAt;
    if (c0 >= nS) break;
    const int cN = min(claim, nS - c0);
    for (int done = 0; done < cN;) {
      // as many of the claimed segments as fit
      if (warp == 0) {
        const int id = c0 + done + lane;
        const int n = done + lane < cN ? a.small.count[id] : 0;
        int inc = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(kFull, inc, o);
          if (lane >= o) inc += y;
        }
        const unsigned fit = __ballot_sync(kFull, n > 0 && inc <= a.cap);
        const int k = __popc(fit);
        slotOf[lane] = inc - n;
        startOf[lane] = n > 0 ? a.small.start[id] : 0;
        countOf[lane] = n;
        if (lane == 0) {
          take = k;
          jobCount = 0;
          listCount[0] = listCount[1] = 0;
        }
        if (lane == k - 1) total = inc;
      }
      __syncthreads();
      const int k = take;
      if (k == 0) {  // unreachable: every small segment fits
        if (threadIdx.x == 0) atomicOr(a.counters + kFlags, 2);
        break;
      }
      const int all = total;
      for (int i = threadIdx.x; i < all; i += blockDim.x) jobAt[i] = 0xffffu;
      for (int s = 0; s < k; ++s) {
        const Rec<T, D>* src = a.recs + startOf[s];
        Rec<T, D>* dst = pts + slotOf[s];
        for (int i = threadIdx.x; i < countOf[s]; i += blockDim.x) dst[i] = src[i];
      }
      __syncthreads();
      if ((int)threadIdx.x < k) {
        const int id = c0 + done + threadIdx.x;
        Node r;
        r.st = slotOf[threadIdx.x];
        r.count = countOf[threadIdx.x];
        r.turns = a.small.turns[id];
        r.depth = a.small.depth[id];
        r.delta = startOf[threadIdx.x] - r.st;
        const T* box = a.small.box + (int64_t)id * 2 * D;
#pragma unroll
        for (int d = 0; d < D; ++d) {
          r.lo[d] = box[d];
          r.hi[d] = box[D + d];
        }
        add(r, 0);
      }
      // nodes of more than 32 points, a generation at a time
      for (int cur = 0;; cur ^= 1) {
        __syncthreads();
        const int nc = listCount[cur];
        if (nc == 0) break;
        for (int i = warp; i < nc; i += warps) {
          Node N = (cur ? list1 : list0)[i];
          Rec<T, D>* node = pts + N.st;
          const int count = N.count;
          if (count > 256) {  // the levels nabo_cuda_batch_create's maxLevels limits
            levels = max(levels, N.depth + 1);
            if (a.maxLevels >= 0 && N.depth >= a.maxLevels) {
              if (lane == 0) {
                atomicOr(a.counters + kFlags, 1);
                mark_leaf(a.marks, N.st + N.delta, N.turns);
              }
              continue;
            }
          }
          T ideal;
          const int cd = widest_dim<T, D>(N.lo, N.hi, a.dim, &ideal);
          int mode, lt, eq;
          T cut;
          const bool median = a.splitRule == 1, sampled = median && count > kHeld;
          if (median)
            ideal = next_up(sampled ? warp_sampled_median(node, count, cd, lane) : warp_median(node, count, cd, lane));
          mode = split_node<T, D>(node, count, cd, ideal, sampled, tab + N.st, lane, &cut, &lt, &eq);
          if (mode == kInside && eq > 0)
            warp_partition<T, D>(node + lt, count - lt, eq, cd, cut, true, tab + N.st + lt, lane);
          const int l = left_count(mode, count, lt, eq);
          if (lane == 0) mark_split(a.marks, N.st + l + N.delta, N.st + N.delta, N.turns, cd, cut);
          if (lane < 2) {
            Node c = N;
            c.st = lane ? N.st + l : N.st;
            c.count = lane ? count - l : l;
            c.turns = lane ? N.turns : N.turns + 1;
            c.depth = N.depth + 1;
#pragma unroll
            for (int d = 0; d < D; ++d) {
              c.lo[d] = lane && d == cd ? cut : N.lo[d];
              c.hi[d] = !lane && d == cd ? cut : N.hi[d];
            }
            add(c, cur ^ 1);
          }
          __syncwarp();
        }
        __syncthreads();
        if (threadIdx.x == 0) listCount[cur] = 0;
      }
      // windows: warp w takes the nodes that begin in its part of the slots
      if (jobCount > 0) {
        const int part = (all + warps - 1) / warps;
        const int end = min(all, (warp + 1) * part);
        for (int cur = warp * part; cur < end;) {
          const int p = cur + lane;
          const int ja = p < end ? (int)jobAt[p] : 0xffff;
          unsigned starts = __ballot_sync(kFull, ja != 0xffff);
          if (starts == 0u) {
            cur += 32;
            continue;
          }
          const int skip = __ffs(starts) - 1;
          if (skip > 0) {  // begin the window at a node
            cur += skip;
            continue;
          }
          const unsigned over = __ballot_sync(kFull, ja != 0xffff && lane + jobs[ja == 0xffff ? 0 : ja].count > 32);
          const int limit = over ? __ffs(over) - 1 : 32;
          if (limit < 32) starts &= (1u << limit) - 1u;
          const unsigned upto = starts & (kFull >> (31 - lane));
          const int s0 = 31 - __clz(upto);  // lane 0 begins a node, so upto is not empty
          const int jid = __shfl_sync(kFull, ja, s0);
          const Node& J = jobs[jid];
          int segS = s0, segE = s0 + J.count;
          const bool mine = lane < segE;
          if (!mine) {
            segS = lane;
            segE = lane + 1;
          }
          int turns = J.turns, depth = J.depth;
          const int at = cur + J.delta;  // lane l's global position is at + l
          T lo[D], hi[D];
#pragma unroll
          for (int d = 0; d < D; ++d) {
            lo[d] = J.lo[d];
            hi[d] = J.hi[d];
          }
          Rec<T, D> r;
          if (mine) {
            r = pts[p];
          } else {
#pragma unroll
            for (int c = 0; c < RecSize<T, D>::chunks; ++c) r.v[c] = make_uint4(0u, 0u, 0u, 0u);
          }
          for (;;) {
            const int count = segE - segS;
            const bool act = mine && count > a.bucket;
            if (!__any_sync(kFull, act)) break;
            const unsigned segMask = (segE == 32 ? 0u : 1u << segE) - (1u << segS);
            T ideal;
            const int cd = widest_dim<T, D>(lo, hi, a.dim, &ideal);
            T v = coord_of(r, cd);
            if (a.splitRule == 1) {
              // the value of rank count / 2: each lane counts the values
              // before its own, walking its node's lanes in a ring
              const int longest = __reduce_max_sync(kFull, act ? count : 0);
              int rank = 0, src = lane;
              for (int o = 1; o < longest; ++o) {
                src = src + 1 == segE ? segS : src + 1;
                const T y = __shfl_sync(kFull, v, src);
                rank += o < count && (y < v || (y == v && src < lane)) ? 1 : 0;
              }
              const unsigned has = __ballot_sync(kFull, rank == count / 2) & segMask;
              ideal = next_up(__shfl_sync(kFull, v, __ffs(has) - 1));
            }
            T mn = v, mx = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              const T y = __shfl_up_sync(kFull, mn, o), z = __shfl_up_sync(kFull, mx, o);
              if (lane - o >= segS) {
                mn = y < mn ? y : mn;
                mx = z > mx ? z : mx;
              }
            }
            mn = __shfl_sync(kFull, mn, segE - 1);
            mx = __shfl_sync(kFull, mx, segE - 1);
            const int mode = ideal < mn ? kBelowMin : (ideal > mx ? kAboveMax : kInside);
            const T cut = mode == kBelowMin ? mn : (mode == kAboveMax ? mx : ideal);
            const unsigned less = __ballot_sync(kFull, v < cut) & segMask;
            const unsigned same = __ballot_sync(kFull, v == cut) & segMask;
            const int lt = __popc(less), eq = __popc(same);
            const int loc = lane - segS;
            uint16_t* const slots = tab + cur + segS;
            // one partition pass: my partner's lane
            const auto partner = [&](bool on, int pos, int mid, unsigned passing) {
              const int ci = __popc(passing & below);
              const bool pass = (passing >> lane) & 1u;
              const bool left = on && pos >= 0 && pos < mid && !pass;
              const bool right = on && pos >= mid && pass;
              const int i = left ? pos - ci : mid - 1 - ci;
              if (left) slots[i] = (uint16_t)lane;
              if (right) slots[count / 2 + i] = (uint16_t)lane;
              __syncwarp();
              const int src = left ? (int)slots[count / 2 + i] : (right ? (int)slots[i] : lane);
              __syncwarp();
              return src;
            };
            const unsigned passing = mode == kBelowMin ? same : less;
            const int mid = __popc(passing);
            r = shfl_rec(r, partner(act, loc, mid, passing));
            const bool again = act && mode == kInside && eq > 0;
            if (__any_sync(kFull, again)) {
              v = coord_of(r, cd);
              const unsigned p2 = __ballot_sync(kFull, loc >= lt && v <= cut) & segMask;
              r = shfl_rec(r, partner(again, loc - lt, eq, p2));
            }
            if (act) {
              const int split = segS + left_count(mode, count, lt, eq);
              if (lane == split) mark_split(a.marks, at + lane, at + segS, turns, cd, cut);
              const bool isLeft = lane < split;
              if (isLeft) {
                segE = split;
                ++turns;
              } else {
                segS = split;
              }
              ++depth;
#pragma unroll
              for (int d = 0; d < D; ++d) {
                hi[d] = isLeft && d == cd ? cut : hi[d];
                lo[d] = !isLeft && d == cd ? cut : lo[d];
              }
            }
          }
          if (mine) {
            if (lane == segS) {
              mark_leaf(a.marks, at + lane, turns);
              hmax = max(hmax, depth);
            }
            pts[p] = r;
          }
          cur += limit;
        }
      }
      __syncthreads();
      for (int s = 0; s < k; ++s) {
        Rec<T, D>* dst = a.recs + startOf[s];
        const Rec<T, D>* src = pts + slotOf[s];
        for (int i = threadIdx.x; i < countOf[s]; i += blockDim.x) dst[i] = src[i];
      }
      done += k;
      __syncthreads();
    }
  }
  hmax = __reduce_max_sync(kFull, hmax);
  levels = __reduce_max_sync(kFull, levels);
  if (lane == 0) {
    if (hmax > 0) atomicMax(a.counters + kHeight, hmax);
    if (levels > 0) atomicMax(a.counters + kLevels, levels);
  }
}

// ---------------------------------------------------------------------------
// Numbering: leaves before each 32-position word, then every node at once.

constexpr int kRankBlock = 1024;

// rank[w]: leaves in the block's earlier words; sums[b]: the block's leaves.
__global__ void __launch_bounds__(kRankBlock) k_leaf_ranks(const uint32_t* __restrict__ bits, int64_t words,
                                                           uint32_t* rank, uint32_t* sums) {
  __shared__ uint32_t warpSum[32];
  const int64_t w = blockIdx.x * (int64_t)kRankBlock + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t c = w < words ? (uint32_t)__popc(bits[w]) : 0u;
  uint32_t inc = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) warpSum[warp] = inc;
  __syncthreads();
  uint32_t before = 0;
  for (int i = 0; i < warp; ++i) before += warpSum[i];
  if (w < words) rank[w] = before + inc - c;
  if (threadIdx.x == kRankBlock - 1) sums[blockIdx.x] = before + inc;
}

// sums becomes its exclusive prefix, sums[blocks] the total (one block). Also
// the build's status: [0] non-finite input (set by k_pack_bounds), [1] build
// did not finish (capacity exceeded, or levels left over: the median rule's in
// *segsLeft), [2] tallest tree's height, [3] top levels run.
__global__ void __launch_bounds__(kRankBlock) k_leaf_rank_sums(uint32_t* sums, int blocks, const int* segsLeft,
                                                               const int* counters, int* status) {
  if (threadIdx.x == 0) {
    status[1] = (counters[kFlags] || *segsLeft > 0) ? 1 : 0;
    status[2] = status[1] ? 0 : counters[kHeight];
    status[3] = counters[kLevels];
  }
  __shared__ uint32_t warpSum[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t carry = 0;
  for (int b0 = 0; b0 < blocks; b0 += kRankBlock) {
    const int b = b0 + threadIdx.x;
    const uint32_t c = b < blocks ? sums[b] : 0u;
    uint32_t inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, inc, o);
      if (lane >= o) inc += y;
    }
    __syncthreads();
    if (lane == 31) warpSum[warp] = inc;
    __syncthreads();
    uint32_t before = 0, all = 0;
    for (int i = 0; i < 32; ++i) {
      before += i < warp ? warpSum[i] : 0u;
      all += warpSum[i];
    }
    if (b < blocks) sums[b] = carry + before + inc - c;
    carry += all;
  }
  if (threadIdx.x == 0) sums[blocks] = carry;
}

// One thread per position. A build that did not finish (status[1]: levels
// left over after a fixed level count, or a capacity guard hit) gets one leaf
// per cloud holding all of its points instead: a well-formed forest that a
// search (or a captured graph's search) can still traverse, and which gives
// exact results for finite clouds.
template <typename T>
__global__ void k_emit(TreeMarks<T> m, const uint32_t* __restrict__ rank, const uint32_t* __restrict__ sums, int n,
                       int rankBlocks, const int64_t* __restrict__ off, int nClouds, int* status, Node<T>* nodes,
                       int64_t nodeCap, int64_t* nodeOffset) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (status[1]) {
    for (int64_t c = p; c <= nClouds; c += (int64_t)gridDim.x * blockDim.x) {
      nodeOffset[c] = c;
      if (c < nClouds && c < nodeCap) store_leaf(nodes + c, (uint32_t)(off[c + 1] - off[c]), (uint32_t)off[c]);
    }
    return;
  }
  if (p == 0) nodeOffset[nClouds] = 2 * (int64_t)sums[rankBlocks] - nClouds;
  if (p >= n) return;
  const int w = (int)(p >> 5), lane = (int)(p & 31);
  const uint32_t bits = m.leafBits[w];
  if (!((bits >> lane) & 1u)) return;
  const auto leaves_before = [&](int q) {
    const int qw = q >> 5;
    return (int64_t)sums[qw / kRankBlock] + rank[qw] + __popc(m.leafBits[qw] & ((1u << (q & 31)) - 1u));
  };
  const int64_t before = leaves_before((int)p);
  // the leaf ends where the next one begins
  int64_t next = n;
  const uint32_t later = bits & ~(kFull >> (31 - lane));
  if (later) {
    next = (p & ~int64_t(31)) + __ffs(later) - 1;
  } else {
    for (int64_t v = w + 1; v * 32 < n; ++v) {
      const uint32_t b = m.leafBits[v];
      if (b) {
        next = v * 32 + __ffs(b) - 1;
        break;
      }
    }
  }
  const int64_t leaf = 2 * before + m.leafTurns[p];
  const Split<T> s = m.split[p];
  bool ok = leaf >= 0 && leaf < nodeCap;
  if (ok) store_leaf(nodes + leaf, (uint32_t)(next - p), (uint32_t)p);
  if (s.start < 0) {
    nodeOffset[s.turnsDim] = 2 * before - (int64_t)s.turnsDim;
  } else {
    const int turns = (int)s.turnsDim >> 4;
    const int64_t node = 2 * leaves_before(s.start) + turns;
    const bool in = node >= 0 && node < nodeCap;
    if (in) store_inner(nodes + node, s.turnsDim & 15u, (uint32_t)(2 * before + turns), s.cut);
    ok = ok && in;
  }
  if (!ok) atomicOr(status + 1, 1);  // unreachable for a finished build
}

}  // namespace
}  // namespace nabo_gb300
