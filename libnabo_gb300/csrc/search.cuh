// search.cuh -- kd-tree and brute-force kNN kernels (templates).
//
// One thread per query. The traversal is the reference's recurseKnn
// (nabo/kdtree_cpu.cpp:367-447) turned into a loop with an explicit stack:
// at an inner node the near child is entered at once and the far child is
// pushed with its incremental box distance
//     rd_far = rd + (-(old_off*old_off) + new_off*new_off)
// and the offset vector it must see; a popped far child is visited iff
//     rd_far <= maxRadius^2  and  rd_far * (1+eps)^2 <= head.
// The far child is pushed only if that test already holds, which changes no
// decision because head never grows. Every +,-,* is separately rounded
// (no FMA contraction) so distances are bit-identical to the CPU oracle.
//
// Top-k: K (dist2, index) entries in registers, kept in descending order so
// the head (largest) is slot 0; slots >= k hold a value below every entry so
// one instantiation serves every k <= K. Entries are ordered by (dist2,
// index): among equal distances the lower index is kept, which makes the
// result independent of visit order (the reference's
// IndexHeapBruteForceVector keeps the first visited, nabo/index_heap.h:
// 322-334). Insertion is branch-free: with g[j] = (slot j > new entry),
// which is true for a prefix of the slots, slot j takes the new entry while
// g[j], then slot j+1 while g[j+1], and keeps its value after (move_if).
#pragma once

#include <type_traits>

#include "common.cuh"

namespace nabo_gb300 {

// dst = src where p, as a predicated multiply-add by a one the compiler cannot
// see through (an integer src * 1 + 0, on the FMA pipe). The searches are bound
// by the ALU pipe, which executes selects and compares; written as selects, an
// insertion into a sorted register list took two thirds of its ALU slots for
// moving entries. (Search kernel, selects -> predicated moves, which the
// compiler turns back into selects for the most part -> these: lidar 1.15 M
// points and queries, k = 10 1053 -> 940 -> 877 us; uniform 1 M 850 -> 768 ->
// 735; lidar 500 k, k = 16 695 -> 620 -> 580; the 512-cloud batch 18.3 -> 16.7
// -> 15.95 ms. The same for the traversal's coordinate picks was slower, 877
// -> 940: they wait on the multiplies' latency.)
static __constant__ uint32_t c_one = 1u;
__device__ __forceinline__ void move_if(bool p, uint32_t& dst, uint32_t src, uint32_t one) {
  asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\t@p mad.lo.u32 %0, %1, %3, 0;\n\t}"
      : "+r"(dst)
      : "r"(src), "r"((int)p), "r"(one));
}
__device__ __forceinline__ void move_if(bool p, int& dst, int src, uint32_t one) {
  uint32_t d = (uint32_t)dst;
  move_if(p, d, (uint32_t)src, one);
  dst = (int)d;
}
template <typename U>
__device__ __forceinline__ std::enable_if_t<sizeof(U) == 8> move_if(bool p, U& dst, U src, uint32_t one) {
  uint32_t l = (uint32_t)dst, h = (uint32_t)(dst >> 32);
  move_if(p, l, (uint32_t)src, one);
  move_if(p, h, (uint32_t)(src >> 32), one);
  dst = (U)h << 32 | l;
}

// double: the distance's 64-bit pattern and the index in separate arrays.
// Distances are >= 0, where the pattern orders like the value, so the
// (dist2, index) order is decided by integer compares on the ALU, keeping
// the scarce FP64 pipe for distances. An empty slot is (+inf, -1): no finite
// distance compares above it, as the reference's strict `dist < head` with
// head = +inf; padding slots (>= k) hold (+0, -1), below every entry.
template <typename T, int K>
struct TopK {
  unsigned long long d[K];
  int i[K];
  static __device__ __forceinline__ bool greater(unsigned long long da, int ia, unsigned long long db, int ib) {
    return da > db || (da == db && ia > ib);
  }
  static __device__ __forceinline__ unsigned long long bits(T x) {
    return (unsigned long long)__double_as_longlong((double)x);
  }
  __device__ __forceinline__ void init(int k, int = 32) {
#pragma unroll
    for (int j = 0; j < K; ++j) {
      d[j] = j < k ? bits(Ar<T>::inf()) : 0ull;
      i[j] = -1;
    }
  }
  __device__ __forceinline__ T head() const { return (T)__longlong_as_double((long long)d[0]); }
  __device__ __forceinline__ bool accepts(T dist, int idx) const { return greater(d[0], i[0], bits(dist), idx); }
  // Drops the head and inserts (dist, idx); requires accepts(dist, idx).
  __device__ __forceinline__ void insert(T dist, int idx) {
    const unsigned long long x = bits(dist);
    const uint32_t one = c_one;
    bool g = true;  // entry j > (dist, idx)
#pragma unroll
    for (int j = 0; j < K; ++j) {
      move_if(g, d[j], x, one);
      move_if(g, i[j], idx, one);
      if (j + 1 < K) {
        g = greater(d[j + 1], i[j + 1], x, idx);
        move_if(g, d[j], d[j + 1], one);
        move_if(g, i[j], i[j + 1], one);
      }
    }
  }
  __device__ __forceinline__ int count(int k) const {
    int c = 0;
#pragma unroll
    for (int j = 0; j < K; ++j) c += (j < k && i[j] >= 0) ? 1 : 0;
    return c;
  }
  // Writes the k entries in ascending order; returns how many are valid.
  __device__ __forceinline__ int store(int k, int32_t* __restrict__ oi, T* __restrict__ od) const {
    int found = 0;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      if (j < k) {
        oi[k - 1 - j] = i[j];
        od[k - 1 - j] = (T)__longlong_as_double((long long)d[j]);
        found += i[j] >= 0 ? 1 : 0;
      }
    }
    return found;
  }
};

// double lists of 16 or more entries in the kd-tree search: a binary
// max-heap of (dist2 bits, index) in (dynamic) shared memory, a section per
// warp, slot-major with one column per searching lane (a call that spreads few
// queries over many warps asks for less shared memory: 6000 queries, 8-D,
// k = 32, 3.50 -> 3.35 ms), the root kept in registers for the accept test. Held in registers, such a list (3
// registers an entry) spilled under the search kernel's register cap, and
// every insertion walked the spilled entries through local memory (8-D,
// k = 32: 2.2 G local loads a launch). Here an insertion sifts down at most
// log2(k) levels. The entries and their order are those of TopK: the k
// smallest (dist2, index) pairs, empty entries (+inf, -1), written out in
// ascending order.
template <int K>
struct SmemTopK {
  unsigned long long* d;  // entry j of this thread's list at d[j * stride]
  int* ix;
  int n;
  int stride;  // lists per warp: the lanes that search
  unsigned long long rootD;
  int rootI;
  static __device__ __forceinline__ bool greater(unsigned long long da, int ia, unsigned long long db, int ib) {
    return da > db || (da == db && ia > ib);
  }
  static __device__ __forceinline__ unsigned long long bits(double x) {
    return (unsigned long long)__double_as_longlong(x);
  }
  __device__ __forceinline__ void init(int k, int lanes = 32) {
    extern __shared__ __align__(16) unsigned char heapSmem[];
    stride = lanes;
    const int column = (threadIdx.x >> 5) * K * lanes + (threadIdx.x & 31);
    d = reinterpret_cast<unsigned long long*>(heapSmem) + column;
    ix = reinterpret_cast<int*>(heapSmem + (size_t)(blockDim.x >> 5) * lanes * K * sizeof(unsigned long long)) + column;
    n = k < K ? k : K;
    rootD = bits(Ar<double>::inf());
    rootI = -1;
    for (int j = 0; j < n; ++j) {
      d[j * stride] = rootD;
      ix[j * stride] = -1;
    }
  }
  __device__ __forceinline__ double head() const { return __longlong_as_double((long long)rootD); }
  __device__ __forceinline__ bool accepts(double dist, int idx) const { return greater(rootD, rootI, bits(dist), idx); }
  // The root (the largest entry) drops out and (x, xi) sifts down from it
  // within the first m entries.
  __device__ __forceinline__ void sift(unsigned long long x, int xi, int m) {
    int j = 0;
    for (;;) {
      const int l = 2 * j + 1;
      if (l >= m) break;
      int c = l;
      unsigned long long cd = d[l * stride];
      int ci = ix[l * stride];
      if (l + 1 < m) {
        const unsigned long long rd = d[(l + 1) * stride];
        const int ri = ix[(l + 1) * stride];
        if (greater(rd, ri, cd, ci)) {
          c = l + 1;
          cd = rd;
          ci = ri;
        }
      }
      if (!greater(cd, ci, x, xi)) break;
      d[j * stride] = cd;
      ix[j * stride] = ci;
      j = c;
    }
    d[j * stride] = x;
    ix[j * stride] = xi;
  }
  // Drops the largest entry and inserts (dist, idx); requires accepts(dist, idx).
  __device__ __forceinline__ void insert(double dist, int idx) {
    sift(bits(dist), idx, n);
    rootD = d[0];
    rootI = ix[0];
  }
  __device__ __forceinline__ int count(int) const {
    int c = 0;
    for (int j = 0; j < n; ++j) c += ix[j * stride] >= 0 ? 1 : 0;
    return c;
  }
  // Writes the entries in ascending order (the largest last), emptying the
  // heap; returns how many are valid.
  __device__ __forceinline__ int store(int, int32_t* __restrict__ oi, double* __restrict__ od) {
    int found = 0;
    for (int m = n; m > 0; --m) {
      const unsigned long long top = d[0];
      const int ti = ix[0];
      oi[m - 1] = ti;
      od[m - 1] = __longlong_as_double((long long)top);
      found += ti >= 0 ? 1 : 0;
      if (m > 1) sift(d[(m - 1) * stride], ix[(m - 1) * stride], m - 1);
    }
    return found;
  }
};

// The list the kd-tree search keeps: shared-memory heaps for double lists
// of 16 or more entries, registers otherwise. (Float lists stay in
// registers: the same heap over packed float keys was slower at every size
// measured -- lidar k = 10 kernel 0.990 -> 1.026 ms, batched k = 16 search
// 13.67 -> 14.60 ms, 8-D k = 32 search 92 -> 126 ms -- since the sorted
// register list's insertion is branch-free and a sift waits on dependent
// shared-memory loads; double lists spilled, float ones hardly.)
template <typename T, int K>
struct SearchHeap {
  using type = TopK<T, K>;
  static constexpr size_t bytes(int) { return 0; }  // dynamic shared memory of a block
};
template <int K>
struct SearchHeap<double, K> {
  using type = std::conditional_t<(K >= 16), SmemTopK<K>, TopK<double, K>>;
  static constexpr size_t bytes(int threads) {
    return K >= 16 ? (size_t)threads * K * (sizeof(unsigned long long) + sizeof(int)) : 0;
  }
};

// float: one 64-bit key per entry, (bit pattern of dist2) << 32 | index.
// Distances are >= 0, where the IEEE bit pattern orders like the value, so
// one unsigned comparison orders (dist2, index). An empty slot is
// (+inf, 0): no finite distance compares above it and no infinite one
// below, as the reference's strict `dist < head` with head = +inf
// (nabo/kdtree_cpu.cpp:392-396); it is written out as (-1, +inf). Padding
// slots (>= k) hold 0.
template <int K>
struct TopK<float, K> {
  uint64_t key[K];
  static __device__ __forceinline__ uint64_t make(float dist, int idx) {
    return (uint64_t(__float_as_uint(dist)) << 32) | (uint32_t)idx;
  }
  __device__ __forceinline__ void init(int k) {
#pragma unroll
    for (int j = 0; j < K; ++j) key[j] = j < k ? (uint64_t(0x7f800000u) << 32) : 0ull;
  }
  __device__ __forceinline__ float head() const { return __uint_as_float((uint32_t)(key[0] >> 32)); }
  __device__ __forceinline__ bool accepts(float dist, int idx) const { return make(dist, idx) < key[0]; }
  __device__ __forceinline__ void insert(float dist, int idx) { insert_key(make(dist, idx)); }
  // requires x < key[0]
  __device__ __forceinline__ void insert_key(uint64_t x) {
    const uint32_t one = c_one;
    bool g = true;  // key[j] > x
#pragma unroll
    for (int j = 0; j < K; ++j) {
      move_if(g, key[j], x, one);
      if (j + 1 < K) {
        g = key[j + 1] > x;
        move_if(g, key[j], key[j + 1], one);
      }
    }
  }
  __device__ __forceinline__ int count(int k) const {
    int c = 0;
#pragma unroll
    for (int j = 0; j < K; ++j) c += (j < k && (uint32_t)(key[j] >> 32) != 0x7f800000u) ? 1 : 0;
    return c;
  }
  __device__ __forceinline__ uint32_t out_idx(int j) const {
    return (uint32_t)(key[j] >> 32) == 0x7f800000u ? 0xffffffffu : (uint32_t)key[j];
  }
  // Writes the k entries in ascending order (slot j goes to position
  // k-1-j); returns how many are valid. When both rows are 8-byte aligned,
  // positions (p, p+1) with p even go out as one 64-bit store per row.
  __device__ __forceinline__ int store(int k, int32_t* __restrict__ oi, float* __restrict__ od) const {
    int found = 0;
    const bool pairs = ((reinterpret_cast<uintptr_t>(oi) | reinterpret_cast<uintptr_t>(od)) & 7u) == 0;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      if (j < k) {
        const int p = k - 1 - j;
        found += (uint32_t)(key[j] >> 32) == 0x7f800000u ? 0 : 1;
        if (!pairs) {
          oi[p] = (int32_t)out_idx(j);
          od[p] = __uint_as_float((uint32_t)(key[j] >> 32));
        } else if ((p & 1) == 0) {
          if (j >= 1) {  // slot j-1 is position p+1
            *reinterpret_cast<uint2*>(oi + p) = make_uint2(out_idx(j), out_idx(j - 1));
            *reinterpret_cast<uint2*>(od + p) = make_uint2((uint32_t)(key[j] >> 32), (uint32_t)(key[j - 1] >> 32));
          } else {
            oi[p] = (int32_t)out_idx(j);
            od[p] = __uint_as_float((uint32_t)(key[j] >> 32));
          }
        }
      }
    }
    return found;
  }
};

// Distances and box distances as values that order like them. A float is its
// own key. Doubles compare as bit patterns on the integer pipe: GB300 runs
// FP64 at 1/64 of the FP32 rate, and a DSETP takes an FP64 slot like the
// arithmetic. They are never negative (a box distance only grows along a
// path: a cell's cut lies no further out than the cell's own face, so
// -(old^2) + new^2 >= 0 in round-to-nearest too), where the pattern orders
// like the value, and a NaN of either sign is above every number.
__device__ __forceinline__ float dist_key(float x) { return x; }
__device__ __forceinline__ unsigned long long dist_key(double x) { return (unsigned long long)__double_as_longlong(x); }
// x <= limit(b) iff x <= b; limit(NaN) admits nothing.
__device__ __forceinline__ float dist_limit(float b) { return b; }
__device__ __forceinline__ unsigned long long dist_limit(double b) {
  const unsigned long long k = dist_key(b);
  return k <= 0x7ff0000000000000ull ? k + 1ull : 0ull;
}
__device__ __forceinline__ bool within(float x, float limit) { return x <= limit; }
__device__ __forceinline__ bool within(double x, unsigned long long limit) { return dist_key(x) < limit; }
// The smaller limit, where a NaN second argument (a radius) wins.
__device__ __forceinline__ float min_limit(float head, float radius) { return head < radius ? head : radius; }
__device__ __forceinline__ unsigned long long min_limit(unsigned long long head, unsigned long long radius) {
  return head < radius ? head : radius;
}
// x > 0; false for NaN
__device__ __forceinline__ bool positive(float x) { return x > 0.0f; }
__device__ __forceinline__ bool positive(double x) { return dist_key(x) - 1ull < 0x7ff0000000000000ull; }

// v[c]: a select per entry, or for 8 and 16 entries a tree of selects on the
// bits of c (half the predicates).
template <typename T, int D>
__device__ __forceinline__ T pick(const T (&v)[D], int c) {
  if constexpr (D == 8 || D == 16) {
    T h[D / 2];
    const bool odd = c & 1;
#pragma unroll
    for (int d = 0; d < D / 2; ++d) h[d] = odd ? v[2 * d + 1] : v[2 * d];
    return pick(h, c >> 1);
  } else {
    T r = v[0];
#pragma unroll
    for (int d = 1; d < D; ++d) {
      if (c == d) r = v[d];
    }
    return r;
  }
}

template <typename T, int D>
__device__ __forceinline__ T dist2_seq(const T (&q)[D], const Rec<T, D>& r) {
  // (q0-p0)^2 first, then +(q1-p1)^2, ... (nabo/kdtree_cpu.cpp:383-391)
  T diff = Ar<T>::sub(q[0], r.p.c[0]);
  T dist = Ar<T>::mul(diff, diff);
#pragma unroll
  for (int d = 1; d < D; ++d) {
    diff = Ar<T>::sub(q[d], r.p.c[d]);
    dist = Ar<T>::add(dist, Ar<T>::mul(diff, diff));
  }
  return dist;
}

// Leaf cells for query ordering: each query's cell is the leaf it reaches
// by always taking its near side (new_off > 0 -> right, as the search
// does). Leaves are numbered in pre-order, so queries sorted by leaf are
// grouped at the scale of the data's own buckets. With `hist` set, also
// counts the queries per leaf and gives each its rank (for a counting
// sort).
template <typename T, int D>
__global__ void k_leaf_cells(const Node<T>* __restrict__ nodes, const T* __restrict__ query, int64_t nq,
                             int64_t qStride, int dim, uint32_t* cell, uint32_t* rank, uint32_t* hist,
                             const int64_t* __restrict__ bQueryOffset = nullptr,
                             const int64_t* __restrict__ bNodeOffset = nullptr, int bClouds = 0) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nq) return;
  T q[D];
#pragma unroll
  for (int d = 0; d < D; ++d) q[d] = d < dim ? query[i * qStride + d] : T(0);
  uint32_t node = bQueryOffset ? (uint32_t)bNodeOffset[cloud_of(bQueryOffset, bClouds, i)] : 0u;
  for (;;) {
    const Node<T> nd = load_node(nodes, node);
    if (node_is_leaf(nd.meta)) break;
    const T newOff = Ar<T>::sub(pick(q, (int)node_dim(nd.meta)), nd.cut);
    node = positive(newOff) ? node_payload(nd.meta) : node + 1;
  }
  cell[i] = node;
  if (hist) rank[i] = atomicAdd(hist + node, 1u);
}

struct KnnLaunch {
  const void* nodes;
  const void* recs;
  const void* query;
  int64_t nq;
  int64_t qStride;
  int dim;
  const int32_t* order;
  int k;
  double maxError2;
  double maxRadius2;
  const void* maxRadii;
  int32_t* outIdx;
  void* outD2;
  unsigned long long* touched;
  int32_t* found;
  int64_t n;  // points (brute force)
  int allowSelf;
  int stats;
  const int32_t* nqDevice;  // if set, only threads t < *nqDevice search (t < nq still bounds the grid)
  double fallbackRadius;    // >= 0: bounded searches that miss rerun with maxRadius2 (see KnnArgs)
  int32_t* fallbacks;
  const void* recs32;       // double clouds: float copies of recs for the leaf pre-filter, or null
  const float* coordMax;    // largest coordinate magnitude of the cloud (device float)
  // batches of clouds (all null for one cloud): queries of cloud c are
  // [bQueryOffset[c], bQueryOffset[c+1]), its tree starts at node
  // bNodeOffset[c], it wants bK[c] neighbours written from bOutOffset[c]
  const int64_t* bQueryOffset;
  const int64_t* bNodeOffset;
  const int32_t* bK;
  const int64_t* bOutOffset;
  int bClouds;
  // one group of a batch's queries (see BatchClassPlan): thread t searches
  // position runPrefix[runBegin] + t of the group's running query count;
  // null runPrefix: thread t searches leaf-order position t
  const int64_t* runPrefix;
  const int32_t* runCloud;
  int runBegin, runEnd;
  // Trees taller than the compiled stacks (the reference's recursion has no
  // depth limit, nabo/kdtree_cpu.cpp:367-447):
  //  - slab/slabBytes: traversal stacks in global memory for the deep
  //    kernels, `cap` entries per query (stackCap, or the tree height read
  //    from *stackHeightDev plus one);
  //  - tallGate (batches, whose tree heights only the device knows): the
  //    tallest tree's height. Kernels with stacks of tallGateLimit entries
  //    return at once when it is larger; the deep kernels return at once
  //    when it is not. Both are launched, and exactly one searches.
  //  - deepFail: set to -1 by a deep kernel whose slab holds no stack.
  void* slab;
  int64_t slabBytes;
  int stackCap;
  const int* stackHeightDev;
  const int* tallGate;
  int tallGateLimit;
  int32_t* deepFail;
  int lanes;  // queries per warp, a power of 2 (see spread_lanes): its first lanes search, the others idle
};

// Leaf scan shared by the kernels: the bucket's records are read in chunks
// of 4 (independent loads in flight; the reference's buckets of at most 8
// hold 3.8 points on average on lidar scans, so wider chunks mostly compute
// empty slots), candidates that beat the current head are collected in a
// bit mask and inserted afterwards. The order of insertion inside a leaf
// does not change the heap after the leaf (the k smallest pairs of the
// union), so this matches the reference's point-by-point loop
// (nabo/kdtree_cpu.cpp:378-398); the warp pays for the largest number of
// insertions of any lane instead of for every point where some lane
// inserts.
// Float pre-filter of leaf points for double clouds (the GB300 runs FP64 at
// 1/64 of its FP32 rate, and the leaf distances are most of a double
// search's arithmetic). With q~ and p~ the float roundings of the query and
// point coordinates and e = (max|q~| + max|p~|) * 2^-22, every float
// difference is within e of q - p (conversion and subtraction errors are at
// most 2.1 * 2^-24 * (|q| + |p|) each), so a point within sqrt(t) of the query
// has a float squared distance of at most (sqrt(t) + e sqrt(D))^2, times
// 1 + 2^-18 for the rounding of the sum and plus 2^-140 for squares that
// underflow. With t a float at or above min(head, maxRadius^2), a point above
// that limit cannot enter the heap, and only the others get the exact double
// distance: results are unchanged. Coordinates beyond the float range make e
// infinite, which rejects nothing. (A sum of squared lower bounds,
// max(0, |q~ - p~| - e)^2, took twice the instructions a coordinate; 8-D
// and 16-D searches 1 % faster without.)
template <typename T, int D>
struct LeafFilter {
  __device__ __forceinline__ void init(const void*, const float*, const T (&)[D]) {}
  __device__ __forceinline__ bool on() const { return false; }
  __device__ __forceinline__ float threshold(T, T) const { return 0.0f; }
  __device__ __forceinline__ float limit(float) const { return 0.0f; }
  __device__ __forceinline__ bool rejects(int64_t, float) const { return false; }
};

template <int D>
struct LeafFilter<double, D> {
  const Rec<float, D>* recs32;
  float qf[D];
  float e;
  __device__ __forceinline__ void init(const void* r32, const float* coordMax, const double (&q)[D]) {
    recs32 = static_cast<const Rec<float, D>*>(r32);
    e = Ar<float>::inf();
    if (recs32) {
      float mq = 0.0f;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        qf[d] = (float)q[d];
        mq = fmaxf(mq, fabsf(qf[d]));
      }
      e = (mq + *coordMax) * 0x1p-22f;
    }
  }
  __device__ __forceinline__ bool on() const { return recs32 != nullptr; }
  // a float at or above min(head, maxRadius2) (a NaN radius: head)
  __device__ __forceinline__ float threshold(double head, double maxRadius2) const {
    const unsigned long long h = dist_key(head), r = dist_key(maxRadius2);
    return __double2float_ru(__longlong_as_double((long long)(r < h ? r : h)));
  }
  // the largest float squared distance of a point within threshold t
  __device__ __forceinline__ float limit(float t) const {
    constexpr float kRoot = D <= 4 ? 2.0f : (D <= 9 ? 3.0f : 4.0f);  // at least sqrt(D)
    const float u = __fadd_ru(__fsqrt_ru(t), __fmul_ru(e, kRoot));
    return __fmaf_ru(__fmul_ru(u, u), 1.0f + 0x1p-18f, 0x1p-140f);
  }
  __device__ __forceinline__ bool rejects(int64_t i, float lim) const {
    Rec<float, D> f;
    load_rec(recs32, i, f);
    float d2 = 0.0f;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const float a = qf[d] - f.p.c[d];
      d2 = fmaf(a, a, d2);
    }
    return d2 > lim;
  }
};

template <typename T, int D, int K, typename H>
__device__ __forceinline__ void scan_leaf(const Rec<T, D>* __restrict__ recs, uint32_t st, uint32_t cnt,
                                          const T (&q)[D], T maxRadius2, T minDist, bool want, H& heap,
                                          const LeafFilter<T, D>& flt) {
  constexpr int kChunk = 4;
  for (uint32_t base = 0; base < cnt; base += kChunk) {
    unsigned mask = 0;
    if constexpr (std::is_same<T, float>::value) {
      // float: one float compare against min(head, maxRadius2) lets a
      // candidate pass (NaN: none), and its packed (dist2 bits, index) key
      // decides ties with the head where it is inserted (1.15 M lidar
      // points, k = 10: 1036 us, against 1053 with the keys compared for
      // every point)
      uint64_t kj[kChunk];
      const float hd = heap.head();
      const float thrF = want ? (hd < maxRadius2 ? hd : maxRadius2) : __int_as_float(0x7fffffff);
#pragma unroll
      for (int j = 0; j < kChunk; ++j) {
        kj[j] = ~0ull;
        if (base + j < cnt) {
          Rec<T, D> r;
          load_rec(recs, (int64_t)st + base + j, r);
          const float d = dist2_seq(q, r);
          kj[j] = TopK<float, K>::make(d, r.p.idx);
          mask |= (d <= thrF && d > minDist) ? (1u << j) : 0u;
        }
      }
      while (mask) {
        const int j = __ffs(mask) - 1;
        mask &= mask - 1;
        uint64_t v = kj[0];
#pragma unroll
        for (int m = 1; m < kChunk; ++m) {
          if (j == m) v = kj[m];
        }
        if (v < heap.key[0]) heap.insert_key(v);
      }
    } else {
      T dj[kChunk];
      int ij[kChunk];
      const float thr = flt.on() ? flt.limit(flt.threshold(heap.head(), maxRadius2)) : 0.0f;
      const auto radLimit = dist_limit(maxRadius2);
      const auto minKey = dist_key(Ar<T>::eps());
#pragma unroll
      for (int j = 0; j < kChunk; ++j) {
        dj[j] = Ar<T>::inf();
        ij[j] = -1;
        if (base + j < cnt && !(flt.on() && flt.rejects((int64_t)st + base + j, thr))) {
          Rec<T, D> r;
          load_rec(recs, (int64_t)st + base + j, r);
          dj[j] = dist2_seq(q, r);
          ij[j] = r.p.idx;
          const bool ok = want && within(dj[j], radLimit) && heap.accepts(dj[j], ij[j]) &&
                          (minDist < T(0) || dist_key(dj[j]) > minKey);
          mask |= ok ? (1u << j) : 0u;
        }
      }
      while (mask) {
        const int j = __ffs(mask) - 1;
        mask &= mask - 1;
        T dv = dj[0];
        int iv = ij[0];
#pragma unroll
        for (int m = 1; m < kChunk; ++m) {
          if (j == m) {
            dv = dj[m];
            iv = ij[m];
          }
        }
        if (heap.accepts(dv, iv)) heap.insert(dv, iv);
      }
    }
  }
}

// Ascending bitonic sort of B (a power of 2) keys held in registers: every
// index is known at compile time, so a compare-exchange is one 64-bit
// compare and two selects.
template <int B>
__device__ __forceinline__ void sort_keys(uint64_t (&s)[B]) {
#pragma unroll
  for (int k2 = 2; k2 <= B; k2 <<= 1) {
#pragma unroll
    for (int j = k2 >> 1; j > 0; j >>= 1) {
#pragma unroll
      for (int i = 0; i < B; ++i) {
        const int l = i ^ j;
        if (l > i) {
          const uint64_t a = s[i], b = s[l];
          const bool sw = ((i & k2) == 0) ? (a > b) : (a < b);
          s[i] = sw ? b : a;
          s[l] = sw ? a : b;
        }
      }
    }
  }
}

// A query's first leaf into its still empty top-k (float, k == K): the
// first B points' keys -- those the leaf scan would not take (outside the
// radius, a forbidden self match, or !want) as the empty key -- sorted by a
// network and placed in the list as they are, then the rest of the leaf by
// the normal scan. The list ends as if the points had been inserted one at
// a time (it holds the K smallest keys, and the scan's order never matters
// to that), for a fraction of the work: about 6 B log2(B)^2 / 4 integer
// instructions against about 6 K per insertion.
template <int D, int K>
__device__ __forceinline__ void scan_first_leaf(const Rec<float, D>* __restrict__ recs, uint32_t st, uint32_t cnt,
                                                const float (&q)[D], float maxRadius2, float minDist, bool want,
                                                TopK<float, K>& heap, const LeafFilter<float, D>& flt) {
  constexpr int B = K <= 10 ? 8 : 16;
  constexpr uint64_t kEmpty = uint64_t(0x7f800000u) << 32;
  const uint64_t radKey = maxRadius2 == maxRadius2 ? ((uint64_t(__float_as_uint(maxRadius2)) << 32) | 0xffffffffull) : 0ull;
  const uint64_t thrKey = (!want || radKey == 0ull) ? 0ull : (kEmpty <= radKey ? kEmpty : radKey + 1ull);
  uint64_t sk[B];
#pragma unroll
  for (int j = 0; j < B; ++j) {
    sk[j] = kEmpty;
    if ((uint32_t)j < cnt) {
      Rec<float, D> r;
      load_rec(recs, (int64_t)st + j, r);
      const float d = dist2_seq(q, r);
      const uint64_t key = TopK<float, K>::make(d, r.p.idx);
      if (key < thrKey && d > minDist) sk[j] = key;
    }
  }
  sort_keys(sk);
#pragma unroll
  for (int j = 0; j < K; ++j) heap.key[j] = (K - 1 - j < B) ? sk[(K - 1 - j) < B ? (K - 1 - j) : 0] : kEmpty;
  if (cnt > (uint32_t)B) scan_leaf<float, D, K>(recs, st + B, cnt - B, q, maxRadius2, minDist, want, heap, flt);
}

// A pushed far child as 32-bit words [rd | off2[0..D-1] | node] (off2: the
// squared offsets, all the box-distance update needs; a T is one
// word for float, two for double) in 16-byte chunks: a push is one 128-bit
// local store per chunk (a lone trailing word is stored alone), a pop reads
// the first chunk, which holds rd, and the rest only if the child is
// visited.
template <typename T, int D>
struct StackRec {
  static constexpr int kTW = (int)(sizeof(T) / 4);
  static constexpr int kWords = kTW * (D + 1) + 1;
  static constexpr int kChunks = (kWords + 3) / 4;
  static constexpr int kNode = kTW * (D + 1);
  uint4 v[kChunks];
};

__device__ __forceinline__ void put_t(uint32_t* w, int i, float x) { w[i] = __float_as_uint(x); }
__device__ __forceinline__ void put_t(uint32_t* w, int i, double x) {
  w[i] = (uint32_t)__double2loint(x);
  w[i + 1] = (uint32_t)__double2hiint(x);
}
template <typename T>
__device__ __forceinline__ T get_t(const uint32_t* w, int i);
template <>
__device__ __forceinline__ float get_t<float>(const uint32_t* w, int i) {
  return __uint_as_float(w[i]);
}
template <>
__device__ __forceinline__ double get_t<double>(const uint32_t* w, int i) {
  return __hiloint2double((int)w[i + 1], (int)w[i]);
}

template <typename T, int D>
__device__ __forceinline__ void stack_push(StackRec<T, D>& e, T rd, const T (&off2)[D], int cd, T new2,
                                           uint32_t node) {
  using R = StackRec<T, D>;
  uint32_t w[R::kChunks * 4];
#pragma unroll
  for (int i = 0; i < R::kChunks * 4; ++i) w[i] = 0u;
  put_t(w, 0, rd);
#pragma unroll
  for (int d = 0; d < D; ++d) {
    put_t(w, R::kTW * (1 + d), d == cd ? new2 : off2[d]);
  }
  w[R::kNode] = node;
#pragma unroll
  for (int c = 0; c < R::kChunks; ++c) {
    if (c == R::kChunks - 1 && R::kWords % 4 == 1)
      e.v[c].x = w[4 * c];
    else
      e.v[c] = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
  }
}

template <typename T, int D>
__device__ __forceinline__ T stack_rd(const StackRec<T, D>& e) {
  const uint4 c0 = e.v[0];
  const uint32_t w[4] = {c0.x, c0.y, c0.z, c0.w};
  return get_t<T>(w, 0);
}

template <typename T, int D>
__device__ __forceinline__ uint32_t stack_take(const StackRec<T, D>& e, T (&off2)[D]) {
  using R = StackRec<T, D>;
  uint32_t w[R::kChunks * 4];
#pragma unroll
  for (int c = 0; c < R::kChunks; ++c) {
    if (c == R::kChunks - 1 && R::kWords % 4 == 1) {
      w[4 * c] = e.v[c].x;
      w[4 * c + 1] = w[4 * c + 2] = w[4 * c + 3] = 0u;
    } else {
      const uint4 v = e.v[c];
      w[4 * c] = v.x;
      w[4 * c + 1] = v.y;
      w[4 * c + 2] = v.z;
      w[4 * c + 3] = v.w;
    }
  }
#pragma unroll
  for (int d = 0; d < D; ++d) off2[d] = get_t<T>(w, R::kTW * (1 + d));
  return w[R::kNode];
}

// Where a query's traversal stack lives: a local array of N entries (the
// compiled kernels), or entries of a global-memory slab shared by the threads
// of a deep launch, thread g's entry sp at slab[sp * stride + g] so that the
// pushes of a warp at one depth are coalesced.
template <typename T, int D, int N>
struct LocalStack {
  StackRec<T, D> s[N];
  __device__ __forceinline__ StackRec<T, D>& operator[](int sp) { return s[sp]; }
};
template <typename T, int D>
struct SlabStack {
  StackRec<T, D>* base;
  int64_t stride;
  __device__ __forceinline__ StackRec<T, D>& operator[](int sp) { return base[(int64_t)sp * stride]; }
};

// What the thread at order position t searches.
template <typename T>
struct QueryTask {
  int64_t qi;       // query
  int64_t outBase;  // its first result entry
  int k;
  uint32_t root;
  T maxRadius2;
  // a bounded search (per-query radius) that misses may run once more
  // without its bound (the learned-radius form's fallback)
  bool mayFall;
};

template <typename T>
__device__ __forceinline__ QueryTask<T> query_task(const KnnLaunch& a, int64_t t) {
  QueryTask<T> w;
  w.k = a.k;
  w.root = 0;
  if (a.runPrefix) {
    const int64_t g = a.runPrefix[a.runBegin] + t;
    int lo = a.runBegin, hi = a.runEnd - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (a.runPrefix[mid] <= g)
        lo = mid;
      else
        hi = mid - 1;
    }
    const int c = a.runCloud[lo];
    w.qi = (int64_t)a.order[a.bQueryOffset[c] + (g - a.runPrefix[lo])];
    w.k = a.bK[c];
    w.root = (uint32_t)a.bNodeOffset[c];
    w.outBase = a.bOutOffset[c] + (w.qi - a.bQueryOffset[c]) * (int64_t)w.k;
  } else {
    w.qi = a.order ? (int64_t)a.order[t] : t;
    w.outBase = w.qi * (int64_t)a.k;
    if (a.bQueryOffset) {
      const int c = cloud_of(a.bQueryOffset, a.bClouds, w.qi);
      w.k = a.bK[c];
      w.root = (uint32_t)a.bNodeOffset[c];
      w.outBase = a.bOutOffset[c] + (w.qi - a.bQueryOffset[c]) * (int64_t)w.k;
    }
  }
  w.maxRadius2 = (T)a.maxRadius2;
  w.mayFall = false;
  if (a.maxRadii) {
    const T r = static_cast<const T*>(a.maxRadii)[w.qi];
    w.maxRadius2 = Ar<T>::mul(r, r);
    w.mayFall = a.fallbackRadius >= 0.0 && (double)r < a.fallbackRadius;
  }
  return w;
}

// One query (order position t) in the reference's visit order, structured
// descend / leaf / pop so the lanes of a warp run each phase together: all
// lanes descend until every lane stands on a leaf, then all scan their
// leaves, then all pop. `cap` entries of `stk` are available; the caller
// guarantees cap >= tree height. Adds the points examined to `touchedOut`.
// EXACT (epsilon 0, so maxError2 = 1 and rd * maxError2 = rd exactly): the
// push test rd <= maxRadius2 && rd <= head is one compare against
// min(maxRadius2, head), refreshed after each leaf; decisions are the same.
template <typename T, int D, int K, bool EXACT, typename S>
__device__ __forceinline__ void knn_query(const KnnLaunch& a, int64_t t, S& stk, int cap, uint32_t& touchedOut) {
  // the reference's self-match rule (nabo/kdtree_cpu.cpp:392-396): without
  // ALLOW_SELF_MATCH a point at distance <= epsilon is skipped; one compare
  // against -1 (everything passes) or epsilon
  const T minDist = a.allowSelf ? T(-1) : Ar<T>::eps();
  const Node<T>* __restrict__ nodes = static_cast<const Node<T>*>(a.nodes);
  const Rec<T, D>* __restrict__ recs = static_cast<const Rec<T, D>*>(a.recs);
  const T* __restrict__ query = static_cast<const T*>(a.query);
  uint32_t touched = 0;  // a query touches at most the cloud's n < 2^31 points
  const QueryTask<T> task = query_task<T>(a, t);
  const int k = task.k;
  T q[D];
#pragma unroll
  for (int d = 0; d < D; ++d) q[d] = d < a.dim ? query[task.qi * a.qStride + d] : T(0);
  T maxRadius2 = task.maxRadius2;
  bool mayFall = task.mayFall;
  const T maxError2 = (T)a.maxError2;
  typename SearchHeap<T, K>::type heap;
  heap.init(k);
  LeafFilter<T, D> flt;
  flt.init(a.recs32, a.coordMax, q);
  // squared offsets to the cell, per dimension: the reference's
  // rd += -(old*old) + new*new (nabo/kdtree_cpu.cpp:415, 433) reads only
  // squares, so the product is kept instead of computed again each step
  T off2[D];
  for (;;) {  // the search, and at most once more without the bound
    const auto radLimit = dist_limit(maxRadius2);
#pragma unroll
    for (int d = 0; d < D; ++d) off2[d] = T(0);
    int sp = 0;
    uint32_t node = task.root;
    T rd = T(0);
    bool fresh = true;  // no leaf scanned yet: the top-k is empty
    for (;;) {
      // descend to a leaf, pushing far children
      // min(maxRadius2, head), where a NaN radius (which passes nothing) wins
      const auto headLimit = dist_limit(heap.head());
      const auto bound = min_limit(headLimit, radLimit);
      Node<T> nd = load_node(nodes, node);
      while (!node_is_leaf(nd.meta)) {
        const int cd = (int)node_dim(nd.meta);
        const T newOff = Ar<T>::sub(pick(q, cd), nd.cut);
        const T new2 = Ar<T>::mul(newOff, newOff);
        const T rdFar = Ar<T>::add(rd, Ar<T>::add(-pick(off2, cd), new2));
        const uint32_t right = node_payload(nd.meta);
        const bool nearRight = positive(newOff);
        const uint32_t nearN = nearRight ? right : node + 1;
        const uint32_t farN = nearRight ? node + 1 : right;
        const bool far = EXACT ? within(rdFar, bound)
                               : (within(rdFar, radLimit) && within(Ar<T>::mul(rdFar, maxError2), headLimit));
        // sp <= tree height <= cap (checked by the caller); the test only
        // makes the bound explicit
        if (far && sp < cap) stack_push(stk[sp++], rdFar, off2, cd, new2, farN);
        node = nearN;
        nd = load_node(nodes, node);
      }
      // leaf
      const uint32_t cnt = node_payload(nd.meta);
      if constexpr (std::is_same<T, float>::value && K >= 8) {
        if (fresh && k == K)
          scan_first_leaf<D, K>(recs, node_start(nd), cnt, q, maxRadius2, minDist, true, heap, flt);
        else
          scan_leaf<T, D, K>(recs, node_start(nd), cnt, q, maxRadius2, minDist, true, heap, flt);
      } else {
        scan_leaf<T, D, K>(recs, node_start(nd), cnt, q, maxRadius2, minDist, true, heap, flt);
      }
      fresh = false;
      touched += cnt;
      // pop the next far child that can still hold a better neighbour
      bool more = false;
      const auto popLimit = dist_limit(heap.head());
      while (sp > 0) {
        --sp;
        const T e = stack_rd(stk[sp]);
        if (within(EXACT ? e : Ar<T>::mul(e, maxError2), popLimit)) {
          rd = e;
          node = stack_take(stk[sp], off2);
          more = true;
          break;
        }
      }
      if (!more) break;
    }
    if (!mayFall || heap.count(k) == k) break;
    mayFall = false;
    maxRadius2 = (T)a.maxRadius2;
    heap.init(k);
    if (a.fallbacks) atomicAdd(a.fallbacks, 1);
  }
  const int f = heap.store(k, a.outIdx + task.outBase, static_cast<T*>(a.outD2) + task.outBase);
  if (a.found) a.found[task.qi] = f;
  touchedOut += touched;
}

// Double searches with local stacks: the traversal above, with its FP64 work
// put off until a decision needs it. GB300 runs FP64 at 1/64 of its FP32
// rate, and with a handful of a warp's lanes active a step's FP64
// instructions cost as much as with all of them, so what counts is how often
// a warp executes them.
//  - The near side is the sign of the float difference of the rounded
//    coordinates when that exceeds its error bound e (LeafFilter), else of
//    the double difference.
//  - A far child is pushed when a float lower bound of its box distance is
//    within the pruning limit: rd - old^2 + new^2 with rd rounded down, the
//    old square from its upper 32 bits rounded up and new = |q~ - cut~| - e.
//    Its error is below 2^-20 of the sum (old^2 and rd are at most the
//    distance itself), covered by the factor 1 - 2^-17, and 2^-120 covers
//    underflow. The exact distance, the reference's rounded update
//    (nabo/kdtree_cpu.cpp:415, 433), is computed when the child is popped
//    and its lower bound is still within the limit: the reference's
//    decision, taken with the head the reference has at that point, so the
//    visits (and TOUCH_STATISTICS) are the same.
//  - A descent shares one frame (rd and the squared offsets it started
//    from), written once, instead of a copy per pushed child; an entry is
//    16 bytes: [far child | cut dimension << 27, lower bound with its low 8
//    bits replaced by the frame's slot, cut].
//  - A leaf's points are filtered in float first; the exact distances run in
//    a loop over the points that passed, so a warp executes them as often as
//    the lane with the most such points, not once per point some lane needs.
// (Search kernel, exact distances at every step -> here: 8-D clusters, 200 k
// points, 50 k queries, k = 32 12.9 -> 9.8 ms; 3-D uniform, 100 k points,
// 30 k queries, k = 10 302 -> 250 us.)
template <int D, int STACK>
struct F64Stack {
  static constexpr int kPairs = (D + 2) / 2;  // rd and D squares, in pairs
  uint4 entry[STACK];
  double2 frame[STACK][kPairs];
  static_assert(STACK <= 256, "frame slots take 8 bits");
};

// A float at or above x >= 0 (less 2^-126) and within 2^-20 of it, from x's
// upper 32 bits; infinity stays.
__device__ __forceinline__ float upper_bound_of_hi(uint32_t hi) {
  const int u = (int)hi + 1 - 0x38000000;
  return hi >= 0x47efffffu ? __int_as_float(0x7f800000) : (u > 0 ? __int_as_float(u << 3) : 0.0f);
}

template <int D, int K, bool EXACT, int STACK>
__device__ __forceinline__ void knn_query_f64(const KnnLaunch& a, int64_t t, F64Stack<D, STACK>& stk,
                                              uint32_t& touchedOut) {
  constexpr unsigned long long kEps = 0x3cb0000000000000ull;  // 2^-52, numeric_limits<double>::epsilon()
  const Node<double>* __restrict__ nodes = static_cast<const Node<double>*>(a.nodes);
  const Rec<double, D>* __restrict__ recs = static_cast<const Rec<double, D>*>(a.recs);
  uint32_t touched = 0;
  const QueryTask<double> task = query_task<double>(a, t);
  const int k = task.k;
  const double* __restrict__ query = static_cast<const double*>(a.query) + task.qi * a.qStride;
  double q[D];
#pragma unroll
  for (int d = 0; d < D; ++d) q[d] = d < a.dim ? query[d] : 0.0;
  double maxRadius2 = task.maxRadius2;
  bool mayFall = task.mayFall;
  const double maxError2 = a.maxError2;
  // a float at or above 1 / maxError2 (inf or NaN where that has none: no
  // child is then left out by its lower bound)
  const float invError = EXACT ? 1.0f : __double2float_ru(1.0 / maxError2) * (1.0f + 0x1p-20f);
  typename SearchHeap<double, K>::type heap;
  heap.init(k, a.lanes);
  LeafFilter<double, D> flt;
  flt.init(a.recs32, a.coordMax, q);
  double off2[D];
  for (;;) {  // the search, and at most once more without the bound
    const unsigned long long radLimit = dist_limit(maxRadius2);
    const bool anyRadius = radLimit != 0ull;  // a NaN radius accepts nothing
#pragma unroll
    for (int d = 0; d < D; ++d) off2[d] = 0.0;
    int sp = 0;
    uint32_t node = task.root;
    double rd = 0.0;
    float rdDown = 0.0f;
    float leafThr = flt.threshold(heap.head(), maxRadius2);
    // a float at or above the largest box distance still searched,
    // min(maxRadius2, head / maxError2)
    const auto prune_threshold = [&]() {
      return EXACT ? leafThr
                   : fminf(__double2float_ru(maxRadius2), __fmul_ru(__double2float_ru(heap.head()), invError));
    };
    float pruneThr = prune_threshold();
    float leafLimit = flt.limit(leafThr);
    for (;;) {
      const int frame = sp;
      bool saved = false;
      Node<double> nd = load_node(nodes, node);
      while (!node_is_leaf(nd.meta)) {
        const int cd = (int)node_dim(nd.meta);
        const float df = pick(flt.qf, cd) - node_cut_float(nd);
        const float ad = fabsf(df);
        bool nearRight = df > 0.0f;
        if (!(ad > flt.e)) nearRight = positive(Ar<double>::sub(query[cd], nd.cut));
        const float nf = fmaxf(ad - flt.e, 0.0f);
        uint32_t hi[D];
#pragma unroll
        for (int d = 0; d < D; ++d) hi[d] = (uint32_t)__double2hiint(off2[d]);
        const float low = fmaf((rdDown - upper_bound_of_hi(pick(hi, cd))) + nf * nf, 1.0f - 0x1p-17f, -0x1p-120f);
        const uint32_t right = node_payload(nd.meta);
        const uint32_t farN = nearRight ? node + 1 : right;
        node = nearRight ? right : node + 1;
        // (a NaN bound, from infinite coordinates, is pushed and decided exactly)
        if (anyRadius && !(low > pruneThr) && sp < STACK) {
          if (!saved) {
            saved = true;
            double v[2 * F64Stack<D, STACK>::kPairs];
            v[0] = rd;
#pragma unroll
            for (int d = 0; d < D; ++d) v[1 + d] = off2[d];
            if (D % 2 == 0) v[D + 1] = 0.0;
#pragma unroll
            for (int p = 0; p < F64Stack<D, STACK>::kPairs; ++p)
              stk.frame[frame][p] = make_double2(v[2 * p], v[2 * p + 1]);
          }
          const uint32_t lowBits = low > 0.0f ? __float_as_uint(low) : 0u;
          stk.entry[sp++] =
              make_uint4(farN | ((uint32_t)cd << 27), (lowBits & ~255u) | (uint32_t)frame,
                         (uint32_t)__double2loint(nd.cut), (uint32_t)__double2hiint(nd.cut));
        }
        nd = load_node(nodes, node);
      }
      // leaf
      const uint32_t cnt = node_payload(nd.meta);
      const uint32_t st = node_start(nd);
      touched += cnt;
      bool changed = false;
      for (uint32_t base = 0; base < cnt; base += 32) {
        const uint32_t m = cnt - base < 32u ? cnt - base : 32u;
        unsigned mask = 0;
        for (uint32_t j0 = 0; j0 < m; j0 += 4) {
#pragma unroll
          for (uint32_t j = 0; j < 4; ++j)
            if (j0 + j < m && !flt.rejects((int64_t)st + base + j0 + j, leafLimit)) mask |= 1u << (j0 + j);
        }
        while (mask) {
          const int j = __ffs(mask) - 1;
          mask &= mask - 1;
          Rec<double, D> r;
          load_rec(recs, (int64_t)st + base + j, r);
          const double dist = dist2_seq(q, r);
          if (within(dist, radLimit) && heap.accepts(dist, r.p.idx) && (a.allowSelf || dist_key(dist) > kEps)) {
            heap.insert(dist, r.p.idx);
            changed = true;
          }
        }
      }
      if (changed) {
        leafThr = flt.threshold(heap.head(), maxRadius2);
        pruneThr = prune_threshold();
        leafLimit = flt.limit(leafThr);
      }
      // pop the next far child that can still hold a better neighbour
      bool more = false;
      const unsigned long long popLimit = dist_limit(heap.head());
      while (sp > 0) {
        --sp;
        const uint4 e = stk.entry[sp];
        if (__uint_as_float(e.y & ~255u) > pruneThr) continue;
        const int cd = (int)(e.x >> 27);
        double v[2 * F64Stack<D, STACK>::kPairs];
#pragma unroll
        for (int p = 0; p < F64Stack<D, STACK>::kPairs; ++p) {
          const double2 x = stk.frame[e.y & 255u][p];
          v[2 * p] = x.x;
          v[2 * p + 1] = x.y;
        }
#pragma unroll
        for (int d = 0; d < D; ++d) off2[d] = v[1 + d];
        const double newOff = Ar<double>::sub(query[cd], __hiloint2double((int)e.w, (int)e.z));
        const double new2 = Ar<double>::mul(newOff, newOff);
        const double rdFar = Ar<double>::add(v[0], Ar<double>::add(-pick(off2, cd), new2));
        if (within(rdFar, radLimit) && within(EXACT ? rdFar : Ar<double>::mul(rdFar, maxError2), popLimit)) {
          rd = rdFar;
          rdDown = __double2float_rd(rd);
#pragma unroll
          for (int d = 0; d < D; ++d) off2[d] = d == cd ? new2 : off2[d];
          node = e.x & kMaxNodeIndex;
          more = true;
          break;
        }
      }
      if (!more) break;
    }
    if (!mayFall || heap.count(k) == k) break;
    mayFall = false;
    maxRadius2 = a.maxRadius2;
    heap.init(k, a.lanes);
    if (a.fallbacks) atomicAdd(a.fallbacks, 1);
  }
  const int f = heap.store(k, a.outIdx + task.outBase, static_cast<double*>(a.outD2) + task.outBase);
  if (a.found) a.found[task.qi] = f;
  touchedOut += touched;
}

// The warp's TOUCH_STATISTICS counts summed into a.touched (every lane of
// the warp calls this).
__device__ __forceinline__ void add_touched(const KnnLaunch& a, uint32_t touched) {
  if (a.stats) {
    unsigned long long sum = touched;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(a.touched, sum);
  }
}

// One thread per query, stack of STACK entries in local memory.
template <typename T, int D, int K, int STACK, bool EXACT>
__device__ __forceinline__ void knn_kdtree_body(const KnnLaunch& a) {
  if (a.tallGate && *a.tallGate > a.tallGateLimit) return;  // the deep kernel searches (uniform)
  const int lane = threadIdx.x & 31;
  const int64_t t = ((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5) * a.lanes + lane;
  uint32_t touched = 0;
  if (lane < a.lanes && t < a.nq && (!a.nqDevice || t < (int64_t)*a.nqDevice)) {
    if constexpr (sizeof(T) == 8) {
      F64Stack<D, STACK> stk;
      knn_query_f64<D, K, EXACT, STACK>(a, t, stk, touched);
    } else {
      LocalStack<T, D, STACK> stk;
      knn_query<T, D, K, EXACT>(a, t, stk, STACK, touched);
    }
  }
  add_touched(a, touched);
}

template <typename T, int D, int K, int STACK, bool EXACT>
__global__ void __launch_bounds__(128) k_knn_kdtree(KnnLaunch a) {
  knn_kdtree_body<T, D, K, STACK, EXACT>(a);
}

// Double searches of 16 or more neighbours: limited to 128 registers a
// thread, so that 4 blocks share an SM (their lists are in shared memory,
// SmemTopK) and more warps hide each other's loads from L2, which bound the
// kernel.
template <typename T, int D, int K, int STACK, bool EXACT>
__global__ void __launch_bounds__(128, 4) k_knn_kdtree_lean(KnnLaunch a) {
  knn_kdtree_body<T, D, K, STACK, EXACT>(a);
}

// Trees of any height: the stacks in a.slab, cap = a.stackCap entries per
// query (or the tree height read from *a.stackHeightDev, plus one, for
// batches whose heights the host does not know). As many threads as the
// slab holds stacks search (the others idle), each taking every active-th
// query. A slab too small for one stack searches nothing and sets
// *a.deepFail to -1.
template <typename T, int D, int K, bool EXACT>
__global__ void __launch_bounds__(128) k_knn_kdtree_deep(KnnLaunch a) {
  if (a.tallGate && *a.tallGate <= a.tallGateLimit) return;  // the local-stack kernel searches (uniform)
  const int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t threads = (int64_t)gridDim.x * blockDim.x;
  const int cap = a.stackCap > 0 ? a.stackCap : (a.stackHeightDev ? *a.stackHeightDev + 1 : 0);
  int64_t active = cap > 0 ? a.slabBytes / ((int64_t)sizeof(StackRec<T, D>) * cap) : 0;
  if (active > threads) active = threads;
  if (active <= 0 && a.nq > 0 && g == 0 && a.deepFail) *a.deepFail = -1;
  uint32_t touched = 0;
  if (g < active) {
    SlabStack<T, D> stk{static_cast<StackRec<T, D>*>(a.slab) + g, active};
    for (int64_t t = g; t < a.nq; t += active) {
      if (a.nqDevice && t >= (int64_t)*a.nqDevice) continue;
      knn_query<T, D, K, EXACT>(a, t, stk, cap, touched);
    }
  }
  add_touched(a, touched);
}

// Bytes of one query's stack in a deep launch's slab, for `cap` entries.
template <typename T, int D>
constexpr size_t deep_stack_bytes(int cap) {
  return sizeof(StackRec<T, D>) * (size_t)cap;
}

template <typename T, int D, int K, int STACK, bool EXACT>
void launch_kdtree_as(int grid, int block, cudaStream_t stream, const KnnLaunch& L) {
  if constexpr (sizeof(T) == 8 && K >= 16)
    k_knn_kdtree_lean<T, D, K, STACK, EXACT><<<grid, block, SearchHeap<T, K>::bytes(block / 32 * L.lanes), stream>>>(L);
  else
    k_knn_kdtree<T, D, K, STACK, EXACT><<<grid, block, 0, stream>>>(L);
}

template <typename T, int D, int K, int STACK>
void launch_kdtree(int grid, int block, cudaStream_t stream, const KnnLaunch& L) {
  if (L.maxError2 == 1.0)
    launch_kdtree_as<T, D, K, STACK, true>(grid, block, stream, L);
  else
    launch_kdtree_as<T, D, K, STACK, false>(grid, block, stream, L);
}

template <typename T, int D, int K>
void launch_kdtree_deep(int grid, cudaStream_t stream, const KnnLaunch& L) {
  constexpr size_t smem = SearchHeap<T, K>::bytes(128);
  if (L.maxError2 == 1.0)
    k_knn_kdtree_deep<T, D, K, true><<<grid, 128, smem, stream>>>(L);
  else
    k_knn_kdtree_deep<T, D, K, false><<<grid, 128, smem, stream>>>(L);
}

// Warp-packet traversal for exact search (epsilon = 0).
//
// The 32 queries of a warp (neighbours along the Morton order) walk the
// tree together: one node sequence for the warp, chosen so that at each
// inner node the child that most lanes see as their near side comes first;
// every lane keeps its own offsets, box distance and top-k, and decides for
// itself whether a node can hold a better neighbour. A node is skipped only
// when no lane wants it, so every lane still examines every point that can
// enter its result. Leaf records are read with warp-uniform addresses
// (broadcast loads) and candidates are inserted after the whole leaf has
// been filtered, so the warp pays for the largest number of insertions of
// any one lane rather than for every point where some lane inserts.
//
// The box distance of a cell is the sequential sum over d of off[d]^2,
// rounded exactly as the point distance is. Rounding is monotone, so a
// point inside the cell is never closer than its cell's bound, and the
// pruning test rd <= head never drops an acceptable point: the result is
// the exact k smallest (dist2, index) pairs -- the brute-force answer.
template <typename T, int D>
__device__ __forceinline__ T box_dist2(const T (&off)[D]) {
  T rd = Ar<T>::mul(off[0], off[0]);
#pragma unroll
  for (int d = 1; d < D; ++d) rd = Ar<T>::add(rd, Ar<T>::mul(off[d], off[d]));
  return rd;
}

template <typename T, int D, int K, int STACK>
__global__ void __launch_bounds__(128) k_knn_kdtree_packet(KnnLaunch a) {
  constexpr unsigned kAll = 0xffffffffu;
  // the reference's self-match rule (nabo/kdtree_cpu.cpp:392-396): without
  // ALLOW_SELF_MATCH a point at distance <= epsilon is skipped; one compare
  // against -1 (everything passes) or epsilon
  const T minDist = a.allowSelf ? T(-1) : Ar<T>::eps();
  const Node<T>* __restrict__ nodes = static_cast<const Node<T>*>(a.nodes);
  const Rec<T, D>* __restrict__ recs = static_cast<const Rec<T, D>*>(a.recs);
  const T* __restrict__ query = static_cast<const T*>(a.query);
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool active = t < a.nq;
  const int64_t qi = active ? (a.order ? (int64_t)a.order[t] : t) : 0;
  T q[D];
#pragma unroll
  for (int d = 0; d < D; ++d) q[d] = (active && d < a.dim) ? query[qi * a.qStride + d] : T(0);
  T maxRadius2 = (T)a.maxRadius2;
  if (a.maxRadii && active) {
    const T r = static_cast<const T*>(a.maxRadii)[qi];
    maxRadius2 = Ar<T>::mul(r, r);
  }
  if (!active) maxRadius2 = -Ar<T>::inf();  // wants nothing
  TopK<T, K> heap;
  heap.init(a.k);
  LeafFilter<T, D> flt;
  flt.init(nullptr, nullptr, q);
  T off[D];
#pragma unroll
  for (int d = 0; d < D; ++d) off[d] = T(0);
  uint32_t sNode[STACK];
  T sOff[STACK][D];
  int sp = 0;
  uint32_t node = 0;
  for (;;) {
    const T rd = box_dist2(off);
    const bool want = rd <= maxRadius2 && rd <= heap.head();
    if (__any_sync(kAll, want)) {
      const Node<T> nd = load_node(nodes, node);
      if (!node_is_leaf(nd.meta)) {
        const int cd = (int)node_dim(nd.meta);
        const T newOff = Ar<T>::sub(pick(q, cd), nd.cut);
        const bool nearRight = newOff > T(0);
        const int votesRight = __popc(__ballot_sync(kAll, want && nearRight));
        const int votes = __popc(__ballot_sync(kAll, want));
        const bool firstRight = 2 * votesRight > votes;
        const uint32_t right = node_payload(nd.meta);
        const uint32_t first = firstRight ? right : node + 1;
        const uint32_t second = firstRight ? node + 1 : right;
        // the second child is this lane's far side iff the first is its near side
        const bool secondFar = nearRight == firstRight;
        T offS[D];
#pragma unroll
        for (int d = 0; d < D; ++d) offS[d] = (d == cd && secondFar) ? newOff : off[d];
        const T rdS = box_dist2(offS);
        const bool wantS = want && rdS <= maxRadius2 && rdS <= heap.head();
        if (__any_sync(kAll, wantS) && sp < STACK) {
          sNode[sp] = second;
#pragma unroll
          for (int d = 0; d < D; ++d) sOff[sp][d] = offS[d];
          ++sp;
        }
#pragma unroll
        for (int d = 0; d < D; ++d)  // the first child is this lane's far side
          if (d == cd && !secondFar) off[d] = newOff;
        node = first;
        continue;
      }
      scan_leaf<T, D, K>(recs, node_start(nd), node_payload(nd.meta), q, maxRadius2, minDist, want, heap, flt);
    }
    if (sp == 0) break;
    --sp;
    node = sNode[sp];
#pragma unroll
    for (int d = 0; d < D; ++d) off[d] = sOff[sp][d];
  }
  if (active) {
    const int f = heap.store(a.k, a.outIdx + qi * a.k, static_cast<T*>(a.outD2) + qi * a.k);
    if (a.found) a.found[qi] = f;
  }
}

// Brute force (nabo/brute_force_cpu.cpp:63-103): every query against every
// point. Doubles, and float clouds of fewer than 512 points or of a range that
// k_bf_tc does not take, run here. The points are staged through shared memory in tiles of 24 KB; a
// thread owns QT queries (blockDim.x apart) and their top-k, so each record
// read from shared memory (a broadcast: every lane reads the same one) feeds
// QT distances. The distance is the reference's separately rounded
// sequential sum. Records are taken J at a time: the J x QT distances are
// computed, each query's smallest is compared with one float threshold,
// min(head, maxRadius^2) (NaN radius: NaN, which passes nothing), and only
// when some distance is at or below its threshold -- rare once the heaps
// are full -- do the group's points take the exact test, the reference's
// radius and self-match rules and the (dist2, index) order against the head
// (nabo/kdtree_cpu.cpp:392-396 with the lower index kept on ties). The
// result, the k smallest pairs, does not depend on the order points are
// offered in.
//
// With gridDim.y > 1 the points are split into chunks of `chunk` (a
// multiple of the tile): block row y offers points [y*chunk, (y+1)*chunk) and
// writes its k best to a.outIdx / a.outD2 + y*partStride, and
// k_bf_merge combines the rows (for searches with too few queries to give
// every SM several blocks).
template <typename T>
__device__ __forceinline__ T bf_threshold(T head, T maxRadius2) {
  return head < maxRadius2 ? head : maxRadius2;
}
__device__ __forceinline__ float fmin_t(float a, float b) { return fminf(a, b); }
__device__ __forceinline__ double fmin_t(double a, double b) { return fmin(a, b); }

// Float brute force filters each group of J points before the reference's
// distance: a = |p|^2 - 2 q.p, D fused multiply-adds per pair from |p|^2
// (computed once per point as the tile is staged, kept in the record's index
// slot, the index itself beside the tile) and -2q. With e the reference's
// distance (separately rounded squares, nabo/kdtree_cpu.cpp:383-391), a
// point it could accept has e <= thr, and then
//   a <= thr - |q|^2 + g (thr + 3 P + 2 |q|^2)
// (the dot product's rounding, bounded with 2|q||p| <= |q|^2 + |p|^2, plus
// e's own rounding and |q|^2's) with g = (D + 2) u / (1 - (D + 2) u),
// u = 2^-24, and P the tile's largest |p|^2; the test's bound
// thr - |q|^2 + 2^-17 (thr + 2 P + 2 |q|^2) exceeds that (g (thr + 3 P +
// 2 |q|^2)) over 4 times for D <= 16 and covers its own rounding, so it
// never drops a point that the exact pass would take. A group that passes
// is computed again exactly, as before.
template <int D>
struct BfFilter {
  float m2q[D];  // -2 q
  float qn;      // |q|^2
  float thrA;    // threshold on a
  __device__ __forceinline__ void init(const float (&q)[D]) {
    qn = 0.0f;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      m2q[d] = -2.0f * q[d];
      qn = fmaf(q[d], q[d], qn);
    }
  }
  // A NaN threshold (an idle slot, or a NaN radius) passes nothing. Where
  // |p|^2, |q|^2 or the bound overflow, thrA is inf or NaN and the test
  // below (!(a > thrA)) passes every group to the exact pass.
  __device__ __forceinline__ void set(float thr, float pmax) {
    thrA = thr != thr ? -__int_as_float(0x7f800000) : (thr - qn) + 0x1p-17f * (thr + 2.0f * pmax + 2.0f * qn);
  }
  __device__ __forceinline__ float eval(const Rec<float, D>& r) const {
    float a = __int_as_float(r.p.idx);
#pragma unroll
    for (int d = 0; d < D; ++d) a = fmaf(m2q[d], r.p.c[d], a);
    return a;
  }
};

template <typename T, int D, int K, int QT, int J>
__global__ void __launch_bounds__(128) k_knn_bruteforce(KnnLaunch a, int64_t chunk, int64_t partStride) {
  constexpr bool kFilter = sizeof(T) == 4;
  const T minDist = a.allowSelf ? T(-1) : Ar<T>::eps();
  // a multiple of J, so that a group never reads past the tile
  constexpr int kTile = (int)((24 * 1024) / sizeof(Rec<T, D>)) / J * J;
  __shared__ Rec<T, D> tile[kTile];
  __shared__ int32_t tileIdx[kFilter ? kTile : 1];  // filter: the points' indices
  __shared__ float warpMax[4];                       // filter: largest |p|^2 per warp
  const Rec<T, D>* __restrict__ recs = static_cast<const Rec<T, D>*>(a.recs);
  const T* __restrict__ query = static_cast<const T*>(a.query);
  const int64_t base0 = (int64_t)blockIdx.x * blockDim.x * QT + threadIdx.x;
  T q[QT][D];
  T maxRadius2[QT];
  T thr[QT];
  int64_t qi[QT];
  bool active[QT];
  TopK<T, K> heap[QT];
  BfFilter<D> flt[kFilter ? QT : 1];
#pragma unroll
  for (int u = 0; u < QT; ++u) {
    const int64_t t = base0 + (int64_t)u * blockDim.x;
    active[u] = t < a.nq;
    qi[u] = active[u] ? (a.order ? (int64_t)a.order[t] : t) : 0;
#pragma unroll
    for (int d = 0; d < D; ++d) q[u][d] = (active[u] && d < a.dim) ? query[qi[u] * a.qStride + d] : T(0);
    maxRadius2[u] = (T)a.maxRadius2;
    if (a.maxRadii && active[u]) {
      const T r = static_cast<const T*>(a.maxRadii)[qi[u]];
      maxRadius2[u] = Ar<T>::mul(r, r);
    }
    // an idle slot wants nothing (a NaN threshold passes no point)
    if (!active[u]) maxRadius2[u] = __builtin_nan("");
    heap[u].init(a.k);
    thr[u] = bf_threshold(heap[u].head(), maxRadius2[u]);
    if constexpr (kFilter) flt[u].init(reinterpret_cast<const float(&)[D]>(q[u]));
  }
  const int64_t first = (int64_t)blockIdx.y * chunk;
  const int64_t last = first + chunk < a.n ? first + chunk : a.n;
  for (int64_t base = first; base < last; base += kTile) {
    const int m = (int)((last - base) < kTile ? (last - base) : kTile);
    __syncthreads();
    if constexpr (kFilter) {
      float pm = 0.0f;
      for (int j = threadIdx.x; j < m; j += blockDim.x) {
        Rec<T, D> r;
        load_rec(recs, base + j, r);
        float pn = 0.0f;
#pragma unroll
        for (int d = 0; d < D; ++d) pn = fmaf(r.p.c[d], r.p.c[d], pn);
        tileIdx[j] = r.p.idx;
        r.p.idx = __float_as_int(pn);
        tile[j] = r;
        pm = fmaxf(pm, pn);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) pm = fmaxf(pm, __shfl_xor_sync(0xffffffffu, pm, o));
      if ((threadIdx.x & 31) == 0) warpMax[threadIdx.x >> 5] = pm;
    } else {
      const uint4* src = reinterpret_cast<const uint4*>(recs + base);
      uint4* dst = reinterpret_cast<uint4*>(tile);
      const int words = m * RecSize<T, D>::chunks;
      for (int w = threadIdx.x; w < words; w += blockDim.x) dst[w] = __ldg(src + w);
    }
    {
      // the last group's missing points: NaN coordinates (and |p|^2), whose
      // distance passes no threshold and lowers no minimum (a group's first
      // point is always a real one)
      const int padEnd = (m + J - 1) / J * J;
      for (int j = m + (int)threadIdx.x; j < padEnd; j += blockDim.x) {
        Rec<T, D> r;
#pragma unroll
        for (int d = 0; d < D; ++d) r.p.c[d] = __builtin_nan("");
        r.p.idx = kFilter ? __float_as_int(__builtin_nanf("")) : -1;
        tile[j] = r;
      }
    }
    __syncthreads();
    if constexpr (kFilter) {
      const float pmax = fmaxf(fmaxf(warpMax[0], warpMax[1]), fmaxf(warpMax[2], warpMax[3]));
#pragma unroll
      for (int u = 0; u < QT; ++u) flt[u].set((float)thr[u], pmax);
      for (int j0 = 0; j0 < m; j0 += J) {
        float amin[QT];
#pragma unroll
        for (int jj = 0; jj < J; ++jj) {
          const Rec<T, D> r = tile[j0 + jj];
#pragma unroll
          for (int u = 0; u < QT; ++u) {
            const float av = flt[u].eval(reinterpret_cast<const Rec<float, D>&>(r));
            amin[u] = jj == 0 ? av : fminf(amin[u], av);
          }
        }
        bool any = false;
#pragma unroll
        for (int u = 0; u < QT; ++u) any = any || !(amin[u] > flt[u].thrA);
        if (any) {  // rare once the heaps are full: the group exactly
#pragma unroll
          for (int jj = 0; jj < J; ++jj) {
            if (j0 + jj < m) {
              const Rec<T, D> r = tile[j0 + jj];
              const int idx = tileIdx[j0 + jj];
#pragma unroll
              for (int u = 0; u < QT; ++u) {
                const T d = dist2_seq(q[u], r);
                if (d <= thr[u] && d <= maxRadius2[u] && heap[u].accepts(d, idx) && d > minDist) {
                  heap[u].insert(d, idx);
                  thr[u] = bf_threshold(heap[u].head(), maxRadius2[u]);
                  flt[u].set((float)thr[u], pmax);
                }
              }
            }
          }
        }
      }
    } else {
      for (int j0 = 0; j0 < m; j0 += J) {
        // each query's smallest distance of the group (fmin ignores the NaN
        // padding; the group's first point is a real one)
        T dmin[QT];
#pragma unroll
        for (int jj = 0; jj < J; ++jj) {
          const Rec<T, D> r = tile[j0 + jj];
#pragma unroll
          for (int u = 0; u < QT; ++u) {
            const T d = dist2_seq(q[u], r);
            dmin[u] = jj == 0 ? d : fmin_t(dmin[u], d);
          }
        }
        bool any = false;
#pragma unroll
        for (int u = 0; u < QT; ++u) any = any || dmin[u] <= thr[u];
        if (any) {  // rare once the heaps are full: the group again, exactly
#pragma unroll
          for (int jj = 0; jj < J; ++jj) {
            if (j0 + jj < m) {
              const Rec<T, D> r = tile[j0 + jj];
#pragma unroll
              for (int u = 0; u < QT; ++u) {
                const T d = dist2_seq(q[u], r);
                if (d <= thr[u] && d <= maxRadius2[u] && heap[u].accepts(d, r.p.idx) && d > minDist) {
                  heap[u].insert(d, r.p.idx);
                  thr[u] = bf_threshold(heap[u].head(), maxRadius2[u]);
                }
              }
            }
          }
        }
      }
    }
  }
  const int64_t part = (int64_t)blockIdx.y * partStride;
#pragma unroll
  for (int u = 0; u < QT; ++u) {
    if (active[u]) {
      const int f = heap[u].store(a.k, a.outIdx + part + qi[u] * a.k, static_cast<T*>(a.outD2) + part + qi[u] * a.k);
      if (a.found) a.found[qi[u]] = f;
    }
  }
}

// The k best of `parts` partial results per query (each k entries, ascending,
// unfound slots index -1), written as the search's result.
template <typename T, int K>
__global__ void k_bf_merge(const int32_t* __restrict__ pIdx, const T* __restrict__ pD2, int parts, int64_t partStride,
                           int64_t nq, int k, int32_t* outIdx, T* outD2, int32_t* found) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nq) return;
  TopK<T, K> heap;
  heap.init(k);
  for (int p = 0; p < parts; ++p) {
    const int64_t o = p * partStride + i * k;
    for (int j = 0; j < k; ++j) {
      const int32_t idx = pIdx[o + j];
      if (idx < 0) break;
      const T d = pD2[o + j];
      if (heap.accepts(d, idx)) heap.insert(d, idx);
    }
  }
  const int f = heap.store(k, outIdx + i * k, outD2 + i * k);
  if (found) found[i] = f;
}

// Shape of the brute force: QT queries per thread (more share each
// shared-memory read, fewer keep long top-k lists in registers) and J
// records per threshold test.
// Float, with the |p|^2 - 2 q.p filter, 100k x 100k 3-D points (kernel ms,
// k = 5 / k = 10): QT x J = 1 x 4 3.50 / 4.79, 1 x 8 3.51 / 5.06, 1 x 12
// 3.76 / 5.95, 2 x 4 3.92 / 6.63, 3 x 4 4.54 / 8.17, 1 x 16 4.59 / 6.58,
// 2 x 8 4.80 / 8.19, 4 x 4 5.89 / 10.97, 4 x 8 8.76 / 18.12.
// Before the filter (separately rounded distances for every pair, k = 5):
// 2 x 4 5.17, 2 x 8 5.72, 1 x 8 6.33, 4 x 4 6.83, 1 x 4 6.90, 4 x 8 7.88,
// 8 x 2 8.49; double, which keeps that kernel, uses 1 x 4.
template <typename T, int K>
struct BfShape {
  static constexpr int QT = 1;
  static constexpr int J = 4;
};

}  // namespace nabo_gb300
