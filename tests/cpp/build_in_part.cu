// Builds on a stream that may use some of the device's SMs only (a green
// context's): the trees are those built on the whole device.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "nabo_gb300.h"

#define CHECK(x)                                                                           \
  do {                                                                                     \
    if (!(x)) {                                                                            \
      std::printf("FAIL %s:%d %s (%s)\n", __FILE__, __LINE__, #x, nabo_cuda_last_error()); \
      std::exit(1);                                                                        \
    }                                                                                      \
  } while (0)

struct Tree {
  std::vector<uint32_t> right, start, count;
  std::vector<int32_t> cutDim, buckets;
  std::vector<double> cut;
  bool operator==(const Tree& o) const {
    return right == o.right && start == o.start && count == o.count && cutDim == o.cutDim && buckets == o.buckets &&
           cut == o.cut;
  }
};

template <typename T>
static Tree build(const std::vector<T>& cloud, int dim, cudaStream_t st) {
  const int64_t n = (int64_t)cloud.size() / dim;
  T* d;
  CHECK(cudaMalloc(&d, cloud.size() * sizeof(T)) == cudaSuccess);
  CHECK(cudaMemcpy(d, cloud.data(), cloud.size() * sizeof(T), cudaMemcpyHostToDevice) == cudaSuccess);
  nabo_cuda_batch* b = nullptr;
  CHECK(nabo_cuda_batch_create(sizeof(T) == 4 ? NABO_CUDA_FLOAT32 : NABO_CUDA_FLOAT64, dim, 1, &n, nullptr, 0, &b) == 0);
  CHECK(nabo_cuda_batch_build_device(b, d, st) == 0);
  CHECK(cudaStreamSynchronize(st) == cudaSuccess);
  int64_t status[8], nodes = 0;
  CHECK(nabo_cuda_batch_status(b, status) == 0 && status[0] == 0);
  CHECK(nabo_cuda_batch_export_tree(b, 0, &nodes, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr) == 0);
  Tree t;
  t.right.resize(nodes);
  t.start.resize(nodes);
  t.count.resize(nodes);
  t.cutDim.resize(nodes);
  std::vector<T> cut(nodes);
  t.buckets.resize(n);
  CHECK(nabo_cuda_batch_export_tree(b, 0, &nodes, t.cutDim.data(), cut.data(), t.right.data(), t.start.data(),
                                    t.count.data(), t.buckets.data()) == 0);
  t.cut.assign(cut.begin(), cut.end());
  CHECK(nabo_cuda_batch_destroy(b) == 0);
  CHECK(cudaFree(d) == cudaSuccess);
  return t;
}

template <typename T>
static void check(int64_t n, int dim, cudaStream_t st) {
  std::mt19937 rng(3);
  std::uniform_real_distribution<T> u(0, 1);
  std::vector<T> c(n * dim);
  for (T& x : c) x = u(rng);
  for (int64_t i = 0; i < n; i += 5) c[i * dim] = T(0.5);  // points on a cut
  const Tree want = build(c, dim, nullptr);
  CHECK(want.right.size() > 1);
  CHECK(build(c, dim, st) == want);
  std::printf("ok n=%lld D=%d\n", (long long)n, dim);
}

int main() {
  CHECK(cudaFree(nullptr) == cudaSuccess);
  CUdevResource all, part;
  unsigned groups = 1;
  CUdevResourceDesc desc;
  CUgreenCtx green;
  CUstream st;
  if (cuDeviceGetDevResource(0, &all, CU_DEV_RESOURCE_TYPE_SM) != CUDA_SUCCESS ||
      cuDevSmResourceSplitByCount(&part, &groups, &all, nullptr, 0, 16) != CUDA_SUCCESS ||
      cuDevResourceGenerateDesc(&desc, &part, 1) != CUDA_SUCCESS ||
      cuGreenCtxCreate(&green, desc, 0, CU_GREEN_CTX_DEFAULT_STREAM) != CUDA_SUCCESS ||
      cuGreenCtxStreamCreate(&st, green, CU_STREAM_NON_BLOCKING, 0) != CUDA_SUCCESS) {
    std::printf("no green context\n");
    return 77;
  }
  std::printf("%u of %u SMs\n", part.sm.smCount, all.sm.smCount);
  for (int64_t n : {3000, 20000, 90000, 1200000}) check<float>(n, 3, st);
  // so many positions a block that its lists do not fit in shared memory
  check<double>(2500000, 16, st);
  CHECK(cudaStreamDestroy(st) == cudaSuccess);
  CHECK(cuGreenCtxDestroy(green) == CUDA_SUCCESS);
}
