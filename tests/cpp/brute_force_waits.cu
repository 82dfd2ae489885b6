// The float brute force when its pipeline's waits give up: each block then
// searches its queries without it, so results stay those of a plain search.
// Runs knn_bruteforce over objects of the library with the poll limit given.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <utility>
#include <vector>

#include "internal.cuh"

using namespace nabo_gb300;

#define CHECK(x)                                                                           \
  do {                                                                                     \
    if (!(x)) {                                                                            \
      std::printf("FAIL %s:%d %s (%s)\n", __FILE__, __LINE__, #x, nabo_cuda_last_error()); \
      std::exit(1);                                                                        \
    }                                                                                      \
  } while (0)

template <int D>
void run(int64_t n, int64_t nq, int k) {
  std::mt19937 rng(7u + (unsigned)n + D);
  std::uniform_real_distribution<float> u(0.0f, 1.0f);
  std::vector<float> cloud(n * D), query(nq * D);
  for (float& x : cloud) x = u(rng);
  for (float& x : query) x = u(rng);
  // the reference's distance: separately rounded squares, summed in order
  std::vector<std::pair<float, int>> want;
  for (int64_t q = 0; q < nq; ++q) {
    std::vector<std::pair<float, int>> all(n);
    for (int64_t i = 0; i < n; ++i) {
      float s = 0.0f;
      for (int d = 0; d < D; ++d) {
        const float x = query[q * D + d] - cloud[i * D + d];
        s += x * x;
      }
      all[i] = {s, (int)i};
    }
    std::partial_sort(all.begin(), all.begin() + k, all.end());
    want.insert(want.end(), all.begin(), all.begin() + k);
  }
  nabo_cuda_search* h = nullptr;
  CHECK(nabo_cuda_create(NABO_CUDA_FLOAT32, cloud.data(), D, n, D, D, NABO_SEARCH_BRUTE_FORCE_CUDA, 0, nullptr, &h) == 0);
  float *dq, *dd;
  int32_t* di;
  CHECK(cudaMalloc(&dq, query.size() * 4) == cudaSuccess);
  CHECK(cudaMalloc(&dd, nq * k * 4) == cudaSuccess);
  CHECK(cudaMalloc(&di, nq * k * 4) == cudaSuccess);
  CHECK(cudaMemcpy(dq, query.data(), query.size() * 4, cudaMemcpyHostToDevice) == cudaSuccess);
  cudaStream_t st;
  CHECK(cudaStreamCreate(&st) == cudaSuccess);
  KnnArgs a;
  const int normal = a.waitPolls;
  a.query = dq;
  a.nq = nq;
  a.qStride = D;
  a.k = k;
  a.optionFlags = NABO_ALLOW_SELF_MATCH | NABO_SORT_RESULTS;
  a.maxRadius = __builtin_huge_val();
  a.indices = di;
  a.dists2 = dd;
  for (int polls : {0, 1, 2, 8, 64, normal}) {
    a.waitPolls = polls;
    CHECK(cudaMemset(di, 0xff, nq * k * 4) == cudaSuccess);
    CHECK((knn_bruteforce<float, D>(*handle_view(h).cloud, a, st) == 0));
    std::vector<float> d2(nq * k);
    std::vector<int32_t> idx(nq * k);
    CHECK(cudaStreamSynchronize(st) == cudaSuccess);
    CHECK(cudaMemcpy(d2.data(), dd, nq * k * 4, cudaMemcpyDeviceToHost) == cudaSuccess);
    CHECK(cudaMemcpy(idx.data(), di, nq * k * 4, cudaMemcpyDeviceToHost) == cudaSuccess);
    for (int64_t i = 0; i < nq * k; ++i) CHECK(d2[i] == want[i].first && idx[i] == want[i].second);
  }
  std::printf("ok D=%d n=%lld nq=%lld k=%d\n", D, (long long)n, (long long)nq, k);
  CHECK(nabo_cuda_destroy(h) == 0);
}

int main() {
  run<3>(20000, 700, 5);   // parts of the points per block row, several stages
  run<3>(3000, 129, 1);
  run<3>(9000, 300, 20);   // two accumulators
  run<8>(7000, 200, 10);
  run<16>(4000, 150, 32);
}
