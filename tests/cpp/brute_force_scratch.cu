// The brute force's scratch. This program's scratch_alloc takes the place of
// the library's (which calls it by its exported name) and counts the calls or
// refuses them: a search that gets none runs in one row with the same results,
// and a captured search with many queries asks for none, so that its graph can
// be instantiated more than once.
#include <cuda_runtime.h>
#include <dlfcn.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "internal.cuh"

static bool g_refuse = false;
static int g_calls = 0;

namespace nabo_gb300 {
cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t stream) {
  ++g_calls;
  if (g_refuse) return cudaErrorMemoryAllocation;
  using F = cudaError_t (*)(void**, size_t, cudaStream_t);
  static const F real = (F)dlsym(RTLD_NEXT, "_ZN10nabo_gb30013scratch_allocEPPvmP11CUstream_st");
  return real(p, bytes, stream);
}
}  // namespace nabo_gb300

using namespace nabo_gb300;

#define CHECK(x)                                                                           \
  do {                                                                                     \
    if (!(x)) {                                                                            \
      std::printf("FAIL %s:%d %s (%s)\n", __FILE__, __LINE__, #x, nabo_cuda_last_error()); \
      std::exit(1);                                                                        \
    }                                                                                      \
  } while (0)

template <typename T>
void run(int64_t n, int64_t nq, int k, bool capture) {
  const int D = 3;
  std::mt19937 rng(9u);
  std::uniform_real_distribution<T> u(0, 1);
  std::vector<T> cloud(n * D), query(nq * D);
  for (T& x : cloud) x = u(rng);
  for (T& x : query) x = u(rng);
  nabo_cuda_search* h = nullptr;
  const int dtype = sizeof(T) == 4 ? NABO_CUDA_FLOAT32 : NABO_CUDA_FLOAT64;
  CHECK(nabo_cuda_create(dtype, cloud.data(), D, n, D, D, NABO_SEARCH_BRUTE_FORCE_CUDA, 0, nullptr, &h) == 0);
  T *dq, *dd;
  int32_t* di;
  const size_t entries = (size_t)nq * k;
  CHECK(cudaMalloc(&dq, query.size() * sizeof(T)) == cudaSuccess);
  CHECK(cudaMalloc(&dd, entries * sizeof(T)) == cudaSuccess);
  CHECK(cudaMalloc(&di, entries * 4) == cudaSuccess);
  CHECK(cudaMemcpy(dq, query.data(), query.size() * sizeof(T), cudaMemcpyHostToDevice) == cudaSuccess);
  cudaStream_t st;
  CHECK(cudaStreamCreate(&st) == cudaSuccess);
  const auto search = [&]() {
    return nabo_cuda_knn_device(h, dq, D, nq, D, k, 0.0, NABO_ALLOW_SELF_MATCH | NABO_SORT_RESULTS, __builtin_huge_val(),
                                nullptr, di, dd, nullptr, st);
  };
  const auto result = [&]() {
    std::vector<char> r(entries * (4 + sizeof(T)));
    CHECK(cudaStreamSynchronize(st) == cudaSuccess);
    CHECK(cudaMemcpy(r.data(), di, entries * 4, cudaMemcpyDeviceToHost) == cudaSuccess);
    CHECK(cudaMemcpy(r.data() + entries * 4, dd, entries * sizeof(T), cudaMemcpyDeviceToHost) == cudaSuccess);
    CHECK(cudaMemset(di, 0xff, entries * 4) == cudaSuccess);
    return r;
  };
  g_calls = 0;
  CHECK(search() == 0);
  const std::vector<char> want = result();
  if (!capture) {
    CHECK(g_calls > 0);  // a search in rows: otherwise nothing is refused below
    g_refuse = true;
    CHECK(search() == 0);
    g_refuse = false;
    CHECK(result() == want);
  } else {
    cudaGraph_t graph;
    cudaGraphExec_t exec[2];
    g_calls = 0;
    CHECK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) == cudaSuccess);
    CHECK(search() == 0);
    CHECK(cudaStreamEndCapture(st, &graph) == cudaSuccess);
    CHECK(g_calls == 0);
    for (cudaGraphExec_t& e : exec) CHECK(cudaGraphInstantiate(&e, graph, 0) == cudaSuccess);
    for (cudaGraphExec_t e : exec) {
      CHECK(cudaGraphLaunch(e, st) == cudaSuccess);
      CHECK(result() == want);
    }
  }
  std::printf("ok n=%lld nq=%lld k=%d\n", (long long)n, (long long)nq, k);
  CHECK(nabo_cuda_destroy(h) == 0);
}

int main() {
  run<float>(100000, 500, 5, false);
  run<float>(20000, 1, 20, false);
  run<double>(100000, 500, 5, false);
  run<float>(100000, 160000, 5, true);
  run<float>(5000, 20000, 10, true);
  run<float>(30000, 200000, 1, true);
}
