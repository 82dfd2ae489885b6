// A kd-tree build whose blocks give up waiting for each other at the grid
// barrier: the build ends, reports that it did not finish, and leaves one leaf
// per cloud that holds the cloud's points, each once.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "internal.cuh"

using namespace nabo_gb300;

#define CHECK(x)                                                      \
  do {                                                                \
    if (!(x)) {                                                       \
      std::printf("FAIL %s:%d %s\n", __FILE__, __LINE__, #x);         \
      std::exit(1);                                                   \
    }                                                                 \
  } while (0)

int main() {
  const int64_t n = 150000, clouds = 2;
  std::mt19937 rng(5);
  std::uniform_real_distribution<float> u(0.0f, 1.0f);
  std::vector<float> cloud(n * 3);
  for (float& x : cloud) x = u(rng);
  const std::vector<int64_t> off = {0, 50000, n};
  float* dCloud;
  int64_t *dOff, *nodeOffset;
  Rec<float, 3>* recs;
  Node<float>* nodes;
  float* box;
  int* status;
  CHECK(cudaMalloc(&dCloud, cloud.size() * 4) == cudaSuccess);
  CHECK(cudaMalloc(&dOff, 3 * 8) == cudaSuccess);
  CHECK(cudaMalloc(&nodeOffset, 3 * 8) == cudaSuccess);
  CHECK(cudaMalloc(&recs, n * sizeof(*recs)) == cudaSuccess);
  CHECK(cudaMalloc(&nodes, 2 * n * sizeof(*nodes)) == cudaSuccess);
  CHECK(cudaMalloc(&box, 2 * clouds * kMaxDim * 4) == cudaSuccess);
  CHECK(cudaMalloc(&status, 16) == cudaSuccess);
  CHECK(cudaMemcpy(dCloud, cloud.data(), cloud.size() * 4, cudaMemcpyHostToDevice) == cudaSuccess);
  CHECK(cudaMemcpy(dOff, off.data(), 3 * 8, cudaMemcpyHostToDevice) == cudaSuccess);
  cudaStream_t st;
  CHECK(cudaStreamCreate(&st) == cudaSuccess);
  ForestOut f;
  f.recs = recs;
  f.nodes = nodes;
  f.nodeCap = 2 * n;
  f.nodeOffset = nodeOffset;
  f.rootLo = box;
  f.rootHi = box + clouds * kMaxDim;
  f.status = status;
  const int normal = f.barrierPolls;
  for (int polls : {0, 2, normal}) {
    f.barrierPolls = polls;
    CHECK((build_forest<float, 3>(dCloud, n, 3, 3, 8, dOff, (int)clouds, -1, st, &f, 0) == 0));
    int hs[4];
    int64_t no[3];
    CHECK(cudaStreamSynchronize(st) == cudaSuccess);
    CHECK(cudaMemcpy(hs, status, 16, cudaMemcpyDeviceToHost) == cudaSuccess);
    CHECK(cudaMemcpy(no, nodeOffset, 24, cudaMemcpyDeviceToHost) == cudaSuccess);
    CHECK(hs[0] == 0);
    CHECK(polls != 0 || hs[1] == 1);
    CHECK(polls != normal || hs[1] == 0);
    if (hs[1]) CHECK(no[1] == 1 && no[2] == 2);
    std::vector<Rec<float, 3>> r(n);
    CHECK(cudaMemcpy(r.data(), recs, n * sizeof(r[0]), cudaMemcpyDeviceToHost) == cudaSuccess);
    for (int64_t c = 0; c < clouds; ++c) {
      std::vector<char> seen(off[c + 1] - off[c], 0);
      for (int64_t p = off[c]; p < off[c + 1]; ++p) {
        const int32_t i = r[p].p.idx;
        CHECK(i >= 0 && i < (int64_t)seen.size() && !seen[i]);
        seen[i] = 1;
        for (int d = 0; d < 3; ++d) CHECK(r[p].p.c[d] == cloud[(off[c] + i) * 3 + d]);
      }
    }
    std::printf("ok polls=%d finished=%d\n", polls, hs[1] == 0);
  }
}
