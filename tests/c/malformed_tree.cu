// The walk over a tree whose root claims children that its slots cannot hold: prints the error word and
// the child tests made, a line for each five arguments: points, points per traversal (1, 16 or 32),
// dimensions, the root's first child slot, its count of children.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../d3-force-3d-webgpu_gb300/csrc/kernels.h"

#define CK(x)                                                                          \
  do {                                                                                 \
    cudaError_t e_ = (x);                                                              \
    if (e_ != cudaSuccess) return std::printf("%s: %s\n", #x, cudaGetErrorString(e_)), 1; \
  } while (0)

static int walk(char** arg) {
  const int n = std::atoi(arg[0]), group = std::atoi(arg[1]), ndim = std::atoi(arg[2]);
  const uint32_t first = (uint32_t)std::strtoul(arg[3], nullptr, 10), count = (uint32_t)std::strtoul(arg[4], nullptr, 10);
  void* tree;
  const size_t bytes = fl_tree_bytes(n);
  CK(cudaMalloc(&tree, bytes));
  CK(cudaMemset(tree, 0, bytes));
  FlTreeBufs t;
  fl_tree_carve(&t, tree, n, ndim);
  std::vector<float4> leaf(n);
  std::vector<uint32_t> perm(n);
  for (int i = 0; i < n; ++i) leaf[i] = make_float4(1.f + i, 2.f + i, 3.f + i, -30.f), perm[i] = i;
  const float cube[5] = {0.f, 0.f, 0.f, 1e6f, 20.f};  // wide: every cell is opened
  const float4 root = make_float4(0.5f, 0.25f, 0.125f, -30.f);
  const uint2 meta = make_uint2(first, count);
  float4* vel;
  float* dcube;
  uint32_t *dperm, *err;
  unsigned long long* stats;
  CK(cudaMalloc(&vel, 16 * n));
  CK(cudaMalloc(&dcube, sizeof(cube)));
  CK(cudaMalloc(&dperm, 4 * n));
  CK(cudaMalloc(&err, 4));
  CK(cudaMalloc(&stats, 48));
  CK(cudaMemset(vel, 0, 16 * n));
  CK(cudaMemset(err, 0, 4));
  CK(cudaMemset(stats, 0, 48));
  CK(cudaMemcpy(dcube, cube, sizeof(cube), cudaMemcpyHostToDevice));
  CK(cudaMemcpy(dperm, perm.data(), 4 * n, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(t.leaf, leaf.data(), 16 * n, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(t.child_data, &root, 16, cudaMemcpyHostToDevice));
  CK(cudaMemcpy(t.child_meta, &meta, 8, cudaMemcpyHostToDevice));
  fl_launch_walk(&t, dperm, dcube, vel, 0.5f, 0.81, 1.0, 1e300, 0, 0, err, stats, group, nullptr);
  CK(cudaGetLastError());
  CK(cudaDeviceSynchronize());
  uint32_t e = 0;
  unsigned long long s[6];
  CK(cudaMemcpy(&e, err, 4, cudaMemcpyDeviceToHost));
  CK(cudaMemcpy(s, stats, 48, cudaMemcpyDeviceToHost));
  std::printf("%u %llu\n", e, s[0]);
  cudaFree(tree), cudaFree(vel), cudaFree(dcube), cudaFree(dperm), cudaFree(err), cudaFree(stats);
  return 0;
}

int main(int argc, char** argv) {
  for (int k = 1; k + 4 < argc; k += 5)
    if (const int rc = walk(argv + k)) return rc;
  return 0;
}
