// octant.cu - the octant copies of a tree's nodes (ONode, device.h).
//
// A file of its own: a program's first build loads this small module, not the
// traversal kernels', which its first trace loads (first mesh build of a process
// 18 ms with the kernels in that module, 0.5 here).
#include <cuda_runtime.h>

#include "device.h"

namespace vmr {
namespace {

// Octant copies of the nodes (octant_child, octant_mchild), a thread per child: a
// thread per copy left trees of few nodes waiting for its chain of loads and stores.
__global__ void k_octant_mnodes(const MNode* __restrict__ nodes, const float* __restrict__ boxes, uint32_t keys,
                                uint32_t n, ONode* __restrict__ out, int* bad) {
  const uint64_t per = (uint64_t)keys * n, total = per * 32;
  for (uint64_t g = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; g < total; g += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t kn = (g >> 2) % per;
    if (!octant_mchild(nodes[kn % n], boxes + kn * 24, (unsigned)g & 3u, (unsigned)(g / (4 * per)), out[g >> 2])) *bad = 1;
  }
}

__global__ void k_octant_nodes(const GNode* __restrict__ nodes, uint32_t n, ONode* __restrict__ out) {
  const uint64_t total = (uint64_t)n * 32;
  for (uint64_t g = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; g < total; g += (uint64_t)gridDim.x * blockDim.x)
    octant_child(nodes[(g >> 2) % n], (unsigned)g & 3u, (unsigned)(g / (4ull * n)), out[g >> 2]);
}

}  // namespace

int launch_octant_nodes(const GNode* nodes, uint32_t n, ONode* out, void* stream) {
  const uint64_t want = ((uint64_t)n * 32 + 127) / 128, cap = (uint64_t)device_sm_count() * 32;
  k_octant_nodes<<<(int)(want < cap ? want : cap), 128, 0, (cudaStream_t)stream>>>(nodes, n, out);
  return (int)cudaGetLastError();
}

int launch_octant_mnodes(const MNode* nodes, const void* mboxes, uint32_t keys, uint32_t n, ONode* out, int* bad,
                         void* stream) {
  const uint64_t want = ((uint64_t)n * keys * 32 + 127) / 128, cap = (uint64_t)device_sm_count() * 32;
  cudaMemsetAsync(bad, 0, sizeof(int), (cudaStream_t)stream);
  k_octant_mnodes<<<(int)(want < cap ? want : cap), 128, 0, (cudaStream_t)stream>>>(
      nodes, static_cast<const float*>(mboxes), keys, n, out, bad);
  return (int)cudaGetLastError();
}

}  // namespace vmr
