// Launches of the layer's kernels as a chain.  A layer call is a sequence of dependent kernels, many of them shorter than
// what lies between two kernels of a stream: the drain of one, the launch of the next, its barriers, tensor memory and
// descriptor fetches (2 to 4 us each time).  Programmatic dependent launch lets a kernel's blocks come up while the previous
// kernel's last ones still run.  One token of a layer with H 2048, I 768, E 64, K 4: 72 -> 64 us a call; a training step of
// 2048 tokens, H 768, I 256, E 8, K 2: 610 -> 579; 64 tokens, H 4096, I 1024, E 128, K 8: 547 -> 540; steps of milliseconds
// are the same.  The contract of every kernel launched through launch_chained:
//   * wait_for_previous() in every thread before the first access to global memory (what is before it works on registers,
//     shared and tensor memory alone).  It returns once the previous kernel of the stream is complete and its writes are
//     visible, and that kernel in turn has waited for its own predecessor, so the order of a stream is kept;
//   * release_next() in every block once the block holds all it needs (shared and tensor memory): the next kernel's blocks
//     may then take what room is left.  It promises nothing about results.
// Pointers that such a kernel loads from are not __restrict__: loads that the compiler takes to be of constant memory could
// move in front of the wait.
#pragma once
#include <cuda_runtime.h>

#include <utility>

#include "device_cache.cuh"

namespace smoe {

__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void release_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// `cluster` blocks per cluster (1: none).
template <class... Params, class... Args>
inline cudaError_t launch_chained(void (*kernel)(Params...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream,
                                  unsigned cluster, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace smoe
