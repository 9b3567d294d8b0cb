// Launches of the layer's kernels as a chain.  A layer call is a sequence of dependent kernels, many of them shorter than
// what lies between two kernels of a stream: the drain of one, the launch of the next, its barriers, tensor memory and
// descriptor fetches (2 to 4 us each time).  Programmatic dependent launch lets a kernel's blocks come up while the previous
// kernel's last ones still run, and takes the launch itself off the way.  Without it and with it, medians of four alternating
// runs: one token of a layer with H 2048, I 768, E 64, K 4 59.4 / 54.0 us a call, 64 tokens, H 4096, I 1024, E 128, K 8 530 / 516, 1027
// tokens, H 4096, I 512, E 256, K 16 732 / 723, training steps of T 8197, H 2048, I 1024, E 64, K 1 778 / 760 and of T 8191, H 1024,
// I 512, E 32, K 4, GELU with biases, 422 / 396; T 24576, H 1536, I 256, E 128, K 8 1943 / 1944.
// The contract of every kernel launched through launch_chained:
//   * wait_for_previous() in every thread before the first access to global memory (what is before it works on registers,
//     shared and tensor memory alone).  It returns once the previous kernel of the stream is complete and its writes are
//     visible, and that kernel in turn has waited for its own predecessor, so the order of a stream is kept;
//   * release_next() at the start of kernels whose blocks do one short piece of work each: the next kernel's blocks may then
//     take what room is left once the last block has started.  It promises nothing about results.  Not in kernels whose blocks
//     stay for many pieces (the GEMMs, the router): their end releases the next one.  A grid that is released before its blocks
//     find room stands in front of the other streams' grids, and with a release at the start of every GEMM a second stream
//     did not get on until the chain ended: 40 small kernels beside a training step of T 32768, H 4096, I 1024, E 128, K 8 took
//     20 ms, the whole step, instead of 1.2.  The release at the end costs next to nothing: one token 55 -> 54 us, 1027 tokens, H 4096, I
//     512, E 256, K 16 730 -> 724, training steps of T 24576, H 1536, I 256, E 128, K 8 1998 -> 1995 and of T 8197, H 2048, I 1024, E 64,
//     K 1 763 -> 767 (means of three to five alternating runs).
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
