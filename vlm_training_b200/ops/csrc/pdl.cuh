// Programmatic dependent launch: a kernel launched through `launch_pdl` may start while the kernel before it in its stream drains, so
// its launch latency and set-up (barriers, tensor memory, shared memory) are off the critical path.  Such a kernel
//   * calls pdl_wait() in every thread before it touches global memory (reads and writes; its own parameters are free, and so are prefetches
//     of data into L2, which is where the GPU's memory is coherent): the call returns when the kernels before it have completed and their writes are visible, as without the attribute;
//   * calls it on every path, also in blocks that have nothing to do: a grid that ends without waiting would no longer order what follows
//     it behind what precedes it.
//   * if it allocates tensor memory, calls pdl_trigger() behind the allocation: the GEMMs allocate before they wait, and a block of theirs
//     on the same SM would hold the columns until this kernel ends, which would wait for them without a bound.
// pdl_trigger() lets the next kernel of the stream be launched into free resources once every block has called it (or exited).  Blocks
// that are launched ahead hold registers and thread slots while they wait, so long kernels call it near their end: at the start of the
// GEMMs it kept the optimizer's updates, which run beside them on a stream of their own, off the SMs (256 experts, 8192 tokens 5.14 -> 5.31 ms).
// Kernels that wait for another GPU do not call it.
// On graphs of equal GEMMs a launch costs 0.8 to 1.5 us less (90 x 1152 x 1152 10.4 -> 8.7 us); one new token of a chat, 37 tokens,
// 47 launches 859 -> 760 us.
#pragma once
#include <cuda_runtime.h>

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Small grids let the next kernel in at once, larger ones when their blocks exit, for the reason above (256 experts, 16384 tokens 6.59 -> 6.68 ms
// with all of them).
__device__ __forceinline__ void pdl_trigger_small() { if (gridDim.x * gridDim.y * gridDim.z <= 296) pdl_trigger(); }
// First statement of a kernel that needs nothing set up before and no tensor memory, and that is over in tens of microseconds where it has so
// few blocks.
__device__ __forceinline__ void pdl_begin() {
  pdl_wait();
  pdl_trigger_small();
}

template <typename... P, typename... A>
inline int launch_pdl(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, int cluster, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = cluster > 1 ? 2 : 1;
  return (int)cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}
