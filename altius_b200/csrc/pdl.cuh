// Programmatic dependent launch: a kernel that is launched through launch_pdl may start while the
// kernel in front of it on the stream still drains. Its prologue (barriers, tables, loads of
// constants) then runs under the predecessor's tail; `pdl_wait` returns once every earlier kernel
// has completed and its writes are visible, so nothing produced by the schedule may be read, and
// nothing at all written, in front of it. Every thread calls it: a block that left without
// waiting would let the chain of completions run ahead of its own predecessors.
#pragma once
#include <cuda_runtime.h>

namespace ac {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The dependent grid may be scheduled once all blocks have said so (or left).
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Loads of what the schedule computes. Not __ldg: the read-only path is for memory that nobody writes
// while the grid exists, and a grid launched this way exists while its predecessors write.
template <typename T>
__device__ __forceinline__ T ld_plain(const T* p) {
  return *p;
}

// `cluster`: blocks per cluster along z (1: none; 0: none, and no overlap either).
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, int cluster,
                       Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = cluster > 0 ? 1 : 0;
  if (cluster > 1) {
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = 1; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = (unsigned)cluster;
    cfg.numAttrs = 2;
  }
  cfg.attrs = at;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

}  // namespace ac
