// Launches that overlap the end of the kernel before them (programmatic
// dependent launch).  A kernel launched by launchAfter may start once every
// thread block of the one before it in the stream has called afterPrevious or
// ended; what it reads before its own afterPrevious must not come from the
// kernel right before it (the kernels before that one have ended by then).
// What it reads after is complete.  Pointers to such data are not
// `const __restrict__`: read-only loads could be moved ahead of the wait.
#pragma once

#include <cuda_runtime.h>

namespace bfg {

// waits for the kernels before (at once if launched the plain way), then lets
// the next one start
__device__ __forceinline__ void afterPrevious() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// the same in clusters of `cluster` consecutive thread blocks
template <typename... P, typename... A>
cudaError_t launchAfterClusters(void (*kernel)(P...), int cluster, dim3 grid, dim3 block,
                                size_t smem, cudaStream_t stream, A... args) {
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
template <typename... P, typename... A>
cudaError_t launchAfter(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                        cudaStream_t stream, A... args) {
  return launchAfterClusters(kernel, 1, grid, block, smem, stream, args...);
}

}  // namespace bfg
