// Host helper: a launch that may begin before the kernel in front of it on the stream has ended.  Its blocks take their SMs, set up barriers and
// tensor memory and then wait in pdl_wait() (common.cuh) for that kernel's end and its writes, so that the set-up and the launch itself are hidden behind it.
// Every kernel launched this way calls pdl_wait() in all threads before it reads or writes global memory; it calls pdl_launch_dependents()
// after that, and after its tensor memory is allocated: a block of the next kernel can then never hold what a block of this one still waits for.
#pragma once
#include <cuda_runtime.h>
#include <utility>

namespace nrl {

// early false: behind the end of the kernel in front, where pdl_wait() finds nothing to wait for; cluster 0: as the kernel itself says
template <class... Params, class... Args>
inline void launch_early_if(bool early, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster, Args&&... args) {
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = early ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 0 ? 2 : 1;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}
template <class... Params, class... Args>
inline void launch_dependent_clusters(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster, Args&&... args) {
  launch_early_if(true, kernel, grid, block, smem, stream, cluster, std::forward<Args>(args)...);
}
template <class... Params, class... Args>
inline void launch_dependent(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  launch_early_if(true, kernel, grid, block, smem, stream, 0, std::forward<Args>(args)...);
}

// how many clusters of `cluster` blocks the GPU runs at a time
template <class... Params>
inline int clusters_at_a_time(void (*kernel)(Params...), dim3 block, size_t smem, int cluster) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = cluster;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

}  // namespace nrl
