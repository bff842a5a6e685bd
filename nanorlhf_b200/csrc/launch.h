// Host helper: a launch that may begin before the kernel in front of it on the stream has ended.  Its blocks take their SMs, set up barriers and
// tensor memory and then wait in pdl_wait() (common.cuh) for that kernel's end and its writes, so that the set-up and the launch itself are hidden behind it.
// Every kernel launched this way calls pdl_wait() in all threads before it reads or writes global memory; it calls pdl_launch_dependents()
// after that, and after its tensor memory is allocated: a block of the next kernel can then never hold what a block of this one still waits for.
#pragma once
#include <cuda_runtime.h>
#include <utility>

namespace nrl {

template <class... Params, class... Args>
inline void launch_dependent(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace nrl
