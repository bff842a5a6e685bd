// CUDA keeps a kernel's attributes and occupancy per device; what is remembered of them on the host is kept per device too.
#pragma once
#include <cuda_runtime_api.h>

namespace nrl {

template <class T>
class PerDevice {
 public:
  // the current device's value, T{} at first; of devices past the last that is remembered a new one each time
  T& here() {
    int d = 0;
    if (cudaGetDevice(&d) == cudaSuccess && d >= 0 && d < kDevices) return values_[d];
    static thread_local T other;
    other = T{};
    return other;
  }

 private:
  static constexpr int kDevices = 64;
  T values_[kDevices] = {};
};

// `kernel` may use `bytes` of dynamic shared memory on the current device
template <class Kernel>
inline cudaError_t allow_smem(PerDevice<bool>& done, Kernel kernel, int bytes) {
  bool& here = done.here();
  if (here) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  here = e == cudaSuccess;
  return e;
}

}  // namespace nrl
