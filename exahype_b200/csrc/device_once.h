// Set-up that a process does once on each device it uses.
//
// A kernel's dynamic shared-memory limit (48 KB unless raised) is a property
// of the kernel on one device, so it is raised on every device that the
// kernel is launched on, by whichever thread comes first there.
#pragma once
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace exa {

class DeviceOnce {
 public:
  // Runs f on the current device unless a run of it has succeeded there. Threads
  // that come at the same time may both run it. Devices past the 64th have no
  // bit: there it runs on every call.
  template <class F>
  cudaError_t operator()(F&& f) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev < 64 ? uint64_t(1) << dev : 0;
    if (done_.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = f();
    if (e == cudaSuccess) done_.fetch_or(bit, std::memory_order_release);
    return e;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

template <class Kernel>
cudaError_t allow_smem(Kernel* kernel, size_t bytes) {
  return cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(bytes));
}

}  // namespace exa
