// per_device.h -- set-up that every CUDA device needs once.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <mutex>

namespace gpb {

// Runs a set-up once on each device, on the thread that first needs it there.
// cudaFuncSetAttribute grants a kernel its shared memory on the current device
// only, so a flag for the whole process would leave a second device without.
// A device counts as set up only after the set-up has succeeded: other threads
// wait for it, and a failure goes to the caller and is tried again.
class PerDevice {
 public:
  static constexpr int kDevices = 64;  // devices remembered; any further one is set up on each call
  // setup() -> cudaError_t
  template <class F>
  cudaError_t once(F&& setup) {
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kDevices) return setup();
    if (done_[dev].load(std::memory_order_acquire)) return cudaSuccess;
    std::lock_guard<std::mutex> lk(mu_);
    if (done_[dev].load(std::memory_order_relaxed)) return cudaSuccess;
    const cudaError_t se = setup();
    if (se == cudaSuccess) done_[dev].store(true, std::memory_order_release);
    return se;
  }

 private:
  std::mutex mu_;
  std::atomic<bool> done_[kDevices] = {};
};

// grants a kernel dynamic shared memory on the current device
template <class K>
cudaError_t grant_smem(K* kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

}  // namespace gpb
