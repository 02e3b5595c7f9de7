// A kernel's attributes (its dynamic shared-memory limit) belong to the device
// that is current when they are set, and a process may have contexts on several.
#pragma once
#include <cuda_runtime.h>
#include <mutex>

// Runs `set` once on each device; a failure is not kept, the next call tries again.
class DeviceOnce {
 public:
  template <class F>
  cudaError_t operator()(const F& set) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu_);
    const bool known = dev >= 0 && dev < 64;
    if (known && done_[dev]) return cudaSuccess;
    e = set();
    if (e == cudaSuccess && known) done_[dev] = true;
    return e;
  }

 private:
  std::mutex mu_;
  bool done_[64] = {};
};
