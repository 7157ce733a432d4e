// One-time set-up of a kernel on each device it is launched on.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

namespace lbm {

// Function attributes, a kernel's opt-in to more than 48 KB of shared memory among them, belong to the
// device that was current when they were set; a simulation may live on any device of its process.
class DeviceOnce {
 public:
  // set_up() with the current device, unless it has succeeded there before; its error. Threads that
  // come first together may all run it.
  template <class F>
  cudaError_t operator()(F set_up) {
    int device = 0;
    if (cudaError_t e = cudaGetDevice(&device)) return e;
    const uint64_t bit = device < 64 ? uint64_t(1) << device : 0;  // (further devices: each time)
    if (done_.load(std::memory_order_acquire) & bit) return cudaSuccess;
    if (cudaError_t e = set_up()) return e;
    done_.fetch_or(bit, std::memory_order_release);
    return cudaSuccess;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

}  // namespace lbm
