// Settings that belong to a kernel on a device (shared-memory size, carve-out, cluster size): `run` calls `set` with the
// launch's device current unless a call of it has succeeded on that device.  The device counts as done only when `set` has
// returned success, so a thread that arrives meanwhile sets the attributes itself (twice is harmless) and never launches
// without them; a `set` that failed is tried again by the next call.
#pragma once
#include <cuda_runtime_api.h>
#include <atomic>

namespace ilb {

struct OncePerDevice {
  static constexpr int kMax = 64;
  std::atomic<bool> done[kMax] = {};
  template <typename Set>
  cudaError_t run(Set set) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMax) return set();
    if (done[dev].load(std::memory_order_acquire)) return cudaSuccess;
    const cudaError_t e = set();
    if (e == cudaSuccess) done[dev].store(true, std::memory_order_release);
    return e;
  }
};

}  // namespace ilb
