// What CUDA keeps of a kernel per device (its function attributes) is set once for each device that launches it, not once per
// process: a second device of the same process would otherwise refuse a launch with more than 48 KB of dynamic shared memory.
#pragma once
#include <atomic>

namespace sb {

struct PerDeviceOnce {
  std::atomic<unsigned long long> done{0};

  // Runs set() on the first call for `device` and returns its result, 0 on success (later calls: 0). A failure is tried
  // again by the next call; threads that come at the same time may each run it. Devices from 64 on run it every time.
  template <class Set>
  int operator()(int device, Set set) {
    const unsigned long long bit = device >= 0 && device < 64 ? 1ull << device : 0;
    if (done.load(std::memory_order_acquire) & bit) return 0;
    const int rc = set();
    if (rc == 0) done.fetch_or(bit, std::memory_order_release);
    return rc;
  }
};

#ifdef __CUDACC__
// Allows `kern` up to `bytes` of dynamic shared memory on the current device.
template <class Kernel>
static inline int allow_smem(PerDeviceOnce& once, Kernel kern, int bytes, int error) {
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return error;
  return once(device, [&] {
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess ? 0 : error;
  });
}
#endif

}  // namespace sb
