// Function attributes of a launch, set once per device.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace hh {

// Devices on which a launcher has set its kernel's attributes. An attribute
// (shared-memory limit, carveout) belongs to the function on one device, and a
// process may hold contexts on several, used from several threads.
class DeviceOnce {
 public:
  // runs `set` unless it has succeeded on the current device; two threads may
  // both run it, which sets the same values twice
  template <class Set> cudaError_t operator()(const Set& set) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev >= 0 && dev < 64 ? 1ull << dev : 0;  // a device past 63 is set each time
    if (done_.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = set();
    if (e == cudaSuccess) done_.fetch_or(bit, std::memory_order_release);
    return e;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

// The shared-memory limit of `kernel`, raised once per device.
template <class Kernel> inline cudaError_t raise_smem(DeviceOnce& once, Kernel* kernel, size_t bytes) {
  return once([&] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); });
}
// ... and with it the largest carveout: where the planes live in shared memory
// the register budget, not the L1 split, is to set the CTAs per SM.
template <class Kernel> inline cudaError_t raise_smem_carveout(DeviceOnce& once, Kernel* kernel, size_t bytes) {
  return once([&] {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                (int)cudaSharedmemCarveoutMaxShared);
  });
}

}  // namespace hh
