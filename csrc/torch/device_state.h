// What the launchers remember from call to call: facts of a device, looked up once.  Backward passes of several devices run
// host code in parallel (the native autograd function holds no interpreter lock), so every such value is atomic, and it is
// kept per device: a kernel's shared-memory limit set on one device is not set on the next.
#pragma once
#include <atomic>
#include <cuda_runtime_api.h>
#include <stdint.h>

namespace fcxhost {

constexpr int MAX_DEVICES = 64;  // devices beyond it are looked up on every call

inline int currentDevice() {
  int dev = 0;
  return cudaGetDevice(&dev) == cudaSuccess ? dev : 0;
}

// SMs of the current device (148 where there is none to ask).
inline int smCount() {
  static std::atomic<int> known[MAX_DEVICES];
  const int dev = currentDevice();
  int n = dev < MAX_DEVICES ? known[dev].load(std::memory_order_relaxed) : 0;
  if (n > 0) return n;
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  if (n <= 0) n = 148;
  if (dev < MAX_DEVICES) known[dev].store(n, std::memory_order_relaxed);
  return n;
}

// Something to be done once per device.  Two threads that come first at the same time both do it.
class OncePerDevice {
  std::atomic<uint64_t> done_{0};

 public:
  template <typename F>
  cudaError_t operator()(F what) {
    const int dev = currentDevice();
    const uint64_t bit = dev < MAX_DEVICES ? 1ull << dev : 0;
    if (done_.load(std::memory_order_acquire) & bit) return cudaSuccess;
    const cudaError_t e = what();
    if (e == cudaSuccess) done_.fetch_or(bit, std::memory_order_release);
    return e;
  }
};

}  // namespace fcxhost
