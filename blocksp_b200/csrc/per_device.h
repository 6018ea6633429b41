// per_device.h — what a process sets up once per device (no CUDA).
#pragma once
#include <atomic>
#include <cstdint>

namespace bsp {

// A kernel's shared-memory limit and its occupancy belong to a device, and
// handles of several devices may run on several threads.  has(d): the set-up
// was done on device d; two threads may both find it missing and both do it,
// so it must be repeatable.  Devices past the mask set up on every call.
class PerDevice {
  std::atomic<uint64_t> done_{0};

 public:
  bool has(int device) const {
    return device >= 0 && device < 64 && (done_.load(std::memory_order_acquire) >> device & 1u);
  }
  void set(int device) {
    if (device >= 0 && device < 64) done_.fetch_or(uint64_t(1) << device, std::memory_order_release);
  }
};

}  // namespace bsp
