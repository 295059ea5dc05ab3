// opt_in.cuh - what a kernel has been granted of dynamic shared memory, per device (host code only, no CUDA headers).
#pragma once

#include <atomic>
#include <mutex>

namespace sgr {

// `set(bytes)` sets the attribute of the kernel on device `dev`; it may also lower it. Callers on several threads ask for
// different sizes of one kernel, so record and attribute change together, under the lock, and only upwards: an attribute
// below the record would refuse every later launch that the record lets through without a call.
class SmemGrant {
 public:
  template <typename Set>
  bool ensure(int dev, int bytes, Set set) {
    if (dev < 0 || dev >= kMaxDevices) return false;
    if (granted_[dev].load(std::memory_order_acquire) >= bytes) return true;
    std::lock_guard<std::mutex> lock(m_);
    if (granted_[dev].load(std::memory_order_relaxed) >= bytes) return true;
    if (!set(bytes)) return false;
    granted_[dev].store(bytes, std::memory_order_release);
    return true;
  }

 private:
  static constexpr int kMaxDevices = 64;
  std::mutex m_;
  std::atomic<int> granted_[kMaxDevices] = {};
};

}  // namespace sgr
