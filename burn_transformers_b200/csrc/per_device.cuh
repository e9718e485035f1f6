// What a process has settled device by device (plain C++: no CUDA in here).
#pragma once
#include <atomic>
#include <cstddef>
#include <mutex>

namespace bt {

// The dynamic shared memory a kernel has been allowed, one number a device: the attribute belongs to the device that is
// current when it is set, so that one flag a process would leave the kernel without it on every device but the first.
class SharedMemoryAllowance {
 public:
  static constexpr int kDevices = 64;

  // Whether the kernel may use `bytes` on device `dev`; set(bytes) is called where it was not allowed that much before.  The
  // allowance only grows, and one thread at a time changes it: a smaller call cannot take back what a larger one asked for.
  template <typename Set>
  bool allow(int dev, size_t bytes, Set set) {
    if (dev < 0 || dev >= kDevices) return set(bytes);      // (a device that is not tracked: each time anew)
    if (most_[dev].load(std::memory_order_acquire) >= bytes) return true;
    std::lock_guard<std::mutex> lock(mutex_);
    if (most_[dev].load(std::memory_order_relaxed) >= bytes) return true;
    if (!set(bytes)) return false;
    most_[dev].store(bytes, std::memory_order_release);
    return true;
  }

 private:
  std::atomic<size_t> most_[kDevices] = {};
  std::mutex mutex_;
};

}  // namespace bt
