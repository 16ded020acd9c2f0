// Which dynamic shared memory limit a kernel has been raised to, on each device: a
// kernel's attribute belongs to the device that is current when it is set, so a
// process that uses several raises it on every one.
#pragma once
#include <atomic>
#include <cstddef>
#include <mutex>

namespace atb {

struct SmemLimit {
  static constexpr int kDevices = 64;
  static constexpr size_t kDefault = 48 * 1024;  // what a launch may take without asking

  // Calls set() (which raises the limit to `bytes` on device `dev` and returns 0 when
  // done) unless the kernel has that much there already.  Never lowers a limit.
  template <class Set> void raise(int dev, size_t bytes, Set set) {
    if (bytes <= kDefault) return;
    const bool known = dev >= 0 && dev < kDevices;
    if (known && bytes <= raised_[dev].load(std::memory_order_acquire)) return;
    std::lock_guard<std::mutex> lock(m_);
    if (known && bytes <= raised_[dev].load(std::memory_order_relaxed)) return;
    if (set() == 0 && known) raised_[dev].store(bytes, std::memory_order_release);
  }

 private:
  std::atomic<size_t> raised_[kDevices] = {};
  std::mutex m_;
};

}  // namespace atb
