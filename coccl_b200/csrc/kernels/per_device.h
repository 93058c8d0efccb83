// What a launch finds out or sets once per device: a process may use several, and function attributes and SM counts are theirs.
#pragma once
#include <atomic>
#include <mutex>

namespace coccl {

template <class T>
class PerDevice {
 public:
  static constexpr int kDevices = 64;

  // *out = the value of device `dev`, filled in by init(value) at its first use. init returns an error code, which is returned;
  // after an error the next use tries again. Devices beyond the table are initialised at every use.
  template <class Init>
  int get(int dev, const T** out, Init init) {
    if (dev < 0 || dev >= kDevices) {
      static thread_local T other;
      other = T{};
      *out = &other;
      return init(other);
    }
    if (!ready_[dev].load(std::memory_order_acquire)) {
      std::lock_guard<std::mutex> lock(mutex_);
      if (!ready_[dev].load(std::memory_order_relaxed)) {
        T v{};
        const int rc = init(v);
        if (rc != 0) return rc;
        value_[dev] = v;
        ready_[dev].store(true, std::memory_order_release);
      }
    }
    *out = &value_[dev];
    return 0;
  }

 private:
  T value_[kDevices] = {};
  std::atomic<bool> ready_[kDevices] = {};
  std::mutex mutex_;
};

}  // namespace coccl
