// One value per device of a process, made by the first caller on that device
// (function attributes, occupancy counts and multiprocessor counts are a device's own).
#pragma once

#include <atomic>
#include <mutex>

namespace mfg {

template <typename T, int kDevices = 64>
class PerDevice {
 public:
  // The value of device dev; make(T &) forms it and says whether it could.  A failure is not
  // kept: null now, and the next caller tries again.
  template <typename F>
  const T *get(int dev, F make) {
    if (dev < 0 || dev >= kDevices) return nullptr;
    if (const T *v = ready_[dev].load(std::memory_order_acquire)) return v;
    std::lock_guard<std::mutex> lock(mu_);
    if (const T *v = ready_[dev].load(std::memory_order_relaxed)) return v;
    if (!make(value_[dev])) return nullptr;
    ready_[dev].store(&value_[dev], std::memory_order_release);
    return &value_[dev];
  }

 private:
  std::mutex mu_;
  std::atomic<const T *> ready_[kDevices] = {};
  T value_[kDevices] = {};
};

}  // namespace mfg
