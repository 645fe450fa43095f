// What a kernel's host side works out once per device. Kernel attributes (the
// dynamic shared memory a launch may ask for, non-portable cluster sizes) and
// figures such as the resident CTAs hold for the device that was current when
// they were set, so a process that uses several devices needs them on each.
// Plain C++.
#pragma once

#include <atomic>
#include <mutex>

namespace alg {

class PerDevice {
 public:
  // The device's value, which f(value) sets (to anything but 0; it starts as 1)
  // on the first call for that device. f returns 0 on success; another result
  // is handed on and not kept, so the next call tries again. Devices past the
  // table's end run f on every call. Safe with several threads.
  template <typename F>
  int get(int device, int& value, F&& f) {
    std::atomic<int>* slot = device >= 0 && device < kDevices ? &values_[device] : nullptr;
    if (slot != nullptr && (value = slot->load(std::memory_order_acquire)) != 0) return 0;
    std::lock_guard<std::mutex> lock(mu_);
    if (slot != nullptr && (value = slot->load(std::memory_order_relaxed)) != 0) return 0;
    value = 1;
    const int error = f(value);
    if (error == 0 && slot != nullptr) slot->store(value, std::memory_order_release);
    return error;
  }

 private:
  static constexpr int kDevices = 64;
  std::atomic<int> values_[kDevices] = {};
  std::mutex mu_;
};

}  // namespace alg
