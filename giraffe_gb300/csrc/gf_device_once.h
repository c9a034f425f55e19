// Settings of a device's kernels made once per device (a kernel's shared-memory limit
// holds for the device that was current when it was set, and a process may have contexts
// on several).
#pragma once
#include <atomic>

namespace gf {

class DeviceOnce {
  static constexpr int kDevices = 64;  // a device beyond is set at every call
  std::atomic<bool> done_[kDevices] = {};

 public:
  // set() for `device` unless it has succeeded there before; it may run twice where two
  // threads come first at once.
  template <typename F> bool operator()(int device, F set) {
    const bool kept = device >= 0 && device < kDevices;
    if (kept && done_[device].load(std::memory_order_acquire)) return true;
    const bool ok = set();
    if (kept && ok) done_[device].store(true, std::memory_order_release);
    return ok;
  }
};

}  // namespace gf
