// A per-device limit of a kernel, raised on demand.
#pragma once

#include <map>
#include <mutex>

namespace sdfgpu {

/// The largest value set so far, per device. cudaFuncSetAttribute applies to the
/// current device only, and a limit belongs to the kernel, not to one of the
/// handles that use it: it only grows, so that a handle with smaller fronts never
/// lowers another's.
class DeviceLimit {
 public:
  /// start: the limit a device has without being set.
  explicit DeviceLimit(int start) : start_(start) {}
  /// Calls set(value), with `device` current, where the device's limit is below
  /// `value`; a call that throws leaves the limit as it was.
  template <typename Set>
  void Raise(int device, int value, Set&& set) {
    const std::lock_guard<std::mutex> lock(mu_);
    int& at = at_.emplace(device, start_).first->second;
    if (value > at) {
      set(value);
      at = value;
    }
  }

 private:
  std::mutex mu_;
  std::map<int, int> at_;
  int start_;
};

}  // namespace sdfgpu
