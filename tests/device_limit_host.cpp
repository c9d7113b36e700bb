// Host build of the per-device kernel limits for tests/test_device_limit.py: a
// fake of the call that sets the current device's attribute.
#include "device_limit.h"

#include <stdexcept>

/// Raises to values[i] on devices[i], i < n; set[i] = whether the attribute was
/// set (fail: the call that fails, -1: none).
extern "C" void device_limit_host(int start, int n, const int* devices, const int* values, int fail, int* set) {
  sdfgpu::DeviceLimit limit(start);
  for (int i = 0; i < n; ++i) {
    set[i] = 0;
    try {
      limit.Raise(devices[i], values[i], [&](int) {
        if (i == fail) {
          throw std::runtime_error("refused");
        }
        set[i] = 1;
      });
    } catch (const std::runtime_error&) {
      set[i] = -1;
    }
  }
}
