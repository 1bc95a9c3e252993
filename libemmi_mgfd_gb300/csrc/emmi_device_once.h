// Set-up that a process does once for every device it uses: a kernel's
// attributes and a __device__ variable's address belong to one device, so a
// single flag a process leaves the second device without them.
#pragma once
#include <mutex>

namespace emmi {

constexpr int kOnceDevices = 64;

struct DeviceOnce {
  std::once_flag flag[kOnceDevices];
};

// f() on the first call for device dev (other threads of that device wait for
// it); on every call for a device past the flags
template <typename F>
inline void device_once(DeviceOnce& once, int dev, F&& f) {
  if (dev >= 0 && dev < kOnceDevices) std::call_once(once.flag[dev], f);
  else f();
}

}  // namespace emmi
