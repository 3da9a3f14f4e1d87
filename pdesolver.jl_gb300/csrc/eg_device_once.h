// eg_device_once.h -- set-up that a kernel needs once on each device of the
// process.  Launch attributes belong to a device: with one flag for the whole
// process, a launch on a second device that needs more than 48 KB of shared
// memory was refused.
#pragma once
#include <mutex>

struct EgDeviceOnce {
  static constexpr int kDevices = 64;  // above: set() at every call
  std::once_flag done[kDevices];

  template <typename F>
  void operator()(int device, F set) {
    if (device >= 0 && device < kDevices)
      std::call_once(done[device], set);
    else
      set();
  }
};
