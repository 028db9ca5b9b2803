// Something to be done once on every device.  A kernel's attributes (dynamic shared memory, cluster
// sizes) hold for the device that is current when they are set, so one flag per process is not
// enough: a context on a second device would launch with the defaults and be refused.
#pragma once

#include <mutex>

namespace gb {

class DeviceOnce {
  static constexpr int DEVICES = 64;
  std::once_flag done_[DEVICES];

 public:
  // f() unless it has run for `device`; contexts may come from several host threads.  After an
  // exception the next call tries again.  Devices beyond the table run it each time.
  template <typename F>
  void operator()(int device, F&& f) {
    if (device >= 0 && device < DEVICES) std::call_once(done_[device], f);
    else f();
  }
};

}  // namespace gb
