// Host-side set-up that holds for one device, done once for each. No CUDA in this header.
#pragma once

#include <mutex>

namespace fl {

// A kernel's shared-memory attribute, for instance, applies to the current
// device only, and a launch without it is refused. run(d, set) returns once
// `set` has ended for device d: the first caller runs it, and other threads
// that ask meanwhile wait for it. Devices beyond the flags are set up each time.
class OncePerDevice {
 public:
  static constexpr int kDevices = 64;

  template <typename F>
  void run(int device, F&& set) {
    if (device < 0 || device >= kDevices)
      set();
    else
      std::call_once(done_[device], set);
  }

 private:
  std::once_flag done_[kDevices];
};

}  // namespace fl
