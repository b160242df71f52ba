// per_device.cuh - set-up that belongs to a device, not to the process (plain
// C++, so that a host test can compile it).
#pragma once

#include <atomic>

namespace d3 {

// Calls f() (true: it worked) until it has worked once on each device. f may
// be called again, also by threads that come first together: it is idempotent.
class PerDevice {
 public:
  template <class F>
  bool operator()(int device, F f) {
    if (device < 0 || device >= DEVICES) return f();
    if (!done_[device].load(std::memory_order_acquire)) {
      if (!f()) return false;
      done_[device].store(true, std::memory_order_release);
    }
    return true;
  }

 private:
  static constexpr int DEVICES = 128;
  std::atomic<bool> done_[DEVICES] = {};
};

}  // namespace d3
