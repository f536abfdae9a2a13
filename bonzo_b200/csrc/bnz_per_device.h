// bnz_per_device.h -- what a launcher finds out or sets once per kernel and
// device (function attributes and occupancy belong to a device's context).
#pragma once

#include <atomic>

class PerDevice {
 public:
  // make()'s value (positive) for device `dev`, asked for on the first call for
  // that device.  Threads that meet on a first call may each ask.
  template <class F>
  int get(int dev, F make) {
    if (dev < 0 || dev >= MAX) return make();
    int x = v_[dev].load(std::memory_order_acquire);
    if (!x) {
      x = make();
      v_[dev].store(x, std::memory_order_release);
    }
    return x;
  }

 private:
  static constexpr int MAX = 64;
  std::atomic<int> v_[MAX] = {};
};
