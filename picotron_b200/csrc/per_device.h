// Host state of a launcher that belongs to a device, not to the process: a kernel's attributes hold for the device that was current
// when they were set, so a launcher that serves a second device has to set them there too.
#pragma once
#include <atomic>

namespace pt {

// A positive number per device, found at the first call there: 1 for "set up", or what a query gave. `find` returns zero or an error
// code where it fails; that is handed on and not kept, so that the next call tries again. Several threads may find the same number at once.
class PerDevice {
 public:
  template <class Find>
  int get(int device, Find&& find) {
    if (device < 0 || device >= MAX_DEVICES) return find();
    int v = found_[device].load(std::memory_order_acquire);
    if (v <= 0) {
      v = find();
      if (v > 0) found_[device].store(v, std::memory_order_release);
    }
    return v;
  }

 private:
  static constexpr int MAX_DEVICES = 64;
  std::atomic<int> found_[MAX_DEVICES] = {};
};

}  // namespace pt
