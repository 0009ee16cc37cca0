// What a launcher looked up or set once per device: an attribute of a kernel belongs to the device that was current, and so do
// numbers that depend on it. No CUDA in here, so that it can be tested on its own.
#pragma once
#include <atomic>

class XlPerDevice {  // zero-initialised when static; 0: not known yet
 public:
  static constexpr int DEVICES = 64;
  int get(int device) const { return device >= 0 && device < DEVICES ? value_[device].load(std::memory_order_acquire) : 0; }
  void set(int device, int value) {  // devices beyond the table are looked up each time
    if (device >= 0 && device < DEVICES) value_[device].store(value, std::memory_order_release);
  }

 private:
  std::atomic<int> value_[DEVICES];
};
