// per_device.h -- a size that is settled once per device of the process (host
// only, no CUDA header needed).
#pragma once

#include <atomic>
#include <cstddef>

// For function attributes, which belong to the device they are set on: a
// process may hold contexts on several devices, each used from its own thread.
// Zero-initialised (a function's static); safe to use from several threads.
class PerDevice {
 public:
  static constexpr int kDevices = 64;

  // The device's value in *value. Until it is settled, `make` is called on the
  // calling thread with a size_t* to fill (> 0); it returns 0, or an error code
  // that is passed on and leaves the device unsettled. Two threads may both call
  // it, so it has to give the same value each time.
  template <class Make>
  int get(int device, size_t* value, Make make) {
    const bool known = device >= 0 && device < kDevices;
    size_t v = known ? value_[device].load(std::memory_order_acquire) : 0;
    if (v == 0) {
      const int rc = make(&v);
      if (rc != 0) return rc;
      if (known) value_[device].store(v, std::memory_order_release);
    }
    *value = v;
    return 0;
  }

 private:
  std::atomic<size_t> value_[kDevices] = {};
};
