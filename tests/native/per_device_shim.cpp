// Test shim: PerDevice of mdsctk_gb300/csrc/per_device.h with a stand-in for
// the attribute call, exposed to ctypes for the CPU tests.
#include <atomic>
#include <thread>
#include <vector>

#include "per_device.h"

static PerDevice g_value;
static std::atomic<int> g_calls[256];

// One use of a kernel on `device`: the attribute call is counted, fails with
// `fail`, and settles 1000 + device.
extern "C" int per_device_use(int device, int fail, size_t* value) {
  return g_value.get(device, value, [&](size_t* v) -> int {
    g_calls[device & 255]++;
    if (fail) return fail;
    *v = 1000 + (size_t)device;
    return 0;
  });
}
extern "C" int per_device_calls(int device) { return g_calls[device & 255]; }

// `threads` threads, each using `devices` devices `rounds` times; returns the
// number of uses that gave a wrong value.
extern "C" int per_device_race(int threads, int devices, int rounds) {
  std::atomic<int> wrong{0};
  std::vector<std::thread> ts;
  for (int t = 0; t < threads; ++t)
    ts.emplace_back([&, t] {
      for (int r = 0; r < rounds; ++r) {
        const int d = 16 + (r + t) % devices;
        size_t v = 0;
        if (per_device_use(d, 0, &v) != 0 || v != 1000 + (size_t)d) ++wrong;
      }
    });
  for (auto& t : ts) t.join();
  return wrong;
}
