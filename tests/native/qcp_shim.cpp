// Test shim: the FP32 screen bound of mdsctk_gb300/csrc/qcp.cuh compiled for
// the host and exposed to ctypes for the CPU tests. The approximate square
// root is the correctly rounded one moved by `root_ulp` units in the last
// place, as far as an approximate instruction may be off.
#include <cmath>

#define __device__
#define __forceinline__ inline
#define __restrict__
static int g_root_ulp = 0;
static inline float sqrt_approx(float x) {
  float r = sqrtf(x);
  for (int i = 0; i < g_root_ulp; ++i) r = nextafterf(r, INFINITY);
  for (int i = 0; i > g_root_ulp; --i) r = nextafterf(r, -INFINITY);
  return r;
}
static inline float __fdividef(float a, float b) { return a / b; }
using std::fmaf;

#include "qcp.cuh"

extern "C" void screen_shim(int n, const float* G, const float* r, const float* q, float guard, float thr, int refine,
                            int root_ulp, float* out) {
  g_root_ulp = root_ulp;
  for (int i = 0; i < n; ++i) {
    const float* a = r + 16 * i;
    const float* b = q + 16 * i;
    out[i] = screen_shifted_f32(G + 9 * i, a, b, false, guard * (a[15] + b[15]), thr, refine != 0);
  }
}
