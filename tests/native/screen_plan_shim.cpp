// Test shim: the size rules of mdsctk_gb300/csrc/screen_plan.h for ctypes.
#include "screen_plan.h"

extern "C" int plan_staged_recheck(int nrows, int k, int same, int fp32) {
  return staged_recheck(nrows, k, same != 0, fp32 != 0);
}
extern "C" int plan_choose_segments(int nrt, int slots, int nct, int smax) {
  return choose_segments(nrt, slots, nct, smax);
}
extern "C" int plan_fp32_skips(int nref, int natoms, int k) { return fp32_skips(nref, natoms, k); }
extern "C" int plan_fp32_skip_segments(int nrt, int num_sms, int natoms, int k, int otherwise) {
  return fp32_skip_segments(nrt, num_sms, natoms, k, otherwise);
}
