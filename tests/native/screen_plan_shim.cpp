// Test shim: the size rules of mdsctk_gb300/csrc/screen_plan.h for ctypes.
#include "screen_plan.h"

extern "C" int plan_staged_recheck(int nrows, int k, int same, int fp32) {
  return staged_recheck(nrows, k, same != 0, fp32 != 0);
}
