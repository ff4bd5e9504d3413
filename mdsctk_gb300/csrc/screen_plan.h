// screen_plan.h -- the size rules of knn_rms: which path a call takes (host
// only, no CUDA header needed).
#pragma once

#include <algorithm>

// Largest k + 1 of the staged recheck: eight candidates to spare of the 128 it
// holds per row, as the block kernel's first chunk.
#define RC3_MAXK1 120

// Whether the staged recheck (four kernels, a warp per row in three of them)
// takes a call's rows rather than the block kernel (a block per row). The
// stages need rows enough to fill the GPU with warps, and a row whose
// candidates exceed their 128 is done twice; against a separate fit set, whose
// thresholds come late, that is every large k. Recheck stage, stages / block
// kernel, 304 to 1,000 atoms:
//   a set against itself   1,000 x 300, k = 50: 73 / 61 us; 2,000 x 1,000, k = 20:
//                          116 / 143; 3,000 x 300, k = 20: 85 / 113, k = 119: 196 / 203;
//                          20,000 x 300, k = 100: 1,099 / 1,234
//   600 against 2,000      k = 20: 54 / 47; k = 60: 194 / 94; k = 110: 376 / 184
//   2,047 against 20,011   k = 20: 105 / 121; k = 30: 163 / 123; k = 100: 341 / 223
//   10,000 against 20,000  k = 50: 542 / 735; k = 60: 644 / 629; k = 119: 1,689 / 1,079
//   3,000 against 4,000    (100 atoms, FP32 screen) k = 60: 159 / 172; k = 119: 234 / 229
inline bool staged_recheck(int nrows, int k, bool same, bool fp32) {
  if (nrows < 2000) return false;
  return k + 1 <= (same ? RC3_MAXK1 : (fp32 || nrows >= 5000) ? 64 : 32);
}
