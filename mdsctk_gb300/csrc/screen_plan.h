// screen_plan.h -- the size rules of knn_rms: which path a call takes (host
// only, no CUDA header needed).
#pragma once

#include <algorithm>
#include <cmath>

// Largest k + 1 of the staged recheck: eight candidates to spare of the 128 it
// holds per row, as the block kernel's first chunk.
#define RC3_MAXK1 120

// Whether the staged recheck (four kernels, a warp per row in three of them)
// takes a call's rows rather than the block kernel (a block per row). The
// stages need rows enough to fill the GPU with warps, and a row whose
// candidates exceed their 128 is done twice; against a separate fit set, whose
// thresholds come late, that is every large k. Recheck, stages / block kernel,
// BF16x3 screen unless said:
//   a set against itself   1,000 x 300, k = 50: 73 / 61 us; 1,500 x 300, k = 20: 62 / 66,
//                          k = 80: 108 / 98; 2,000 x 1,000, k = 20: 116 / 143; 3,000 x
//                          300, k = 20: 85 / 113, k = 119: 196 / 203; 20,000 x 300,
//                          k = 100: 1,099 / 1,234
//     FP32 screen          600 x 300, k = 20: 48 / 35; 1,000 x 300, k = 20: 54 / 61,
//                          k = 119: 105 / 90; 1,500 x 300, k = 100: 114 / 119 (whole calls:
//                          600 x 60, k = 5 230 / 217; 700 x 60 252 / 264)
//   600 against 2,000      1,000 atoms, k = 20: 54 / 47; k = 60: 194 / 94; k = 110: 376 / 184
//   2,047 against 20,011   304 atoms, k = 20: 105 / 121; k = 30: 163 / 123; k = 100: 341 / 223
//   10,000 against 20,000  304 atoms, k = 50: 542 / 735; k = 60: 644 / 629; k = 119: 1,689 / 1,079
//   3,000 against 4,000    100 atoms, FP32 screen, k = 60: 159 / 172; k = 119: 234 / 229
//   1,500 against 2,000    60 atoms, FP32 screen, k = 10, whole calls: 455 / 509
inline bool staged_recheck(int nrows, int k, bool same, bool fp32) {
  if (k + 1 > RC3_MAXK1) return false;
  if (same) return nrows >= (fp32 ? (k < 32 ? 700 : k < 64 ? 1000 : 1500) : (k < 32 ? 1500 : 2000));
  if (fp32) return nrows >= (k < 32 ? 1500 : 2000) && k < 64;
  return nrows >= (k < 32 ? 2000 : 5000) && k < 64;
}

// Column segments (at most smax) for nrt row tiles against nct column tiles on
// `slots` blocks at a time: the fewest that leave the last wave nearly full.
// (With the gain asked for in slots instead of relative to what there is, 5 x 3
// tiles on 304 got two segments, the longer one of two tiles: 130 frames of
// 1,000 atoms, k = 20, 543 us a call; three, a tile each: 376.)
inline int choose_segments(int nrt, int slots, int nct, int smax) {
  int best = 1;
  double besteff = 0;
  for (int s = 1; s <= smax && s <= nct; ++s) {
    const double waves = (double)nrt * s / slots, eff = waves / std::ceil(waves);
    if (eff > 1.022 * besteff) {
      besteff = eff;
      best = s;
    }
    if (eff >= 0.95) break;
  }
  return best;
}

// Whether a set against itself skips tiles by pivots in the FP32 screen. Below
// some 80-frame column tiles the pivots cost more than the tiles they save; for
// few neighbours of many atoms a tile is worth more and thresholds are tight
// early. Whole calls, with skipping / without, frames on the device:
//   k = 20  1,000 x 60 309 / 264 us; 1,600 x 60 374 / 341; 1,600 x 200 575 / 616; 1,530 x
//           200 584 / 531; 1,600 x 400 801 / 895; 1,600 x 1,200 1,697 / 2,031; 1,450 x
//           1,200 1,690 / 1,685; 1,740 x 60 384 / 363; 2,000 x 304 (host frames) 767 /
//           1,045
//   k = 10  1,450 x 400 716 / 759; 1,450 x 1,200 1,484 / 1,662
//   k = 60  1,600 x 1,000 1,893 / 1,831; 1,700 x 1,000 1,789 / 2,198
inline bool fp32_skips(int nref, int natoms, int k) {
  const int tiles = (nref + 79) / 80;
  return tiles >= (natoms >= 400 && k < 48 ? (k <= 12 ? 18 : 20) : 22);
}

// Segments of the FP32 screen of a set against itself that skips tiles. Every
// segment starts without thresholds, so its first tiles are computed; for few
// neighbours, whose thresholds then skip most of the rest, one block per SM
// with long segments is best while that leaves two segments or more; for many
// neighbours or few atoms (where the lists, not the multiply-adds, fill the
// time) as without skipping. One segment alone is not taken: a row tile that
// can skip little then holds up the call (4,800 x 400, k = 20 815 / 800 us, k = 30
// 5,367 / 3,524). Calls with these / with choose_segments for two blocks per SM:
//   k = 20  2,200 x 1,200 1,746 / 2,319 us; 1,800 x 200 581 / 701; 2,200 x 60 418 / 428
//   k = 45  2,000 x 1,000 1,706 / 2,041; 2,200 x 200 663 / 662
//   k = 60  2,000 x 1,000 2,246 / 2,134;  k = 80  2,000 x 1,000 3,239 / 2,554
inline int fp32_skip_segments(int nrt, int num_sms, int natoms, int k, int otherwise) {
  if (natoms >= 100 && k < 48 && 2 * nrt <= num_sms) return std::min(8, num_sms / nrt);
  return otherwise;
}
