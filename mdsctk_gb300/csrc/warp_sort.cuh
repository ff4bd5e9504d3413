// warp_sort.cuh -- sorting networks over the registers of one warp.
#pragma once
#include <cstdint>

// Ascending bitonic sort of 32 PER 64-bit keys held PER per lane (element
// e = 32 i + lane in register i): in-register compare-exchanges for the
// strides of 32 and more, shuffles below.
template <int PER>
__device__ __forceinline__ void wsort_u64(uint64_t (&v)[PER], int lane) {
#pragma unroll
  for (int k = 2; k <= 32 * PER; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= 32) {
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          const int p = i ^ (j >> 5);
          if (p > i) {
            const bool up = ((i * 32 + lane) & k) == 0;
            const uint64_t a = v[i], b = v[p];
            if ((a > b) == up) {
              v[i] = b;
              v[p] = a;
            }
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          const int e = i * 32 + lane;
          const uint64_t o = __shfl_xor_sync(0xffffffffu, v[i], j);
          v[i] = (((e & j) == 0) == ((e & k) == 0)) ? min(v[i], o) : max(v[i], o);
        }
      }
    }
  }
}

// Ascending sort of a[0, n), n <= 32 PER, by one warp (a in shared or global
// memory; the warp's writes to it are ordered by the __syncwarp before).
template <int PER>
__device__ __noinline__ void wsort_mem(uint64_t* a, int n, int lane) {
  uint64_t v[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) v[i] = i * 32 + lane < n ? a[i * 32 + lane] : ~0ull;
  wsort_u64<PER>(v, lane);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < PER; ++i)
    if (i * 32 + lane < n) a[i * 32 + lane] = v[i];
  __syncwarp();
}

// The same for any n <= 512, in the registers that n needs. A network over
// shared memory costs a round trip per step: with eight warps at it, 128 keys
// take 9,800 cycles there and 2,000 here.
#define WSORT_MAX 512
__device__ __forceinline__ void warp_sort_keys(uint64_t* a, int n, int lane) {
  __syncwarp();
  if (n <= 32)
    wsort_mem<1>(a, n, lane);
  else if (n <= 64)
    wsort_mem<2>(a, n, lane);
  else if (n <= 128)
    wsort_mem<4>(a, n, lane);
  else if (n <= 256)
    wsort_mem<8>(a, n, lane);
  else
    wsort_mem<16>(a, n, lane);
}

// Element e (any e < 32 PER, per lane) of a warp-distributed array.
template <int PER>
__device__ __forceinline__ uint64_t lane_elem(const uint64_t (&v)[PER], int e) {
  uint64_t r = 0;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const uint64_t y = __shfl_sync(0xffffffffu, v[i], e & 31);
    if (i == (e >> 5)) r = y;
  }
  return r;
}


// Sums of v[i] over the 32 lanes for i < 32, the sum of v[i] returned in lane
// i (v is consumed): each step halves the values a lane holds and exchanges
// the other half with the partner lane, 31 shuffles in all instead of 32 x 5.
__device__ __forceinline__ float warp_sum_transpose32(float (&v)[32], int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool upper = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float send = upper ? v[i] : v[i + o];
      const float keep = upper ? v[i + o] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return v[0];
}
