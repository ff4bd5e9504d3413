// overlap_tc.cu -- knn_data_sparse on binary vectors on the 5th generation
// tensor cores: |A & B| of every pair as one matrix product of 0/1 rows.
//
// The reference's distance of two binary vectors is sqrt(|A| + |B| - 2|A & B|)
// bit for bit (knn_sparse.cu). The rows become e4m3 bytes (0 or 1.0), every
// product is 0 or 1 and the FP32 accumulator holds integers below 2^24, so
// the overlaps are exact whatever the order of the sums (compared with counts
// on the CPU up to overlaps of 5 million in rows of 10,000,003 indices, the
// widest that 16 GiB of byte rows hold for the fewest rows that come here:
// tests/test_overlap_range_gpu.py).
//
//  1. k_rows_e4m3    CSR rows -> byte rows [n][K], with the check that they
//                    are binary (every value 1.0, indices strictly ascending).
//  2. k_overlap      squared distances of a panel of fit rows against every
//                    reference row, as 32-bit integers.
//  3. k_select_rows  per fit row the k+1 smallest (value, index) pairs in order,
//                    position 0 dropped as in the reference.
#include <cuda.h>

#include <algorithm>

#include "overlap_tc.cuh"
#include "tc_ptx.cuh"

#define OV_M 128
#define OV_N 256
#define OV_KB 128  // bytes of a row per K-block (one 128-byte swizzle row)
#define OV_STAGES 4
#define OV_A_BYTES (OV_M * OV_KB)
#define OV_B_BYTES (OV_N * OV_KB)
#define OV_STAGE_BYTES (OV_A_BYTES + OV_B_BYTES)
#define OV_THREADS 192  // producer, MMA, 4 epilogue warps
#define OV_GROUP 12     // row tiles of a group: the CTAs at work cover about 12 x 13 tiles

// ---------------------------------------------------------------------------
// 1. byte rows
// ---------------------------------------------------------------------------
// One block per row, 64 KB of the row at a time built in shared memory and
// written in one piece (memory-bound: the CSR entries are read once and the
// bytes written once; no clearing pass, no atomics: 37 M entries into 185 MB
// in 0.16 ms). cnt[row] = entries.
// *bad is set when the rows are not binary.
#define OV_ROWCHUNK 65536
__global__ void __launch_bounds__(256) k_rows_e4m3(const int64_t* __restrict__ off, const int* __restrict__ idx,
                                                   const double* __restrict__ val, int64_t K,
                                                   unsigned char* __restrict__ out, int* __restrict__ cnt,
                                                   int* __restrict__ bad) {
  extern __shared__ __align__(16) unsigned char row[];
  const int r = blockIdx.x;
  const int64_t e0 = off[r], e1 = off[r + 1];
  if (threadIdx.x == 0) cnt[r] = (int)(e1 - e0);
  bool wrong = false;
  int64_t e = e0;  // first entry not yet placed (the same in every thread)
  for (int64_t c0 = 0; c0 < K; c0 += OV_ROWCHUNK) {
    const int m = (int)min((int64_t)OV_ROWCHUNK, K - c0);
    for (int x = threadIdx.x; x < m / 16; x += blockDim.x) reinterpret_cast<uint4*>(row)[x] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    // entries of this chunk: indices ascend, so they are a contiguous range;
    // the loop stops after the first batch that reaches past the chunk
    bool more = e < e1;
    while (more) {
      const int64_t p = e + threadIdx.x;
      bool here = false;
      if (p < e1) {
        const int i = idx[p];
        const bool first = p == e0;
        if (val[p] != 1.0 || i < 0 || i >= K || (!first && i <= idx[p - 1])) wrong = true;
        here = !wrong && i >= c0 && i < c0 + m;
        if (here) row[i - c0] = 0x38;  // e4m3 1.0
      }
      const int placed = __syncthreads_count(here);
      e += placed;
      more = placed == (int)blockDim.x && e < e1;
    }
    __syncthreads();
    for (int x = threadIdx.x; x < m / 16; x += blockDim.x)
      reinterpret_cast<uint4*>(out + (int64_t)r * K + c0)[x] = reinterpret_cast<const uint4*>(row)[x];
    __syncthreads();
  }
  if (wrong || (threadIdx.x == 0 && e < e1)) *bad = 1;  // (entries left over: an index out of order or past K)
}

// ---------------------------------------------------------------------------
// 2. squared distances
// ---------------------------------------------------------------------------
struct OvShared {
  uint64_t full[OV_STAGES], empty[OV_STAGES], tfull[2], tempty[2], done;
  uint32_t tmem_base;
  int abortf;
};
#define OV_SMEM (OV_STAGES * OV_STAGE_BYTES + sizeof(OvShared) + 1024)
static_assert(OV_SMEM <= 227 * 1024, "overlap kernel shared memory");

// Tile -> (row tile, column tile): groups of OV_GROUP row tiles, the row tile
// running fastest, so that the CTAs at work share operand rows in L2.
__device__ __forceinline__ int2 ov_tile(int item, int nrt, int nct) {
  const int per = OV_GROUP * nct, g = item / per, in = item % per;
  const int rows = min(OV_GROUP, nrt - g * OV_GROUP);
  return make_int2(g * OV_GROUP + in % rows, in / rows);
}

// Persistent, one CTA per SM, tile 128 x 256, K-blocks of 128 bytes through a
// 4-stage TMA pipeline, two accumulators of 256 TMEM columns, so that the
// epilogue of one tile runs under the MMAs of the next.
// out[row][nref_ld] = cf[row] + cr[j] - 2 |A & B| for the rows [row0, row0 +
// nrows). Bound by the operand traffic from L2 (48 KB per 588 cycles of MMA).
// 8,000 rows of 23,104 indices: 0.90 ms, 3.3 PFLOP/s of fp8; the popcount
// tiles take 13.3 ms (the popcount pipe's limit).
__global__ void __launch_bounds__(OV_THREADS, 1)
k_overlap(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const int* __restrict__ cf,
          const int* __restrict__ cr, int row0, int nrows, int nref, int nkb, uint32_t idesc, int64_t ld,
          unsigned* __restrict__ out, int* __restrict__ err, int stall) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  unsigned char* stages = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  OvShared* S = reinterpret_cast<OvShared*>(stages + OV_STAGES * OV_STAGE_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nrt = (nrows + OV_M - 1) / OV_M, nct = (nref + OV_N - 1) / OV_N, nitems = nrt * nct;
  if (threadIdx.x == 0) {
    for (int s = 0; s < OV_STAGES; ++s) {
      mbar_init(&S->full[s], 1);
      mbar_init(&S->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&S->tfull[b], 1);
      mbar_init(&S->tempty[b], 4);
    }
    mbar_init(&S->done, 1);
    S->abortf = 0;
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(&S->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = S->tmem_base;
  volatile int* abortf = &S->abortf;
  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmA);
      tma_prefetch_desc(&tmB);
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < nitems && ok; item += gridDim.x) {
        const int2 t = ov_tile(item, nrt, nct);
        for (int kb = 0; kb < nkb; ++kb) {
          if (!mbar_wait(&S->empty[stage], phase ^ 1, abortf)) {
            ok = false;
            break;
          }
          // (stall: an injected fault for the failure-path tests -- the first
          // K-block is not loaded, so the MMA thread's wait for it runs out)
          if (!stall || kb > 0 || item >= (int)gridDim.x) {
            unsigned char* st = stages + stage * OV_STAGE_BYTES;
            mbar_expect_tx(&S->full[stage], OV_STAGE_BYTES);
            tma_load_2d(st, &tmA, &S->full[stage], kb * OV_KB, row0 + t.x * OV_M);
            tma_load_2d(st + OV_A_BYTES, &tmB, &S->full[stage], kb * OV_KB, t.y * OV_N);
          }
          if (++stage == OV_STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (!ok) {
        atomicMax(err, 1);
        *abortf = 1;
        for (int s = 0; s < OV_STAGES; ++s) {  // every issued stage completes or times out
          volatile int dummy = 0;
          mbar_wait(&S->full[s], 0, &dummy, 50000000ull);
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      uint32_t stage = 0, phase = 0, acc = 0;
      bool ok = true;
      const uint32_t sbase = smem_u32(stages);
      for (int item = blockIdx.x; item < nitems && ok; item += gridDim.x, ++acc) {
        const uint32_t b = acc & 1, aph = (acc >> 1) & 1;
        if (!mbar_wait(&S->tempty[b], aph ^ 1, abortf, 1000000000ull, 64)) {
          ok = false;
          break;
        }
        tc_fence_after();
        for (int kb = 0; kb < nkb; ++kb) {
          if (!mbar_wait(&S->full[stage], phase, abortf, 1000000000ull, 64)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t st = sbase + stage * OV_STAGE_BYTES;
#pragma unroll
          for (int ks = 0; ks < OV_KB / 32; ++ks)
            umma_f8(tbase + b * 256, umma_desc_sw128(st + ks * 32), umma_desc_sw128(st + OV_A_BYTES + ks * 32), idesc,
                    (kb | ks) != 0);
          umma_commit(&S->empty[stage]);
          if (++stage == OV_STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) umma_commit(&S->tfull[b]);
      }
      if (!ok) {
        atomicMax(err, 2);
        *abortf = 1;
      }
      umma_commit(&S->done);  // all MMAs of this thread retire before TMEM is freed
      volatile int dummy = 0;
      mbar_wait(&S->done, 0, &dummy, 200000000ull);
    }
    __syncwarp();
  } else {
    const int q = warp & 3;  // TMEM lane quarter of this warp
    uint32_t acc = 0;
    for (int item = blockIdx.x; item < nitems; item += gridDim.x, ++acc) {
      const int2 t = ov_tile(item, nrt, nct);
      const uint32_t b = acc & 1, aph = (acc >> 1) & 1;
      const bool ready = mbar_wait(&S->tfull[b], aph, abortf);
      if (!__all_sync(0xffffffffu, ready)) {
        if (lane == 0) {
          atomicMax(err, 3);
          *abortf = 1;
        }
        break;
      }
      tc_fence_after();
      const int r = t.x * OV_M + q * 32 + lane;  // row of the panel
      const bool rowok = r < nrows;
      const int cnt = rowok ? __ldg(cf + row0 + r) : 0;
      unsigned* o = out + (int64_t)r * ld;
      for (int c = 0; c < OV_N / 32; ++c) {
        uint32_t v[32];
        tmem_ld32(tbase + ((uint32_t)(q * 32) << 16) + b * 256 + 32 * c, v);
        tmem_wait_ld();
        const int j0 = t.y * OV_N + 32 * c;
        // (cr and out are padded to whole column tiles)
        if (rowok) {
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const int4 cc = __ldg(reinterpret_cast<const int4*>(cr + j0 + i));
            uint4 w;
            w.x = (unsigned)(cnt + cc.x - 2 * (int)__uint_as_float(v[i]));
            w.y = (unsigned)(cnt + cc.y - 2 * (int)__uint_as_float(v[i + 1]));
            w.z = (unsigned)(cnt + cc.z - 2 * (int)__uint_as_float(v[i + 2]));
            w.w = (unsigned)(cnt + cc.w - 2 * (int)__uint_as_float(v[i + 3]));
            *reinterpret_cast<uint4*>(o + j0 + i) = w;
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&S->tempty[b]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tbase, 512);
  }
}

// ---------------------------------------------------------------------------
// 3. selection
// ---------------------------------------------------------------------------
// One block per row of the panel: a histogram of the row's integers over its
// own range (OV_BINS bins; a second one inside the bin of the (k+1)-th value
// where the range is wider) gives the (k+1)-th smallest value v and the number
// below it; those are collected in any order, the values equal to v in index
// order as far as they are wanted, and the k+1 pairs sorted. The row is read
// from shared memory when it fits (staged), so from DRAM once. 0.25 ms for
// 8,000 rows of 8,000.
#define OV_BINS 4096
#define OV_SEL_THREADS 256
__global__ void __launch_bounds__(OV_SEL_THREADS)
k_select_rows(const unsigned* __restrict__ d2, int64_t ld, int row0, int nref, int k, int staged,
              double* __restrict__ out_d, int* __restrict__ out_i) {
  constexpr int NW = OV_SEL_THREADS / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned* hist = reinterpret_cast<unsigned*>(smem_raw);                   // [OV_BINS]
  uint64_t* top = reinterpret_cast<uint64_t*>(hist + OV_BINS);              // [next_pow2(k + 1)]
  const int k1 = k + 1, P2 = next_pow2(k1);
  unsigned* row_s = reinterpret_cast<unsigned*>(top + P2);                  // [nref] when staged
  __shared__ unsigned wa[NW], wb[NW];
  __shared__ unsigned s_bin, s_less;
  __shared__ int s_n;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned* g = d2 + (int64_t)blockIdx.x * ld;
  unsigned lo = 0xffffffffu, hi = 0u;
  for (int j = tid; j < nref; j += OV_SEL_THREADS) {
    const unsigned v = g[j];
    if (staged) row_s[j] = v;
    lo = min(lo, v);
    hi = max(hi, v);
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if (lane == 0) {
    wa[warp] = lo;
    wb[warp] = hi;
  }
  __syncthreads();
  for (int w = 0; w < NW; ++w) {
    lo = min(lo, wa[w]);
    hi = max(hi, wb[w]);
  }
  const unsigned* v = staged ? row_s : g;
  // the (k+1)-th value lies in [base, base + width]; `less` values below base
  // (an inclusive width: the panel of a product that timed out holds anything,
  // and the counts have to be right for any values, since they place the writes)
  unsigned base = lo, less = 0, width = hi - lo;
  while (true) {
    int sh = 0;
    while ((width >> sh) >= OV_BINS) ++sh;
    for (int i = tid; i < OV_BINS; i += OV_SEL_THREADS) hist[i] = 0;
    __syncthreads();
    for (int j = tid; j < nref; j += OV_SEL_THREADS) {
      const unsigned x = v[j] - base;
      if (v[j] >= base && x <= width) atomicAdd(&hist[x >> sh], 1u);
    }
    __syncthreads();
    // bins 16 t .. 16 t + 15 by thread t
    unsigned c = 0;
    for (int i = 0; i < OV_BINS / OV_SEL_THREADS; ++i) c += hist[tid * (OV_BINS / OV_SEL_THREADS) + i];
    unsigned inc = c;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) wa[warp] = inc;
    __syncthreads();
    unsigned before = less + inc - c;
    for (int w = 0; w < warp; ++w) before += wa[w];
    if (before < (unsigned)k1 && (unsigned)k1 <= before + c) {
      unsigned acc = before;
      for (int i = 0; i < OV_BINS / OV_SEL_THREADS; ++i) {
        const unsigned h = hist[tid * (OV_BINS / OV_SEL_THREADS) + i];
        if (acc + h >= (unsigned)k1) {
          s_bin = tid * (OV_BINS / OV_SEL_THREADS) + i;
          s_less = acc;
          break;
        }
        acc += h;
      }
    }
    __syncthreads();
    base += s_bin << sh;
    less = s_less;
    if (sh == 0) break;
    width = (1u << sh) - 1;
    __syncthreads();
  }
  const unsigned vk = base;            // the (k+1)-th smallest value
  const int ties = k1 - (int)less;     // how many of the values equal to it are wanted
  if (tid == 0) s_n = 0;
  for (int x = tid; x < P2; x += OV_SEL_THREADS) top[x] = MDS_KEY_INF;
  __syncthreads();
  // warp w takes a contiguous piece, so that its ties are in index order
  const int per = ((nref + NW - 1) / NW + 31) & ~31, j0 = warp * per, j1 = min(nref, j0 + per);
  int mine = 0;
  for (int b = j0; b < j1; b += 32) {
    const int j = b + lane;
    const unsigned x = j < j1 ? v[j] : 0xffffffffu;
    if (j < j1 && x < vk) top[atomicAdd(&s_n, 1)] = ((uint64_t)x << 32) | (unsigned)j;
    mine += __popc(__ballot_sync(0xffffffffu, j < j1 && x == vk));
  }
  if (lane == 0) wb[warp] = mine;
  __syncthreads();
  int run = 0;
  for (int w = 0; w < warp; ++w) run += wb[w];
  for (int b = j0; b < j1 && run < ties; b += 32) {
    const int j = b + lane;
    const bool eq = j < j1 && v[j] == vk;
    const unsigned bal = __ballot_sync(0xffffffffu, eq);
    const int p = run + __popc(bal & ((1u << lane) - 1u));
    if (eq && p < ties) top[less + p] = ((uint64_t)vk << 32) | (unsigned)j;
    run += __popc(bal);
  }
  __syncthreads();
  block_bitonic_sort(top, P2);
  double* od = out_d + (int64_t)(row0 + blockIdx.x) * k;
  int* oi = out_i + (int64_t)(row0 + blockIdx.x) * k;
  for (int x = tid; x < k; x += OV_SEL_THREADS) {
    const uint64_t key = top[x + 1];
    od[x] = sqrt((double)(unsigned)(key >> 32));
    oi[x] = (int)(unsigned)(key & 0xffffffffu);
  }
}

// ---------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------
typedef CUresult (*PFN_encodeTiled_t)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                      const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                      CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static int ov_map(mds_ctx* ctx, CUtensorMap* map, const void* ptr, int rows, int64_t K, int boxrows) {
  static PFN_encodeTiled_t fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !p)
      return mds_fail(ctx, MDS_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
    fn = reinterpret_cast<PFN_encodeTiled_t>(p);
  }
  cuuint64_t gdim[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t gstride[1] = {(cuuint64_t)K};
  cuuint32_t box[2] = {OV_KB, (cuuint32_t)boxrows};
  cuuint32_t estr[2] = {1, 1};
  // rows past the last one read as zero
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), gdim, gstride, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return mds_fail(ctx, MDS_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return MDS_OK;
}

int64_t overlap_width(int dim) { return ((int64_t)std::max(dim, 1) + OV_KB - 1) / OV_KB * OV_KB; }
int overlap_tiles(int nfit, int nref) { return (nfit + OV_M - 1) / OV_M * ((nref + OV_N - 1) / OV_N); }
int overlap_count_pad(int n) { return mds_round_up(n, OV_N); }

int launch_rows_e4m3(mds_ctx* ctx, const int64_t* off, const int* idx, const double* val, int n, int64_t K,
                     unsigned char* out, int* cnt, int* bad) {
  const size_t smem = (size_t)std::min<int64_t>(K, OV_ROWCHUNK);
  static PerDevice attr;
  size_t attr_limit = 0;
  MDS_TRY(mds_allow_dyn_smem(ctx, k_rows_e4m3, &attr, &attr_limit));
  ctx->stats.launches++;
  k_rows_e4m3<<<n, 256, smem, ctx->stream>>>(off, idx, val, K, out, cnt, bad);
  MDS_CUDA(ctx, cudaGetLastError());
  return MDS_OK;
}

int overlap_knn(mds_ctx* ctx, const unsigned char* Bf, const int* cf, int nfit, const unsigned char* Br, const int* cr,
                int nref, int64_t K, int k, double* out_d, int* out_i) {
  cudaStream_t s = ctx->stream;
  CUtensorMap mA, mB;
  MDS_TRY(ov_map(ctx, &mA, Bf, nfit, K, OV_M));
  MDS_TRY(ov_map(ctx, &mB, Br, nref, K, OV_N));
  static PerDevice attr, sel_attr;
  size_t attr_limit = 0, sel_limit = 0;
  MDS_TRY(mds_allow_dyn_smem(ctx, k_overlap, &attr, &attr_limit));
  MDS_TRY(mds_allow_dyn_smem(ctx, k_select_rows, &sel_attr, &sel_limit));
  // panels of rows whose distances take about a gigabyte at most
  const int64_t ld = mds_round_up(nref, OV_N);
  int panel = (int)std::max<int64_t>(OV_M, std::min<int64_t>(mds_round_up(nfit, OV_M),
                                                                   ((int64_t)1 << 28) / ld / OV_M * OV_M));
  DevBuf d2(ctx), err(ctx);
  while (d2.alloc(ctx, sizeof(unsigned) * (size_t)panel * ld) != MDS_OK) {
    if (panel <= OV_M) return MDS_ERR_NOMEM;
    panel = std::max(OV_M, panel / 2 / OV_M * OV_M);  // (a small HBM budget)
  }
  MDS_TRY(err.alloc(ctx, sizeof(int)));
  MDS_CUDA(ctx, cudaMemsetAsync(err.p, 0, sizeof(int), s));
  // the selection stages its row where two blocks still share an SM
  const size_t fixed = sizeof(unsigned) * OV_BINS + sizeof(uint64_t) * next_pow2(k + 1);
  const bool staged = fixed + sizeof(unsigned) * (size_t)nref <= 100 * 1024;
  const size_t sel_smem = fixed + (staged ? sizeof(unsigned) * (size_t)nref : 0);
  if (sel_smem > sel_limit) return mds_fail(ctx, MDS_ERR_UNSUPPORTED, "k=%d too large", k);
  const int stall = (ctx->inject & MDS_INJECT_OVERLAP_STALL) ? 1 : 0;
  ctx->inject &= ~MDS_INJECT_OVERLAP_STALL;
  for (int r0 = 0; r0 < nfit; r0 += panel) {
    const int nr = std::min(panel, nfit - r0);
    const int grid = std::min(overlap_tiles(nr, nref), ctx->num_sms);
    ctx->stats.launches += 2;
    k_overlap<<<grid, OV_THREADS, OV_SMEM, s>>>(mA, mB, cf, cr, r0, nr, nref, (int)(K / OV_KB),
                                                umma_idesc_e4m3(OV_M, OV_N), ld, d2.as<unsigned>(), err.as<int>(), stall);
    k_select_rows<<<nr, OV_SEL_THREADS, sel_smem, s>>>(d2.as<unsigned>(), ld, r0, nref, k, staged ? 1 : 0, out_d,
                                                       out_i);
    MDS_CUDA(ctx, cudaGetLastError());
  }
  int herr = 0;
  MDS_CUDA(ctx, cudaMemcpyAsync(&herr, err.p, sizeof(int), cudaMemcpyDeviceToHost, s));
  MDS_CUDA(ctx, cudaStreamSynchronize(s));
  if (herr) return mds_fail(ctx, MDS_ERR_TIMEOUT, "overlap product: a bounded wait timed out (role %d)", herr);
  return MDS_OK;
}
