// sparse.cu -- sparse assembly of the neighbour graph on sm_103a:
// make_sysparse (symmetric, one strict triangle) and make_gesparse (general).
//
// Replaces the Berkeley-DB B-tree of make_sysparse.cpp:184-313 /
// make_gesparse.cpp:184-335 (keys ordered by compare_edge, mdsctk.cpp:567-577;
// a put overwrites; the cursor walk of split_edges, mdsctk.cpp:580-604) with
// a sort: every kept (row, neighbour) entry becomes a 64-bit key (from, to)
// in the B-tree's order plus its sequence number in the reference's insertion
// order. A stable LSD radix sort over the key digits that vary, then "last of
// each run of equal keys" is exactly "the last put wins". The cursor walk
// emits column c = the keys whose from == c, in ascending to; it never moves
// past a key whose from is not the current column, so the columns are the
// keys with 0 <= from < n unless the smallest key has from < 0 (then every
// column is empty).
#include <algorithm>
#include <vector>

#include "mds_common.cuh"

#define RS_THREADS 256
#define RS_ITEMS 16
#define RS_TILE (RS_THREADS * RS_ITEMS)

// signed 32-bit -> order-preserving unsigned
__device__ __forceinline__ uint32_t ord32(int v) { return (uint32_t)v ^ 0x80000000u; }
__device__ __forceinline__ int unord32(uint32_t u) { return (int)(u ^ 0x80000000u); }

// ---------------------------------------------------------------------------
// tiles: every pass over the entries works on tiles of RS_TILE entries, one
// block each, RS_ITEMS per thread. A pass that keeps some of its entries, in
// order, is a count per tile, an exclusive scan of the tiles' counts
// (k_tile_scan) and a second pass that ranks its entries within the tile.
// (One block scanning the entries themselves, 1,024 threads walking a
// contiguous piece each, took 12.3 ms for the 12.8 M slots of a 100,000 x 64
// graph: uncoalesced, on one SM.)
// ---------------------------------------------------------------------------
// Sum over the block's threads (every thread gets it).
__device__ __forceinline__ int block_sum_int(int v, int* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  int t = 0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
  return t;
}
// Exclusive prefix of v over the block's threads in thread order.
__device__ __forceinline__ int block_prefix_int(int v, int* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = v;
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  __syncthreads();
  if (lane == 31) red[warp] = inc;
  __syncthreads();
  int before = 0;
  for (int w = 0; w < warp; ++w) before += red[w];
  return before + inc - v;
}

// cnt[0..n) -> its exclusive scan in off[0..n), the total in *total. One block
// of 1,024 threads; n is a number of tiles (1,600 at 6.4 M entries).
__global__ void __launch_bounds__(1024) k_tile_scan(const int* __restrict__ cnt, int n, int64_t* __restrict__ off,
                                                    int64_t* __restrict__ total) {
  __shared__ long long part[32];
  __shared__ long long s_run;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_run = 0;
  __syncthreads();
  for (int b = 0; b < n; b += 1024) {
    const int i = b + threadIdx.x;
    const long long v = (i < n) ? cnt[i] : 0;
    long long inc = v;
    for (int o = 1; o < 32; o <<= 1) {
      const long long t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) part[warp] = inc;
    __syncthreads();
    long long before = s_run;
    for (int w = 0; w < warp; ++w) before += part[w];
    if (i < n) off[i] = before + inc - v;
    __syncthreads();
    if (threadIdx.x == 1023) s_run = before + inc;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = s_run;
}

// ---------------------------------------------------------------------------
// key generation, in the reference's insertion order
// ---------------------------------------------------------------------------
// sysparse: for r, x < k: j = idx[r*maxk+x]; r<j -> (r,j); j<r -> (j,r).
// gesparse: (r, j) always; with `sym` (mode 2), also (j, r), inserted only
// where that key is absent when it is put (make_gesparse.cpp:259-271).
// Slot e*2 holds the direct put of entry e = r*k + x, slot e*2+1 the
// transposed one; seq = slot, so seq order is the order of the puts.
__device__ __forceinline__ unsigned long long edge_key(int from, int to) {
  return ((unsigned long long)ord32(from) << 32) | ord32(to);
}
// Entry e = r * k + x -> r (a 32-bit division where it can be one).
__device__ __forceinline__ int64_t entry_row(int64_t e, int k) {
  return (e >> 32) ? e / k : (int64_t)((uint32_t)e / (uint32_t)k);
}
// The keys of entry e: 0, 1 or 2 of them.
__device__ __forceinline__ int edge_keys(const int* __restrict__ idx, int64_t e, int maxk, int k, int mode,
                                         unsigned long long& direct, unsigned long long& transposed) {
  const int r = (int)entry_row(e, k), x = (int)(e - (int64_t)r * k);
  const int j = idx[(int64_t)r * maxk + x];
  if (mode == 0) {
    direct = edge_key(min(r, j), max(r, j));
    return j != r ? 1 : 0;
  }
  direct = edge_key(r, j);
  transposed = edge_key(j, r);
  return mode == 2 ? 2 : 1;
}

// Puts per tile of entries, and over all puts the AND (bits[0], preset to all
// ones) and the OR (bits[1], preset to 0) of their keys: the bits that vary,
// for the sort, and whether a key's `from` is negative.
__global__ void __launch_bounds__(RS_THREADS) k_edge_count(const int* __restrict__ idx, int64_t nent, int maxk, int k,
                                                           int mode, int* __restrict__ cnt,
                                                           unsigned long long* __restrict__ bits) {
  __shared__ int red[RS_THREADS / 32];
  const int64_t base = (int64_t)blockIdx.x * RS_TILE;
  int n = 0;
  unsigned long long ka = ~0ull, ko = 0ull;
  for (int i = 0; i < RS_ITEMS; ++i) {
    const int64_t e = base + (int64_t)i * RS_THREADS + threadIdx.x;
    if (e >= nent) break;
    unsigned long long d, t;
    const int m = edge_keys(idx, e, maxk, k, mode, d, t);
    n += m;
    if (m > 0) {
      ka &= d;
      ko |= d;
    }
    if (m > 1) {
      ka &= t;
      ko |= t;
    }
  }
  const int total = block_sum_int(n, red);
  if (threadIdx.x == 0) cnt[blockIdx.x] = total;
  const unsigned a0 = __reduce_and_sync(0xffffffffu, (unsigned)ka), a1 = __reduce_and_sync(0xffffffffu, (unsigned)(ka >> 32));
  const unsigned o0 = __reduce_or_sync(0xffffffffu, (unsigned)ko), o1 = __reduce_or_sync(0xffffffffu, (unsigned)(ko >> 32));
  if ((threadIdx.x & 31) == 0) {
    atomicAnd(bits, ((unsigned long long)a1 << 32) | a0);
    atomicOr(bits + 1, ((unsigned long long)o1 << 32) | o0);
  }
}

// Warp w of a tile takes its entries [512 w, 512 w + 512), 32 at a time, so
// that one ballot ranks 32 entries and the block meets once.
__global__ void __launch_bounds__(RS_THREADS) k_edge_write(const int* __restrict__ idx, int64_t nent, int maxk, int k,
                                                           int mode, const int64_t* __restrict__ off,
                                                           unsigned long long* __restrict__ keys,
                                                           int64_t* __restrict__ seq) {
  __shared__ int red[RS_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t base = (int64_t)blockIdx.x * RS_TILE + warp * (32 * RS_ITEMS) + lane;
  unsigned bal[RS_ITEMS];
  int n = 0;
#pragma unroll
  for (int i = 0; i < RS_ITEMS; ++i) {
    const int64_t e = base + 32 * i;
    unsigned long long d, t;
    bal[i] = __ballot_sync(0xffffffffu, e < nent && edge_keys(idx, e, maxk, k, mode, d, t) > 0);
    n += __popc(bal[i]);
  }
  const int per = mode == 2 ? 2 : 1;  // puts of an entry that has any
  if (lane == 0) red[warp] = n * per;
  __syncthreads();
  int64_t run = off[blockIdx.x];
  for (int w = 0; w < warp; ++w) run += red[w];
#pragma unroll
  for (int i = 0; i < RS_ITEMS; ++i) {
    if ((bal[i] >> lane) & 1u) {
      const int64_t e = base + 32 * i;
      unsigned long long d, t;
      edge_keys(idx, e, maxk, k, mode, d, t);
      const int64_t p = run + per * __popc(bal[i] & ((1u << lane) - 1u));
      keys[p] = d;
      seq[p] = 2 * e;
      if (per == 2) {
        keys[p + 1] = t;
        seq[p + 1] = 2 * e + 1;
      }
    }
    run += per * __popc(bal[i]);
  }
}

// ---------------------------------------------------------------------------
// LSD radix sort (8-bit digits) of (uint64 key, int64 value), stable
// ---------------------------------------------------------------------------
// A digit is up to 8 of the key's varying bits, taken from at most two runs
// of them (a graph's keys vary in the low bits of `from` and of `to` only, so
// 2 x 17 bits are five digits instead of six).
struct RsDigit {
  int s0, n0;  // bits [s0, s0 + n0) ...
  int s1, n1;  // ... and above them bits [s1, s1 + n1)
};
__device__ __forceinline__ int rs_digit(unsigned long long key, RsDigit g) {
  return (int)((key >> g.s0) & ((1u << g.n0) - 1u)) | ((int)((key >> g.s1) & ((1u << g.n1) - 1u)) << g.n0);
}

// hist[digit][block]
__global__ void __launch_bounds__(RS_THREADS) k_rs_hist(const unsigned long long* __restrict__ keys, int64_t n,
                                                        RsDigit g, unsigned* __restrict__ hist, int nblocks) {
  __shared__ unsigned h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * RS_TILE;
#pragma unroll 4
  for (int i = 0; i < RS_ITEMS; ++i) {
    const int64_t e = base + (int64_t)i * RS_THREADS + threadIdx.x;
    if (e < n) atomicAdd(&h[rs_digit(keys[e], g)], 1u);
  }
  __syncthreads();
  hist[(int64_t)threadIdx.x * nblocks + blockIdx.x] = h[threadIdx.x];
}

// One block per digit: the exclusive scan of its blocks' counts in place, the
// digit's total in tot[digit]. (One block scanning all 256 x blocks entries
// took 330 us of each pass at 6.4 M keys; this takes 7 us.)
__global__ void __launch_bounds__(RS_THREADS) k_rs_scan(unsigned* __restrict__ hist, int nblocks,
                                                        unsigned* __restrict__ tot) {
  __shared__ int red[RS_THREADS / 32];
  unsigned* h = hist + (int64_t)blockIdx.x * nblocks;
  unsigned run = 0;
  for (int b = 0; b < nblocks; b += RS_THREADS) {
    const int i = b + threadIdx.x;
    const int v = (i < nblocks) ? (int)h[i] : 0;
    const int before = block_prefix_int(v, red);
    if (i < nblocks) h[i] = run + (unsigned)before;
    run += (unsigned)block_sum_int(v, red);
  }
  if (threadIdx.x == 0) tot[blockIdx.x] = run;
}

// One tile of keys to its place in the pass's output. Warp w ranks the keys
// [512 w, 512 w + 512) of the tile in order, 32 at a time, with its own
// digit counters (lanes of equal digit found by __match_any_sync;
// eight ballots took the same time), so no
// block barrier falls between them; the tile is then ordered by digit in
// shared memory and written out, so that keys of one digit leave as one run.
// (Ranking 256 keys at a time with block barriers and a cleared counter
// table each time: 103 us a pass at 6.4 M keys; now 94 us, 2.2 TB/s, held by
// the shared-memory round trips of the ranking and the short runs.)
__global__ void __launch_bounds__(RS_THREADS)
k_rs_scatter(const unsigned long long* __restrict__ kin, const int64_t* __restrict__ vin, int64_t n, RsDigit g,
             const unsigned* __restrict__ hist, const unsigned* __restrict__ tot, int nblocks,
             unsigned long long* __restrict__ kout, int64_t* __restrict__ vout) {
  constexpr int NW = RS_THREADS / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned long long* sk = reinterpret_cast<unsigned long long*>(smem_raw);  // [RS_TILE]
  int64_t* sv = reinterpret_cast<int64_t*>(sk + RS_TILE);                    // [RS_TILE]
  __shared__ unsigned wcnt[NW][256];
  __shared__ unsigned lofs[256];   // the digit's first place in the ordered tile
  __shared__ unsigned gofs[256];   // its first place in the output, less lofs
  __shared__ int red[NW];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < NW * 256; i += RS_THREADS) (&wcnt[0][0])[i] = 0;
  // exclusive scan of the digits' totals (thread d holds digit d)
  const unsigned digit_base = (unsigned)block_prefix_int((int)tot[threadIdx.x], red);
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * RS_TILE + warp * (32 * RS_ITEMS) + lane;
  unsigned long long key[RS_ITEMS];
  unsigned rank[RS_ITEMS];
#pragma unroll
  for (int i = 0; i < RS_ITEMS; ++i) key[i] = (base + 32 * i < n) ? kin[base + 32 * i] : 0ull;
#pragma unroll
  for (int i = 0; i < RS_ITEMS; ++i) {
    const bool valid = base + 32 * i < n;
    const int d = rs_digit(key[i], g);
    const unsigned peers = __match_any_sync(0xffffffffu, valid ? d : 256 + lane);
    const unsigned below = peers & ((1u << lane) - 1u);
    unsigned first = 0;
    if (valid && below == 0) {  // the lowest lane of the digit
      first = wcnt[warp][d];
      wcnt[warp][d] = first + __popc(peers);
    }
    first = __shfl_sync(0xffffffffu, first, __ffs(peers) - 1);
    rank[i] = first + __popc(below);
    __syncwarp();
  }
  __syncthreads();
  // digit d = threadIdx.x: its count per warp -> prefix over the warps
  unsigned c = 0;
#pragma unroll
  for (int w = 0; w < NW; ++w) {
    const unsigned t = wcnt[w][threadIdx.x];
    wcnt[w][threadIdx.x] = c;
    c += t;
  }
  const unsigned lo = (unsigned)block_prefix_int((int)c, red);
  lofs[threadIdx.x] = lo;
  gofs[threadIdx.x] = digit_base + hist[(int64_t)threadIdx.x * nblocks + blockIdx.x] - lo;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < RS_ITEMS; ++i)
    if (base + 32 * i < n) {
      const int d = rs_digit(key[i], g);
      const unsigned p = lofs[d] + wcnt[warp][d] + rank[i];
      sk[p] = key[i];
      sv[p] = vin[base + 32 * i];
    }
  __syncthreads();
  const int m = (int)min((int64_t)RS_TILE, n - (int64_t)blockIdx.x * RS_TILE);
  for (int p = threadIdx.x; p < m; p += RS_THREADS) {
    const unsigned long long k = sk[p];
    const int64_t q = (int64_t)(unsigned)(gofs[rs_digit(k, g)] + (unsigned)p);
    kout[q] = k;
    vout[q] = sv[p];
  }
}

// Stable sort of n (key, value) pairs by the key bits in `mask`; ping-pongs
// between (k0,v0) and (k1,v1); returns the index (0/1) holding the result.
// (n < 2^32: the places are 32-bit, modulo 2^32 where lofs is taken off.)
int radix_sort(mds_ctx* ctx, unsigned long long* k0, int64_t* v0, unsigned long long* k1, int64_t* v1,
               int64_t n, unsigned long long mask, int* which) {
  cudaStream_t s = ctx->stream;
  *which = 0;
  if (n <= 1) return MDS_OK;
  if (n >= (int64_t)1 << 32) return mds_fail(ctx, MDS_ERR_UNSUPPORTED, "sort of %lld entries", (long long)n);
  const int nblocks = (int)((n + RS_TILE - 1) / RS_TILE);
  DevBuf hist(ctx);
  MDS_TRY(hist.alloc(ctx, sizeof(unsigned) * 256 * ((size_t)nblocks + 1)));
  unsigned* tot = hist.as<unsigned>() + (size_t)256 * nblocks;
  const size_t smem = (size_t)RS_TILE * (sizeof(unsigned long long) + sizeof(int64_t));
  static PerDevice attr;
  size_t attr_limit = 0;
  MDS_TRY(mds_allow_dyn_smem(ctx, k_rs_scatter, &attr, &attr_limit));
  unsigned long long* ka = k0;
  int64_t* va = v0;
  unsigned long long* kb = k1;
  int64_t* vb = v1;
  for (int bit = 0; bit < 64;) {
    // the next digit: a run of varying bits, and where that is short of 8
    // the start of the next run
    while (bit < 64 && !((mask >> bit) & 1ull)) ++bit;
    if (bit == 64) break;
    RsDigit g{bit, 0, 0, 0};
    while (bit < 64 && g.n0 < 8 && ((mask >> bit) & 1ull)) ++bit, ++g.n0;
    if (g.n0 < 8) {
      int b2 = bit;
      while (b2 < 64 && !((mask >> b2) & 1ull)) ++b2;
      if (b2 < 64) {
        g.s1 = b2;
        while (b2 < 64 && g.n0 + g.n1 < 8 && ((mask >> b2) & 1ull)) ++b2, ++g.n1;
        bit = b2;
      }
    }
    ctx->stats.launches += 3;
    k_rs_hist<<<nblocks, RS_THREADS, 0, s>>>(ka, n, g, hist.as<unsigned>(), nblocks);
    k_rs_scan<<<256, RS_THREADS, 0, s>>>(hist.as<unsigned>(), nblocks, tot);
    k_rs_scatter<<<nblocks, RS_THREADS, smem, s>>>(ka, va, n, g, hist.as<unsigned>(), tot, nblocks, kb, vb);
    MDS_CUDA(ctx, cudaGetLastError());
    std::swap(ka, kb);
    std::swap(va, vb);
    *which ^= 1;
  }
  return MDS_OK;
}

// ---------------------------------------------------------------------------
// resolution of the puts and CSC emission
// ---------------------------------------------------------------------------
// Keys sorted by (key, seq). Symmetric / plain general mode: keep the last
// entry of each run of equal keys (last put wins). General with `sym`:
// a transposed put (odd seq) only inserts when the key is absent, so in a
// run the winner is the last direct put if any, else the first transposed
// put; later transposed puts never overwrite. Keys whose `from` is no column
// are dropped.
__device__ __forceinline__ bool edge_kept(const unsigned long long* __restrict__ keys, const int64_t* __restrict__ seq,
                                          int64_t e, int64_t n, int mode, int ncol) {
  const unsigned long long key = keys[e];
  const int from = unord32((uint32_t)(key >> 32));
  if (from < 0 || from >= ncol) return false;
  if (mode != 2) return e + 1 == n || keys[e + 1] != key;
  if ((seq[e] & 1) == 0) {
    // a direct put wins over every put before it: kept if no direct put of
    // the key comes later
    for (int64_t f = e + 1; f < n && keys[f] == key; ++f)
      if ((seq[f] & 1) == 0) return false;
    return true;
  }
  // a transposed put is kept if it is the key's first put and no direct put
  // replaces it later
  if (e > 0 && keys[e - 1] == key) return false;
  for (int64_t f = e + 1; f < n && keys[f] == key; ++f)
    if ((seq[f] & 1) == 0) return false;
  return true;
}

// kept entries per tile
__global__ void __launch_bounds__(RS_THREADS) k_kept_count(const unsigned long long* __restrict__ keys,
                                                           const int64_t* __restrict__ seq, int64_t n, int mode,
                                                           int ncol, int* __restrict__ cnt) {
  __shared__ int red[RS_THREADS / 32];
  const int64_t base = (int64_t)blockIdx.x * RS_TILE;
  int m = 0;
#pragma unroll 4
  for (int i = 0; i < RS_ITEMS; ++i) {
    const int64_t e = base + (int64_t)i * RS_THREADS + threadIdx.x;
    if (e < n && edge_kept(keys, seq, e, n, mode, ncol)) ++m;
  }
  const int total = block_sum_int(m, red);
  if (threadIdx.x == 0) cnt[blockIdx.x] = total;
}

// the kept entries, in order, as (from, to, value); warps as in k_edge_write
__global__ void __launch_bounds__(RS_THREADS) k_emit(const unsigned long long* __restrict__ keys,
                                                     const int64_t* __restrict__ seq, int64_t n, int mode, int ncol,
                                                     const int64_t* __restrict__ off, const double* __restrict__ dist,
                                                     int maxk, int k, int* __restrict__ colof, int* __restrict__ irow,
                                                     double* __restrict__ val) {
  __shared__ int red[RS_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t base = (int64_t)blockIdx.x * RS_TILE + warp * (32 * RS_ITEMS) + lane;
  unsigned bal[RS_ITEMS];
  int c = 0;
#pragma unroll
  for (int i = 0; i < RS_ITEMS; ++i) {
    const int64_t e = base + 32 * i;
    bal[i] = __ballot_sync(0xffffffffu, e < n && edge_kept(keys, seq, e, n, mode, ncol));
    c += __popc(bal[i]);
  }
  if (lane == 0) red[warp] = c;
  __syncthreads();
  int64_t run = off[blockIdx.x];
  for (int w = 0; w < warp; ++w) run += red[w];
#pragma unroll
  for (int i = 0; i < RS_ITEMS; ++i) {
    if ((bal[i] >> lane) & 1u) {
      const int64_t e = base + 32 * i, p = run + __popc(bal[i] & ((1u << lane) - 1u));
      const unsigned long long key = keys[e];
      const int64_t t = seq[e] >> 1, r = entry_row(t, k);  // t = r * k + x
      colof[p] = unord32((uint32_t)(key >> 32));
      irow[p] = unord32((uint32_t)key);
      val[p] = dist[r * maxk + (t - r * k)];
    }
    run += __popc(bal[i]);
  }
}

__global__ void k_pcol(const int* __restrict__ colof, int64_t nnz, int ncol, int* __restrict__ pcol) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c > ncol) return;
  // lower_bound of c in colof (ascending)
  int64_t lo = 0, hi = nnz;
  while (lo < hi) {
    int64_t mid = (lo + hi) / 2;
    if (colof[mid] < c) lo = mid + 1; else hi = mid;
  }
  pcol[c] = (int)lo;
}

// mode 0: sysparse; 1: gesparse; 2: gesparse with -s
static int assemble(mds_ctx* ctx, const double* ddist, const int* didx, int n, int maxk, int k, int mode,
                    int* dpcol, int* dirow, double* dval, int64_t cap, int64_t* nnz_out) {
  cudaStream_t s = ctx->stream;
  const int64_t nent = (int64_t)n * k;                  // list entries
  const int64_t nput = nent * (mode == 2 ? 2 : 1);      // keys at most
  const int64_t tiles = (nput + RS_TILE - 1) / RS_TILE;
  DevBuf k0(ctx), v0(ctx), k1(ctx), v1(ctx), cnt(ctx), off(ctx), scal(ctx), colof(ctx);
  MDS_TRY(k0.alloc(ctx, sizeof(unsigned long long) * std::max<int64_t>(nput, 1)));
  MDS_TRY(v0.alloc(ctx, sizeof(int64_t) * std::max<int64_t>(nput, 1)));
  MDS_TRY(k1.alloc(ctx, sizeof(unsigned long long) * std::max<int64_t>(nput, 1)));
  MDS_TRY(v1.alloc(ctx, sizeof(int64_t) * std::max<int64_t>(nput, 1)));
  MDS_TRY(cnt.alloc(ctx, sizeof(int) * std::max<int64_t>(tiles, 1)));
  MDS_TRY(off.alloc(ctx, sizeof(int64_t) * std::max<int64_t>(tiles, 1)));
  MDS_TRY(scal.alloc(ctx, 3 * sizeof(int64_t)));  // the keys' AND and OR, a total
  unsigned long long* bits = scal.as<unsigned long long>();
  int64_t* total = scal.as<int64_t>() + 2;
  unsigned long long hs[3] = {0, 0, 0};
  if (nent > 0) {
    const int g = (int)((nent + RS_TILE - 1) / RS_TILE);
    MDS_CUDA(ctx, cudaMemsetAsync(bits, 0xff, sizeof(unsigned long long), s));
    MDS_CUDA(ctx, cudaMemsetAsync(bits + 1, 0, sizeof(unsigned long long), s));
    ctx->stats.launches += 3;
    k_edge_count<<<g, RS_THREADS, 0, s>>>(didx, nent, maxk, k, mode, cnt.as<int>(), bits);
    k_tile_scan<<<1, 1024, 0, s>>>(cnt.as<int>(), g, off.as<int64_t>(), total);
    k_edge_write<<<g, RS_THREADS, 0, s>>>(didx, nent, maxk, k, mode, off.as<int64_t>(), k0.as<unsigned long long>(),
                                          v0.as<int64_t>());
    MDS_CUDA(ctx, cudaGetLastError());
    MDS_CUDA(ctx, cudaMemcpyAsync(hs, scal.p, sizeof(hs), cudaMemcpyDeviceToHost, s));
    MDS_CUDA(ctx, cudaStreamSynchronize(s));
  }
  const int64_t m = (int64_t)hs[2];
  // the cursor walk: nothing is emitted if the smallest key's from < 0, that
  // is if some key has the order bit of `from` clear
  const bool blocked = m > 0 && !(hs[0] >> 63);
  int64_t nnz = 0;
  unsigned long long* keys = k0.as<unsigned long long>();
  int64_t* seq = v0.as<int64_t>();
  const int gm = (int)((m + RS_TILE - 1) / RS_TILE);
  if (m > 0 && !blocked) {
    int which = 0;
    MDS_TRY(radix_sort(ctx, k0.as<unsigned long long>(), v0.as<int64_t>(), k1.as<unsigned long long>(),
                       v1.as<int64_t>(), m, hs[1] & ~hs[0], &which));
    if (which) {
      keys = k1.as<unsigned long long>();
      seq = v1.as<int64_t>();
    }
    ctx->stats.launches += 2;
    k_kept_count<<<gm, RS_THREADS, 0, s>>>(keys, seq, m, mode, n, cnt.as<int>());
    k_tile_scan<<<1, 1024, 0, s>>>(cnt.as<int>(), gm, off.as<int64_t>(), total);
    MDS_CUDA(ctx, cudaGetLastError());
    MDS_CUDA(ctx, cudaMemcpyAsync(&nnz, total, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    MDS_CUDA(ctx, cudaStreamSynchronize(s));
  }
  if (nnz > cap) return mds_fail(ctx, MDS_ERR_ARG, "output capacity %lld < nnz %lld", (long long)cap, (long long)nnz);
  MDS_TRY(colof.alloc(ctx, sizeof(int) * std::max<int64_t>(nnz, 1)));
  if (nnz > 0) {
    ctx->stats.launches++;
    k_emit<<<gm, RS_THREADS, 0, s>>>(keys, seq, m, mode, n, off.as<int64_t>(), ddist, maxk, k, colof.as<int>(), dirow,
                                     dval);
  }
  ctx->stats.launches++;
  k_pcol<<<(n + 1 + 255) / 256, 256, 0, s>>>(colof.as<int>(), nnz, n, dpcol);
  MDS_CUDA(ctx, cudaGetLastError());
  MDS_CUDA(ctx, cudaStreamSynchronize(s));
  *nnz_out = nnz;
  return MDS_OK;
}

static int assemble_api(mds_ctx* ctx, const double* dist, const int32_t* idx, int n_rows, int maxk, int k,
                        unsigned flags, int mode, int32_t* pcol, int32_t* irow, double* val, int64_t cap,
                        int64_t* nnz) {
  if (!ctx) return MDS_ERR_ARG;
  ctx->stats = mds_knn_stats{};
  if (!dist || !idx || !pcol || !irow || !val || !nnz) return mds_fail(ctx, MDS_ERR_ARG, "null argument");
  if (n_rows < 0 || maxk < 1 || k < 0 || k > maxk)
    return mds_fail(ctx, MDS_ERR_ARG, "invalid sizes n_rows=%d maxk=%d k=%d (need k <= maxk)", n_rows, maxk, k);
  if ((int64_t)n_rows * k * 2 >= (1ll << 40)) return mds_fail(ctx, MDS_ERR_UNSUPPORTED, "too many entries");
  cudaSetDevice(ctx->device);
  cudaStream_t s = ctx->stream;
  const bool dev = (flags & MDS_DEVICE_IO) != 0;
  DevBuf dd(ctx), di(ctx), dp(ctx), dr(ctx), dv(ctx);
  const double* pdist = dist;
  const int* pidx = idx;
  int* ppcol = pcol;
  int* pirow = irow;
  double* pval = val;
  const size_t ent = (size_t)n_rows * maxk;
  if (!dev) {
    MDS_TRY(dd.alloc(ctx, sizeof(double) * std::max<size_t>(ent, 1)));
    MDS_TRY(di.alloc(ctx, sizeof(int) * std::max<size_t>(ent, 1)));
    if (ent) {
      MDS_CUDA(ctx, cudaMemcpyAsync(dd.p, dist, sizeof(double) * ent, cudaMemcpyHostToDevice, s));
      MDS_CUDA(ctx, cudaMemcpyAsync(di.p, idx, sizeof(int) * ent, cudaMemcpyHostToDevice, s));
    }
    MDS_TRY(dp.alloc(ctx, sizeof(int) * (n_rows + 1)));
    MDS_TRY(dr.alloc(ctx, sizeof(int) * std::max<int64_t>(cap, 1)));
    MDS_TRY(dv.alloc(ctx, sizeof(double) * std::max<int64_t>(cap, 1)));
    pdist = dd.as<double>();
    pidx = di.as<int>();
    ppcol = dp.as<int>();
    pirow = dr.as<int>();
    pval = dv.as<double>();
  }
  int64_t m = 0;
  MDS_TRY(assemble(ctx, pdist, pidx, n_rows, maxk, k, mode, ppcol, pirow, pval, cap, &m));
  if (!dev) {
    MDS_CUDA(ctx, cudaMemcpyAsync(pcol, ppcol, sizeof(int) * (n_rows + 1), cudaMemcpyDeviceToHost, s));
    if (m) {
      MDS_CUDA(ctx, cudaMemcpyAsync(irow, pirow, sizeof(int) * m, cudaMemcpyDeviceToHost, s));
      MDS_CUDA(ctx, cudaMemcpyAsync(val, pval, sizeof(double) * m, cudaMemcpyDeviceToHost, s));
    }
    MDS_CUDA(ctx, cudaStreamSynchronize(s));
  }
  *nnz = m;
  return MDS_OK;
}

extern "C" int mds_sysparse(mds_ctx* ctx, const double* dist, const int32_t* idx, int n_rows, int maxk, int k,
                            unsigned flags, int32_t* pcol, int32_t* irow, double* val, int64_t cap,
                            int64_t* nnz) {
  return assemble_api(ctx, dist, idx, n_rows, maxk, k, flags, 0, pcol, irow, val, cap, nnz);
}

extern "C" int mds_gesparse(mds_ctx* ctx, const double* dist, const int32_t* idx, int n_rows, int maxk, int k,
                            int symmetric, unsigned flags, int32_t* pcol, int32_t* irow, double* val,
                            int64_t cap, int64_t* nnz) {
  return assemble_api(ctx, dist, idx, n_rows, maxk, k, flags, symmetric ? 2 : 1, pcol, irow, val, cap, nnz);
}
