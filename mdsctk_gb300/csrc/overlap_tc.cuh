// overlap_tc.cuh -- tensor-core kNN of binary vectors (overlap_tc.cu).
#pragma once

#include "knn_common.cuh"

// Bytes of a row of `dim` indices; tiles of the product; the length of a
// reference set's count array (whole column tiles, the padding readable).
int64_t overlap_width(int dim);
int overlap_tiles(int nfit, int nref);
int overlap_count_pad(int n);
// CSR rows -> e4m3 byte rows [n][K] and their counts; *bad (device, zeroed by
// the caller) is set when a value is not 1.0 or a row's indices do not ascend
// strictly within [0, K).
int launch_rows_e4m3(mds_ctx* ctx, const int64_t* off, const int* idx, const double* val, int n, int64_t K,
                     unsigned char* out, int* cnt, int* bad);
// The k nearest reference rows of every fit row, position 0 dropped (device
// arrays; counts below 2^24 in all).
int overlap_knn(mds_ctx* ctx, const unsigned char* Bf, const int* cf, int nfit, const unsigned char* Br, const int* cr,
                int nref, int64_t K, int k, double* out_d, int* out_i);
