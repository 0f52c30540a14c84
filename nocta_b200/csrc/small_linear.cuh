// Host interface of the small matrix products (small_linear.cu), FP32 on CUDA cores.
#pragma once
#include "nc_common.cuh"

namespace ncc {

// d[m][n] = sum_k a[m][k] * b[n][k] + bias[n]; rows of a and b contiguous along k.  round_b: b rounded to TF32 as it is read
int small_rows(float* d, long long ldd, const float* a, long long lda, const float* b, long long ldb, const float* bias, int M, int N,
               int K, bool round_b, cudaStream_t st);

// d[r][c] = sum_k a[r * a_sr + k * a_sk] * b[k * ldb + c]; row_sums (may be null): sum over k of a(r, k).  d == nullptr: no job
struct ColumnsJob {
    float* d;
    long long ldd;
    const float* a;
    long long a_sr, a_sk;
    const float* b;
    long long ldb;
    float* row_sums;
    int R, C, K;
    int round_b;                  // b rounded to TF32 as it is read
    int col_tiles, blocks, vec;   // set by small_columns
};
int small_columns(ColumnsJob j0, ColumnsJob j1, cudaStream_t st);

}  // namespace ncc
