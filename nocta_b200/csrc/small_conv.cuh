// Host interface of the direct convolutions for few channels (small_conv.cu), FP32 on CUDA cores.
#pragma once
#include "nc_common.cuh"

namespace smallconv {

// Stride-1 convolution with square 3 x 3, 5 x 5 or 7 x 7 filters and few channels:
//   y[n][co][h][w] = sum x[n][ci][h + kh - pad][w + kw - pad] * w(co, ci, kh, kw) + bias[co]
// xs, ys: element strides (n, c, h, w).  flip: weights are stored (Cin, Cout, k, k) and taken with both filter axes reversed
// (input gradient).  NC_CUDA_ERR_UNSUPPORTED (status not set) outside its range.
int conv(float* y, const long long ys[4], const float* x, const long long xs[4], const float* w, const float* bias, int N, int Cin,
         int H, int W, int Cout, int k, int pad, bool flip, cudaStream_t st);

// weight and bias gradient of the same convolution in one launch (db may be null)
int weight_grad(float* dW, float* db, const float* dy, const long long ys[4], const float* x, const long long xs[4], int N, int Cin,
                int H, int W, int Cout, int k, int pad, cudaStream_t st);

}  // namespace smallconv
