// Host-side interface of the tcgen05 / TMEM / TMA contraction kernels (tc_gemm.cu).
#pragma once
#include "nc_common.cuh"

namespace tc {

// D(M,N) row-major (ldd) = alpha * A * B^T + beta * D + bias[n].
//   a_mn == false: A stored (M,K) row-major, lda;  a_mn == true: A stored (K,M) row-major, lda.
//   b_mn == false: B stored (N,K) row-major, ldb;  b_mn == true: B stored (K,N) row-major, ldb.
// mode: NC_CUDA_MATH_TF32 / _TF32_RNA / _3XTF32.
// Returns NC_CUDA_ERR_UNSUPPORTED (without setting the sticky status) when the problem is too small to be worth a 128-row
// tile; the caller then uses a CUDA-core kernel.  Operands TMA cannot describe (leading dimension or base not made of 16-byte
// pieces) are copied first.
int gemm(float* D, int ldd, const float* A, int lda, bool a_mn, const float* B, int ldb, bool b_mn, int M, int N,
         int K, const float* bias, float alpha, float beta, int mode, cudaStream_t st);

// The same in plain TF32 on pairs of SMs (tc_gemm2.cu), 256 x 256 tiles, no split; operands TMA can describe, an MN-major operand's
// extent a multiple of 32; NC_CUDA_ERR_UNSUPPORTED otherwise.
int gemm_pair(float* D, int ldd, const float* A, int lda, bool a_mn, const float* B, int ldb, bool b_mn, int M, int N, int K,
              const float* bias, float alpha, float beta, cudaStream_t st);

// whether gemm() takes a product of these sizes; aligned: both operands are made of 16-byte pieces
bool gemm_eligible(int M, int N, int K, bool aligned);

// planes of the packed weights in a math mode: 2 (value rounded to TF32, rounded remainder) for 3xTF32, else 1
int mode_planes(int mode);

// Channels-last implicit-GEMM convolution, stride 1:
//   y(N,Ho,Wo,Cout) = conv(x(N,H,W,Cin), wpacked) + bias,  Ho = H + 2*pad - kH + 1.
// wpacked is (plane, tap, Cout, Cin) dense - see pack_weights_*.
int conv_nhwc(float* y, const float* x, const float* wpacked, const float* bias, int N, int H, int W, int Cin,
              int Cout, int kH, int kW, int pad, int mode, cudaStream_t st);

bool conv_eligible(int Cin, int Cout, long long pixels);   // whether conv_nhwc takes these channel counts and output pixels

// The same with stride 2, and its input gradient: dx(N,H,W,Cin) from dy and weights packed per residue class.
bool conv_strided_eligible(int Cin, int Cout, long long pixels, int kH, int kW, int stride);
int conv_strided_nhwc(float* y, const float* x, const float* wpacked, const float* bias, int N, int H, int W, int Cin, int Cout,
                      int kH, int kW, int stride, int pad, int mode, cudaStream_t st);
int conv_dx_strided_nhwc(float* dx, const float* dy, const float* wpacked, int N, int H, int W, int Cin, int Cout, int kH, int kW,
                         int stride, int pad, int mode, cudaStream_t st);

// dW partials for a channels-last convolution of stride 1 or 2 and their ordered reduction into the
// reference weight layout (Cout, Cin, kH, kW).
int conv_dw_nhwc(float* dW, const float* dy, const float* x, int N, int H, int W, int Cin, int Cout, int kH, int kW,
                 int stride, int pad, int mode, cudaStream_t st);

// Halo-resident kernels (tc_conv.cu), stride 1, filters up to 3 x 3; NC_CUDA_ERR_UNSUPPORTED otherwise.  planes: 1, or 2 when x, dy
// and the weights are split into hi and lo planes.
//   conv_halo_nhwc:    forward / input gradient with the activation halo of a pixel tile resident in shared memory
//   conv_dw_halo_nhwc: weight gradient with one dY tile and one x halo tile serving all filter taps of a row
int conv_halo_nhwc(float* y, const float* x, const float* wpacked, const float* bias, int N, int H, int W, int Cin, int Cout,
                   int kH, int kW, int pad, int planes, cudaStream_t st);
int conv_dw_halo_nhwc(float* dW, const float* dy, const float* x, int N, int H, int W, int Cin, int Cout, int kH, int kW,
                      int pad, int planes, cudaStream_t st);
// partial[z][co][(kh*kW+kw)*Cp + ci] summed over z in order -> dW (Cout, Cin, kH, kW); Cp = Cin in whole 32-channel chunks
int dw_reduce(float* dW, const float* partial, int splits, int Cout, int Cin, int kH, int kW, cudaStream_t st);

// (Cout,Cin,kH,kW) -> (plane,kH,kW,Cout,Cin) for the forward; for dX -> (plane,taps,Cin,Cout), the filter reversed, or for stride 2
// the reversed filters of the residue classes (0,0), (0,1), (1,0), (1,1) one after the other.
int pack_weights_fwd(float* wp, const float* w, int Cout, int Cin, int kH, int kW, int planes, cudaStream_t st);
int pack_weights_dx(float* wp, const float* w, int Cout, int Cin, int kH, int kW, int stride, int pad, int planes, cudaStream_t st);

}  // namespace tc
