// Direct convolutions for layers with fewer channels than a tensor-core tile wants (1 -> 6 -> 16 channels and the like), FP32.
//
// A layer of this kind is a fraction of a GFLOP; what it costs is latency: address arithmetic per operand element, half-empty
// 64 x 64 tiles, separate launches for the bias gradient and the split reduction.  Here a block stages the rows it needs and
// all weights in shared memory once and then runs on registers: a thread owns four neighbouring pixels x 4 output channels and
// slides a window of k + 3 inputs along the filter row.
// Batch 64, 6 -> 16 channels, 12 x 12: forward 28 -> 4 us, input gradient 102 -> 6 us, weight + bias gradient 29 -> 8 us.
#include "small_conv.cuh"

namespace smallconv {
namespace {

struct Geo {
    int N, Cin, H, W, Cout, Ho, Wo, pad;
    long long xs[4], ys[4];
    int rows, bands;      // output rows per block, blocks per image
    int pitch, in_rows;   // staged input rows of `pitch` floats
    int cog;              // groups of four output channels
};

constexpr int kMaxSmem = 96 * 1024;

// rows [h0, h0 + in_rows) of image n with zero padding: tile[c][row][col], col 0 = image column -pad
__device__ __forceinline__ void stage_image(float* tile, const float* __restrict__ t, const long long s[4], int n, int C, int H, int W,
                                            int h0, int pad, int in_rows, int pitch) {
    const int per = in_rows * pitch, total = C * per;
    const bool cl = s[1] == 1 && C > 1;   // channels-last: consecutive threads along the channels
#pragma unroll 4
    for (int i = threadIdx.x; i < total; i += blockDim.x) {
        int c, r;
        if (cl) { c = i % C; r = i / C; } else { c = i / per; r = i - c * per; }
        const int row = r / pitch, col = r - row * pitch, h = h0 + row, w = col - pad;
        float v = 0.f;
        if (h >= 0 && h < H && w >= 0 && w < W) v = __ldg(t + n * s[0] + c * s[1] + h * s[2] + w * s[3]);
        tile[c * per + r] = v;
    }
}

// A thread owns kPX pixels x 4 output channels over the input channels ci = slice, slice + slices, ...; the slices of one output
// are added through shared memory in slice order, which also puts consecutive channels on consecutive threads for the store.
// A forward pass is not sliced but takes fewer pixels per thread: its sums then run in the order of the general path, and the
// ReLU and max-pool decisions behind it come out the same whichever of the two takes the layer.
template <int K, int kPX>
__global__ void __launch_bounds__(256) conv_kernel(float* __restrict__ y, const float* __restrict__ x, const float* __restrict__ w,
                                                   const float* __restrict__ bias, Geo g, int flip, int slices) {
    ncc::pdl_wait();
    extern __shared__ __align__(16) float sm[];
    constexpr int KK = K * K;
    const int taps = g.Cin * KK, c4 = g.cog * 4;
    float* wsm = sm;                          // [tap][c4]
    float* tile = sm + taps * c4;
    const int n = blockIdx.x / g.bands, band = blockIdx.x - n * g.bands;
    const int ho0 = band * g.rows, nrows = (g.Ho - ho0) < g.rows ? (g.Ho - ho0) : g.rows;
    // weights in their own order (coalesced); four requests in flight per thread
#pragma unroll 4
    for (int i = threadIdx.x; i < taps * g.Cout; i += 256) {
        int co, tap;
        if (!flip) { co = i / taps; tap = i - co * taps; }
        else { const int r = i / KK, kk = i - r * KK, ci = r / g.Cout; co = r - ci * g.Cout; tap = ci * KK + KK - 1 - kk; }
        wsm[tap * c4 + co] = __ldg(w + i);
    }
    if (c4 != g.Cout)
        for (int i = threadIdx.x; i < taps * (c4 - g.Cout); i += 256) wsm[i / (c4 - g.Cout) * c4 + g.Cout + i % (c4 - g.Cout)] = 0.f;
    stage_image(tile, x, g.xs, n, g.Cin, g.H, g.W, ho0 - g.pad, g.pad, g.in_rows, g.pitch);
    __syncthreads();
    const int pxg = (g.Wo + kPX - 1) / kPX, items = nrows * pxg * g.cog;
    float* red = tile + ((g.Cin * g.in_rows * g.pitch + 3) & ~3);   // [slice][item][kPX * 4] when there are slices
    for (int it0 = threadIdx.x; it0 < items * slices; it0 += 256) {
        const int slice = it0 / items, it = it0 - slice * items;
        const int cg = it % g.cog, t = it / g.cog, w0 = (t % pxg) * kPX, row = t / pxg;
        float acc[kPX][4];
#pragma unroll
        for (int p = 0; p < kPX; p++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[p][e] = 0.f;
        const float* wp = wsm + cg * 4;
        for (int ci = slice; ci < g.Cin; ci += slices) {
#pragma unroll
            for (int kh = 0; kh < K; kh++) {
                const float* xr = tile + (ci * g.in_rows + row + kh) * g.pitch + w0;
                float xv[kPX + K - 1];
#pragma unroll
                for (int j = 0; j < kPX + K - 1; j++) xv[j] = xr[j];
#pragma unroll
                for (int kw = 0; kw < K; kw++) {
                    const float4 q = *reinterpret_cast<const float4*>(wp + ((ci * K + kh) * K + kw) * c4);
#pragma unroll
                    for (int p = 0; p < kPX; p++) {
                        acc[p][0] = fmaf(xv[p + kw], q.x, acc[p][0]);
                        acc[p][1] = fmaf(xv[p + kw], q.y, acc[p][1]);
                        acc[p][2] = fmaf(xv[p + kw], q.z, acc[p][2]);
                        acc[p][3] = fmaf(xv[p + kw], q.w, acc[p][3]);
                    }
                }
            }
        }
        if (slices == 1) {
            float* dst = y + n * g.ys[0] + (long long)(ho0 + row) * g.ys[2] + w0 * g.ys[3] + (long long)(cg * 4) * g.ys[1];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                if (cg * 4 + e >= g.Cout) break;
                const float b = bias ? bias[cg * 4 + e] : 0.f;
#pragma unroll
                for (int p = 0; p < kPX; p++)
                    if (w0 + p < g.Wo) dst[p * g.ys[3] + e * g.ys[1]] = acc[p][e] + b;
            }
        } else {
#pragma unroll
            for (int p = 0; p < kPX; p++)
                *reinterpret_cast<float4*>(red + ((size_t)slice * items * kPX + (size_t)t * kPX * g.cog + p * g.cog + cg) * 4) =
                    make_float4(acc[p][0], acc[p][1], acc[p][2], acc[p][3]);
        }
    }
    if (slices == 1) return;
    __syncthreads();
    const int outs = items * kPX * 4;   // (row, pixel group, pixel, channel)
    for (int i = threadIdx.x; i < outs; i += 256) {
        const int co = i % c4, px = i / c4, p = px % kPX, t = px / kPX, wo = (t % pxg) * kPX + p, row = t / pxg;
        if (co >= g.Cout || wo >= g.Wo) continue;
        float s = 0.f;
        for (int k = 0; k < slices; k++) s += red[(size_t)k * outs + i];
        y[n * g.ys[0] + (long long)(ho0 + row) * g.ys[2] + wo * g.ys[3] + co * g.ys[1]] = s + (bias ? bias[co] : 0.f);
    }
}

// Weight gradient: a block walks its share of the images; thread (row group, co, ci, kh) keeps the K taps of one filter row in
// registers and takes four pixels at a time (three 16-byte shared-memory reads for 4 K multiply-adds).  Row groups are combined
// through shared memory, the eight blocks of a cluster through distributed shared memory, clusters through `partial` by the
// block that arrives last (fixed orders, in double): the whole gradient is one launch and bit-stable.
__device__ unsigned int g_ticket;   // wraps to zero with the last block of a launch
constexpr int kCluster = 8;

template <int K>
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(1024)
dw_kernel(float* __restrict__ dW, float* __restrict__ db, const float* __restrict__ dy, const float* __restrict__ x,
          float* __restrict__ partial, Geo g, int filters, int rgroups, int images, int dpitch) {
    ncc::pdl_wait();
    extern __shared__ __align__(16) float sm[];
    __shared__ bool last;
    __shared__ float bias_sh[32];
    constexpr int XV = (4 + K - 1 + 3) / 4 * 4;   // inputs of four pixels, whole 16-byte reads
    const int dper = g.Ho * dpitch, xper = g.in_rows * g.pitch;
    float* xt = sm;                       // [ci][row][col]
    float* dt = sm + g.Cin * xper;        // [co][row][col], zeros beyond Wo
    const int n0 = blockIdx.x * images, n1 = (n0 + images) < g.N ? n0 + images : g.N;
    const int item = threadIdx.x, rg = item / filters, f = item - rg * filters;   // f = (co, ci, kh), kh fastest
    const int kh = f % K, ci = (f / K) % g.Cin, co = f / (K * g.Cin);
    const bool live = rg < rgroups;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float acc[K];
#pragma unroll
    for (int j = 0; j < K; j++) acc[j] = 0.f;
    double bsum = 0.0;   // this lane's share of the bias gradient of channel `warp`
    for (int n = n0; n < n1; n++) {
        __syncthreads();
        stage_image(xt, x, g.xs, n, g.Cin, g.H, g.W, -g.pad, g.pad, g.in_rows, g.pitch);
        stage_image(dt, dy, g.ys, n, g.Cout, g.Ho, g.Wo, 0, 0, g.Ho, dpitch);
        __syncthreads();
        if (live) {
            for (int r = rg; r < g.Ho; r += rgroups) {
                const float* xr = xt + ci * xper + (r + kh) * g.pitch;
                const float* dr = dt + co * dper + r * dpitch;
                int w = 0;
#pragma unroll 2
                for (; w + 4 <= g.Wo; w += 4) {
                    float xv[XV];
#pragma unroll
                    for (int j = 0; j < XV; j += 4) *reinterpret_cast<float4*>(xv + j) = *reinterpret_cast<const float4*>(xr + w + j);
                    const float4 d = *reinterpret_cast<const float4*>(dr + w);
#pragma unroll
                    for (int j = 0; j < K; j++) acc[j] = fmaf(d.w, xv[3 + j], fmaf(d.z, xv[2 + j], fmaf(d.y, xv[1 + j], fmaf(d.x, xv[j], acc[j]))));
                }
                // one by one: a zero of the padding times an infinity further along the row would be a NaN in taps that never see it
                for (; w < g.Wo; w++) {
                    const float d = dr[w];
#pragma unroll
                    for (int j = 0; j < K; j++) acc[j] = fmaf(d, xr[w + j], acc[j]);
                }
            }
        }
        if (db && warp < g.Cout)
            for (int i = lane; i < dper; i += 32) bsum += (double)dt[warp * dper + i];
    }
    __syncthreads();
    float* red = sm;   // [row group][co][ci][kh][kw]; after the row groups are added: group 0 holds the block's gradient
    if (live)
#pragma unroll
        for (int j = 0; j < K; j++) red[(rg * filters + f) * K + j] = acc[j];
    if (db && warp < g.Cout) {
        bsum = ncc::warp_sum(bsum);
        if (lane == 0) bias_sh[warp] = (float)bsum;
    }
    __syncthreads();
    const int outs = filters * K;   // (co, ci, kh, kw) order = dW's own
    for (int i = threadIdx.x; i < outs; i += blockDim.x) {
        float s = red[i];
        for (int r = 1; r < rgroups; r++) s += red[r * outs + i];
        red[i] = s;
    }
    ncc::cluster_sync();
    const uint32_t rank = ncc::cluster_rank();
    const int all = outs + g.Cout;   // one row of `partial`: the weight gradient, then the bias gradient
    float* prow = partial + (size_t)(blockIdx.x / kCluster) * all;
    for (int i = (int)rank * blockDim.x + threadIdx.x; i < all; i += kCluster * blockDim.x) {
        const float* src = i < outs ? red + i : bias_sh + (i - outs);
        float v[kCluster];
#pragma unroll
        for (uint32_t b = 0; b < kCluster; b++) v[b] = ncc::ld_cluster(src, b);
        double s = 0.0;
#pragma unroll
        for (int b = 0; b < kCluster; b++) s += (double)v[b];
        prow[i] = (float)s;
    }
    __threadfence();
    ncc::cluster_sync();   // no block of the cluster leaves while its shared memory is read
    if (threadIdx.x == 0) last = atomicInc(&g_ticket, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    const int clusters = gridDim.x / kCluster;
    for (int i = threadIdx.x; i < (db ? all : outs); i += blockDim.x) {
        double s = 0.0;
#pragma unroll 8
        for (int b = 0; b < clusters; b++) s += (double)__ldcg(partial + (size_t)b * all + i);
        if (i < outs) dW[i] = (float)s;
        else db[i - outs] = (float)s;
    }
}

Geo make(int N, int Cin, int H, int W, int Cout, int k, int pad, const long long xs[4], const long long ys[4]) {
    Geo g = {};
    g.N = N; g.Cin = Cin; g.H = H; g.W = W; g.Cout = Cout; g.pad = pad;
    g.Ho = H + 2 * pad - k + 1; g.Wo = W + 2 * pad - k + 1;
    for (int i = 0; i < 4; i++) { g.xs[i] = xs[i]; g.ys[i] = ys[i]; }
    g.cog = (Cout + 3) / 4;
    return g;
}

template <int K, int kPX>
int launch_conv(float* y, const float* x, const float* w, const float* bias, Geo g, bool flip, cudaStream_t st) {
    g.pitch = (g.Wo + kPX - 1) / kPX * kPX + K - 1;   // the last pixel group may read beyond the image: zeros
    g.in_rows = g.rows + K - 1;
    const int items = g.rows * ((g.Wo + kPX - 1) / kPX) * g.cog;
    // input gradient: slices of the channels until the 256 threads of a block have work
    int slices = flip ? 256 / items : 1;
    if (slices > g.Cin) slices = g.Cin;
    if (slices < 1) slices = 1;
    const size_t tile = (((size_t)g.Cin * g.in_rows * g.pitch) + 3) & ~(size_t)3;
    size_t smem = sizeof(float) * ((size_t)g.Cin * K * K * g.cog * 4 + tile);
    if (slices > 1) smem += sizeof(float) * (size_t)slices * items * kPX * 4;
    if (smem > kMaxSmem || (long long)g.N * g.bands > 0x7fffffffLL) return NC_CUDA_ERR_UNSUPPORTED;
    static bool set = false;
    if (!set) { NCC_TRY(cudaFuncSetAttribute(conv_kernel<K, kPX>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem)); set = true; }
    ncc::launch(conv_kernel<K, kPX>, g.N * g.bands, 256, smem, st, y, x, w, bias, g, flip ? 1 : 0, slices);
    NCC_COUNT_LAUNCH();
    return ncc::launch_status("small_conv");
}
// pixels per thread: four, fewer in a forward pass whose block has no work for 256 threads then
template <int K>
int pick_conv(float* y, const float* x, const float* w, const float* bias, const Geo& g, bool flip, cudaStream_t st) {
    auto items = [&](int px) { return (long long)g.rows * ((g.Wo + px - 1) / px) * g.cog; };
    if (flip || items(2) > 256) return launch_conv<K, 4>(y, x, w, bias, g, flip, st);
    if (items(1) > 256) return launch_conv<K, 2>(y, x, w, bias, g, flip, st);
    return launch_conv<K, 1>(y, x, w, bias, g, flip, st);
}

template <int K>
int launch_dw(float* dW, float* db, const float* dy, const float* x, Geo g, cudaStream_t st) {
    const int filters = g.Cout * g.Cin * K;
    if (filters > 1024) return NC_CUDA_ERR_UNSUPPORTED;
    int rgroups = 1024 / filters;
    if (rgroups > g.Ho) rgroups = g.Ho;
    int threads = (filters * rgroups + 31) / 32 * 32;
    if (threads < 32 * g.Cout) threads = 32 * g.Cout;   // one warp per channel sums the bias gradient
    if (threads > 1024) return NC_CUDA_ERR_UNSUPPORTED;
    const int dpitch = (g.Wo + 3) & ~3;
    g.in_rows = g.H + 2 * g.pad;
    g.pitch = (dpitch + K - 1 + 3 + 3) & ~3;   // whole 16-byte reads, also for the last four pixels
    size_t smem = sizeof(float) * ((size_t)g.Cin * g.in_rows * g.pitch + (size_t)g.Cout * g.Ho * dpitch);
    const size_t red = sizeof(float) * (size_t)filters * rgroups * K;
    if (red > smem) smem = red;
    if (smem > kMaxSmem) return NC_CUDA_ERR_UNSUPPORTED;
    const int images = (g.N + ncc::sm_count() - 1) / ncc::sm_count();   // about a block per SM
    const int blocks = ((g.N + images - 1) / images + kCluster - 1) / kCluster * kCluster;
    float* partial = (float*)ncc::scratch(2, sizeof(float) * (size_t)(filters * K + g.Cout) * (blocks / kCluster), st);
    if (!partial) return NC_CUDA_ERR_RUNTIME;
    static bool set = false;
    if (!set) { NCC_TRY(cudaFuncSetAttribute(dw_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem)); set = true; }
    ncc::launch(dw_kernel<K>, blocks, threads, smem, st, dW, db, dy, x, partial, g, filters, rgroups, images, dpitch);
    NCC_COUNT_LAUNCH();
    return ncc::launch_status("small_conv weight gradient");
}

}  // namespace

int conv(float* y, const long long ys[4], const float* x, const long long xs[4], const float* w, const float* bias, int N, int Cin,
         int H, int W, int Cout, int k, int pad, bool flip, cudaStream_t st) {
    // few channels on one side: what the tensor-core kernels do not take
    if ((Cin >= 16 && Cout >= 16) || Cin > 32 || Cout > 32) return NC_CUDA_ERR_UNSUPPORTED;
    Geo g = make(N, Cin, H, W, Cout, k, pad, xs, ys);
    if (g.Ho <= 0 || g.Wo <= 0) return NC_CUDA_ERR_UNSUPPORTED;
    // bands of rows until there is a block per SM, or more when a band would not fit
    int bands = 1;
    while (bands * 4 <= g.Ho && (long long)N * bands < ncc::sm_count()) bands *= 2;
    while (bands < g.Ho && (size_t)Cin * (((g.Ho + bands - 1) / bands) + k - 1) * (g.Wo + k + 3) > 12 * 1024) bands *= 2;
    g.rows = (g.Ho + bands - 1) / bands;
    g.bands = (g.Ho + g.rows - 1) / g.rows;
    switch (k) {
        case 3: return pick_conv<3>(y, x, w, bias, g, flip, st);
        case 5: return pick_conv<5>(y, x, w, bias, g, flip, st);
        case 7: return pick_conv<7>(y, x, w, bias, g, flip, st);
    }
    return NC_CUDA_ERR_UNSUPPORTED;
}

int weight_grad(float* dW, float* db, const float* dy, const long long ys[4], const float* x, const long long xs[4], int N, int Cin,
                int H, int W, int Cout, int k, int pad, cudaStream_t st) {
    Geo g = make(N, Cin, H, W, Cout, k, pad, xs, ys);
    if (g.Ho <= 0 || g.Wo <= 0) return NC_CUDA_ERR_UNSUPPORTED;
    switch (k) {
        case 3: return launch_dw<3>(dW, db, dy, x, g, st);
        case 5: return launch_dw<5>(dW, db, dy, x, g, st);
        case 7: return launch_dw<7>(dW, db, dy, x, g, st);
    }
    return NC_CUDA_ERR_UNSUPPORTED;
}

}  // namespace smallconv
