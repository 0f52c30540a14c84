// FP32 CUDA-core kernels for matrix products too small (or too thin) for 128-row tensor-core tiles: the Linear layers of small
// networks, a handful of rows against a large weight matrix, ten output columns.  Each product is one launch, the bias, the
// split reduction and the bias gradient included: at these sizes a launch costs the host about 3 us, more than most of the
// kernels run.
//
//   rows_kernel     y[m][n] = sum_k a[m][k] * b[n][k] + bias[n]       both operands contiguous along k
//   columns_kernel  d[r][c] = sum_k a(r, k) * b[k][c]                 b contiguous along c, lanes along c; two such products
//                   (input and weight gradient of a Linear layer) and the bias gradient share one launch
//
// Every output is summed by a fixed assignment of k to lanes and warps and combined in a fixed order: bit-stable.
#include "nc_common.cuh"
#include "small_linear.cuh"
#include "tc_ptx.cuh"

namespace ncc {
namespace {

constexpr int kWarps = 8;

// rows_kernel: a block owns MT rows of a, 32 rows of b (one per lane) and up to 1024 k; longer sums are split over a cluster of up
// to eight blocks.  Every row arrives as one bulk copy, all of them in flight at once; a warp then takes one of KS slices of k from
// shared memory, b one row per lane, a broadcast, with MR accumulators a thread and no exchange between lanes.  Slices, then the
// blocks of the cluster, are added in order.  KS = 8, all warps along k, but for sums of up to 256 the slices are those of the
// general path (simt_matmul: none below 256, then of 64) and the other warps take other rows: the layers of small networks get the
// same sums from both, and so the same ReLU decisions.
// Bound by reading b and by the copy engine: whole rows (4 KB) per copy; with a copy per row and warp (512 bytes) the same kernel
// took 11 us for 16 rows against 4096 x 1024 weights, as did loads into registers with k across the lanes; 64 x 64 tiles 53 us.
constexpr int kSlice = 128;   // k per warp at most

template <int MT, int KS>
__global__ void __launch_bounds__(kWarps * 32) rows_kernel(float* __restrict__ d, long long ldd, const float* __restrict__ a, long long lda,
                                                           const float* __restrict__ b, long long ldb, const float* __restrict__ bias,
                                                           int M, int N, int K, int slice, int wpitch, int blocks_k, int round_b,
                                                           unsigned int* err) {
    extern __shared__ __align__(128) float sm[];   // a [MT][KS * slice], b [32][wpitch]
    constexpr int MR = MT * KS / kWarps;           // rows a warp sums
    static_assert(MR >= 1, "a row per warp");
    __shared__ float red[KS][MT][32];
    __shared__ __align__(8) uint64_t bar[2];
    __shared__ int abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, chunk = KS * slice, ks = warp % KS, r0 = warp / KS * MR;
    const int n = blockIdx.x / blocks_k * 32 + lane, m0 = blockIdx.y * MT;
    const int k0 = (int)(blockIdx.x % blocks_k) * chunk, kb = (K - k0) < chunk ? (K - k0) : chunk;   // this block's k
    float* xs = sm;
    float* ws = sm + MT * chunk;
    if (threadIdx.x == 0) {
        tc::mbar_init(tc::smem_u32(&bar[0]), 1);
        tc::mbar_init(tc::smem_u32(&bar[1]), 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    ncc::pdl_wait();
    // Rows over 512 values come in two halves, the second one in flight while the first is multiplied (each half dealt to the warps).
    const int half = (KS == kWarps && kb > 512) ? (kb / 2 + 3) & ~3 : kb;
    if (warp == 0) {
        const int rows_a = (M - m0) < MT ? (M - m0) : MT, rows_b = (N - (n - lane)) < 32 ? (N - (n - lane)) : 32;
        for (int h = 0; h * half < kb; h++) {
            const uint32_t full = tc::smem_u32(&bar[h]), bytes = (uint32_t)((kb - h * half) < half ? (kb - h * half) : half) * 4u;
            if (lane == 0) tc::mbar_expect_tx(full, bytes * (uint32_t)(rows_a + rows_b));
            __syncwarp();
            if (lane < rows_b) tc::bulk_copy(tc::smem_u32(ws + lane * wpitch + h * half), b + (long long)n * ldb + k0 + h * half, bytes, full);
            if (lane < rows_a) tc::bulk_copy(tc::smem_u32(xs + lane * chunk + h * half), a + (long long)(m0 + lane) * lda + k0 + h * half, bytes, full);
        }
    }
    float acc[MR];
#pragma unroll
    for (int m = 0; m < MR; m++) acc[m] = 0.f;
    bool ok = true;
    for (int h = 0; h * half < kb && ok; h++) {
        ok = tc::mbar_wait(tc::smem_u32(&bar[h]), 0u, err, 0xD00u + h, &abort_flag);
        if (!ok) break;
        // this warp's part of the half
        const int hn = (kb - h * half) < half ? (kb - h * half) : half, part = half == kb ? slice : ((hn + KS - 1) / KS + 3) & ~3;
        const int kn = (hn - ks * part) < part ? (hn - ks * part) : part;   // may be <= 0
        const float4* wq = reinterpret_cast<const float4*>(ws + lane * wpitch + h * half + ks * part);
        const float4* xq = reinterpret_cast<const float4*>(xs + r0 * chunk + h * half + ks * part);
#pragma unroll 4
        for (int q = 0; q < kn >> 2; q++) {
            float4 w = wq[q];
            if (round_b) w = make_float4(round_tf32(w.x), round_tf32(w.y), round_tf32(w.z), round_tf32(w.w));
#pragma unroll
            for (int m = 0; m < MR; m++) {
                const float4 x = xq[m * (chunk >> 2) + q];
                acc[m] = fmaf(x.w, w.w, fmaf(x.z, w.z, fmaf(x.y, w.y, fmaf(x.x, w.x, acc[m]))));
            }
        }
    }
    if (!ok) {
        const unsigned long long t0 = tc::global_ns();   // copies in flight land before the block gives its memory back
        while (tc::global_ns() - t0 < 2000000ull) { }
    }
#pragma unroll
    for (int m = 0; m < MR; m++) red[ks][r0 + m][lane] = acc[m];
    __syncthreads();
    for (int i = threadIdx.x; i < MT * 32; i += kWarps * 32) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < KS; w++) s += red[w][i >> 5][i & 31];
        red[0][i >> 5][i & 31] = s;   // only this thread reads it before
        const int m = m0 + (i >> 5), nn = n - lane + (i & 31);
        if (blocks_k == 1 && m < M && nn < N) d[(long long)m * ldd + nn] = s + (bias ? bias[nn] : 0.f);
    }
    if (blocks_k == 1) return;
    cluster_sync();
    const int rank = (int)cluster_rank();
    for (int i = threadIdx.x * blocks_k + rank; i < MT * 32; i += kWarps * 32 * blocks_k) {
        float s = 0.f;
        for (int r = 0; r < blocks_k; r++) s += ld_cluster(&red[0][i >> 5][i & 31], (uint32_t)r);
        const int m = m0 + (i >> 5), nn = n - lane + (i & 31);
        if (m < M && nn < N) d[(long long)m * ldd + nn] = s + (bias ? bias[nn] : 0.f);
    }
    cluster_sync();   // no block leaves while its sums are read
}

// the same product for operands that are not made of whole 16-byte pieces: lanes along k, a warp owns four rows of b and eight of a
template <int T>
__device__ __forceinline__ void reduce_lanes(float (&acc)[T], float* red, int lane) {
    // every exchange halves the values a lane still carries: value lane ends in red[lane]
    static_assert(T == 32, "one value per lane");
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < 16; i++)
            if (i < o) {
                const float send = up ? acc[i] : acc[i + o], keep = up ? acc[i + o] : acc[i];
                acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
    }
    red[lane] = acc[0];
}
__global__ void __launch_bounds__(kWarps * 32) rows_odd_kernel(float* __restrict__ d, long long ldd, const float* __restrict__ a,
                                                               long long lda, const float* __restrict__ b, long long ldb,
                                                               const float* __restrict__ bias, int M, int N, int K, int ks_log2,
                                                               int round_b) {
    ncc::pdl_wait();
    constexpr int NW = 4, MT = 8;
    __shared__ float red[kWarps][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int KS = 1 << ks_log2, ks = warp & (KS - 1), ng = warp >> ks_log2, groups = kWarps >> ks_log2;
    const int nb0 = blockIdx.x * groups * NW, n0 = nb0 + ng * NW, m0 = blockIdx.y * MT;
    const int steps = (K + 31) / 32, s0 = (int)((long long)steps * ks / KS), s1 = (int)((long long)steps * (ks + 1) / KS);
    float acc[32];
#pragma unroll
    for (int t = 0; t < 32; t++) acc[t] = 0.f;
    for (int s = s0; s < s1; s++) {
        const int k = s * 32 + lane;
        if (k >= K) break;
        float w[NW], x[MT];
#pragma unroll
        for (int j = 0; j < NW; j++) w[j] = __ldg(b + (long long)(n0 + j < N ? n0 + j : N - 1) * ldb + k);
#pragma unroll
        for (int m = 0; m < MT; m++) x[m] = __ldg(a + (long long)(m0 + m < M ? m0 + m : M - 1) * lda + k);
#pragma unroll
        for (int j = 0; j < NW; j++) {
            if (round_b) w[j] = round_tf32(w[j]);
#pragma unroll
            for (int m = 0; m < MT; m++) acc[m * NW + j] = fmaf(x[m], w[j], acc[m * NW + j]);
        }
    }
    __syncwarp();
    reduce_lanes<32>(acc, red[warp], lane);
    __syncthreads();
    for (int i = threadIdx.x; i < groups * 32; i += kWarps * 32) {
        const int g = i >> 5, t = i & 31, m = m0 + t / NW, nn = nb0 + g * NW + t % NW;
        if (m >= M || nn >= N) continue;
        float s = 0.f;
        for (int k = 0; k < KS; k++) s += red[(g << ks_log2) + k][t];
        d[(long long)m * ldd + nn] = s + (bias ? bias[nn] : 0.f);
    }
}

// Eight output rows x 128 columns per block; the eight warps take every eighth k and are combined in order.  a(r, k) goes through
// shared memory as [k][8] so that one k costs a lane two broadcast reads, one 16-byte read of b and 32 multiply-adds.
// Up to 16 k (the input gradient of a classifier's last layer): every warp takes all of k for eight rows of its own, nothing is
// exchanged (128 x 8192 outputs, K = 10, with its weight gradient: 22 -> 13 us).
constexpr int kRT = 8, kKC = 128, kShortK = 16;

template <bool VEC>
__device__ __forceinline__ void columns_load(float (&bv)[4], const float* __restrict__ bp, const int (&col)[4], int C, int round_b) {
    if (VEC) {
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
        if (col[0] < C) q = __ldg(reinterpret_cast<const float4*>(bp + col[0]));
        bv[0] = q.x; bv[1] = q.y; bv[2] = q.z; bv[3] = q.w;
    } else {
#pragma unroll
        for (int e = 0; e < 4; e++) bv[e] = col[e] < C ? __ldg(bp + col[e]) : 0.f;
    }
    if (round_b)
#pragma unroll
        for (int e = 0; e < 4; e++) bv[e] = round_tf32(bv[e]);
}

template <bool VEC>
__device__ __forceinline__ void columns_short(const ColumnsJob& j, int block, float* as) {
    constexpr int kRows = kWarps * kRT;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r0 = (block / j.col_tiles) * kRows, ct = block % j.col_tiles, c0 = ct * 128;
    for (int i = threadIdx.x; i < j.K * kRows; i += kWarps * 32) {
        const int kk = j.a_sk == 1 ? i % j.K : i / kRows, r = j.a_sk == 1 ? i / j.K : i % kRows;
        as[kk * kRows + r] = r0 + r < j.R ? j.a[(long long)(r0 + r) * j.a_sr + (long long)kk * j.a_sk] : 0.f;
    }
    __syncthreads();
    int col[4];
#pragma unroll
    for (int e = 0; e < 4; e++) col[e] = VEC ? c0 + lane * 4 + e : c0 + lane + 32 * e;
    float acc[kRT][4];
#pragma unroll
    for (int r = 0; r < kRT; r++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[r][e] = 0.f;
#pragma unroll 4
    for (int kk = 0; kk < j.K; kk++) {
        float bv[4];
        columns_load<VEC>(bv, j.b + (long long)kk * j.ldb, col, j.C, j.round_b);
#pragma unroll
        for (int r = 0; r < kRT; r++) {
            const float av = as[kk * kRows + warp * kRT + r];
#pragma unroll
            for (int e = 0; e < 4; e++) acc[r][e] = fmaf(av, bv[e], acc[r][e]);
        }
    }
    const bool vec_out = VEC && j.ldd % 4 == 0 && (reinterpret_cast<uintptr_t>(j.d) & 15u) == 0;
#pragma unroll
    for (int r = 0; r < kRT; r++) {
        const int row = r0 + warp * kRT + r;
        if (row >= j.R) break;
        float* d = j.d + (long long)row * j.ldd;
        if (vec_out) {
            if (col[0] < j.C) *reinterpret_cast<float4*>(d + col[0]) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++) if (col[e] < j.C) d[col[e]] = acc[r][e];
        }
    }
    if (j.row_sums && ct == 0 && threadIdx.x < kRows && r0 + (int)threadIdx.x < j.R) {
        double s = 0.0;
        for (int kk = 0; kk < j.K; kk++) s += (double)as[kk * kRows + threadIdx.x];
        j.row_sums[r0 + threadIdx.x] = (float)s;
    }
}

template <bool VEC>
__device__ __forceinline__ void columns_job(const ColumnsJob& j, int block, float* as, float* red) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r0 = (block / j.col_tiles) * kRT, ct = block % j.col_tiles, c0 = ct * 128;
    float acc[kRT][4];
#pragma unroll
    for (int r = 0; r < kRT; r++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[r][e] = 0.f;
    double rowsum = 0.0;   // sum of a(r, k) over k: the bias gradient, by the blocks of column tile 0
    const bool sums = j.row_sums != nullptr && ct == 0;
    int col[4];
#pragma unroll
    for (int e = 0; e < 4; e++) col[e] = VEC ? c0 + lane * 4 + e : c0 + lane + 32 * e;
    for (int k0 = 0; k0 < j.K; k0 += kKC) {
        const int kn = (j.K - k0) < kKC ? (j.K - k0) : kKC;
        __syncthreads();
        for (int i = threadIdx.x; i < kKC * kRT; i += kWarps * 32) {
            // consecutive threads along whichever index of a is contiguous
            const int kk = j.a_sk == 1 ? i % kKC : i / kRT, r = j.a_sk == 1 ? i / kKC : i % kRT;
            as[kk * kRT + r] = (kk < kn && r0 + r < j.R) ? j.a[(long long)(r0 + r) * j.a_sr + (long long)(k0 + kk) * j.a_sk] : 0.f;
        }
        __syncthreads();
        if (sums && warp < kRT)
            for (int kk = lane; kk < kn; kk += 32) rowsum += (double)as[kk * kRT + warp];
#pragma unroll 4
        for (int kk = warp; kk < kn; kk += kWarps) {
            float bv[4];
            columns_load<VEC>(bv, j.b + (long long)(k0 + kk) * j.ldb, col, j.C, j.round_b);
            const float4 a0 = *reinterpret_cast<const float4*>(as + kk * kRT), a1 = *reinterpret_cast<const float4*>(as + kk * kRT + 4);
            const float av[kRT] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
            for (int r = 0; r < kRT; r++)
#pragma unroll
                for (int e = 0; e < 4; e++) acc[r][e] = fmaf(av[r], bv[e], acc[r][e]);
        }
    }
    // red[warp][row][column], columns of a lane 32 apart so that the writes do not conflict
#pragma unroll
    for (int r = 0; r < kRT; r++)
#pragma unroll
        for (int e = 0; e < 4; e++) red[(warp * kRT + r) * 128 + e * 32 + lane] = acc[r][e];
    __syncthreads();
    for (int i = threadIdx.x; i < kRT * 128; i += kWarps * 32) {
        const int r = i >> 7, x = i & 127, e = x >> 5, ln = x & 31;
        const int c = VEC ? c0 + ln * 4 + e : c0 + ln + 32 * e;
        if (r0 + r >= j.R || c >= j.C) continue;
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; w++) s += red[(w * kRT + r) * 128 + x];
        j.d[(long long)(r0 + r) * j.ldd + c] = s;
    }
    if (sums && warp < kRT) {
        rowsum = warp_sum(rowsum);
        if (lane == 0 && r0 + warp < j.R) j.row_sums[r0 + warp] = (float)rowsum;
    }
}

__global__ void __launch_bounds__(kWarps * 32) columns_kernel(ColumnsJob j0, ColumnsJob j1) {
    ncc::pdl_wait();
    __shared__ __align__(16) float as[kKC * kRT];
    __shared__ float red[kWarps * kRT * 128];
    const bool second = (int)blockIdx.x >= j0.blocks;
    const ColumnsJob& j = second ? j1 : j0;
    const int block = second ? (int)blockIdx.x - j0.blocks : (int)blockIdx.x;
    if (j.K <= kShortK) {
        if (j.vec) columns_short<true>(j, block, as);
        else columns_short<false>(j, block, as);
    } else if (j.vec) columns_job<true>(j, block, as, red);
    else columns_job<false>(j, block, as, red);
}

inline bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

template <int MT, int KS>
static int launch_rows(float* d, long long ldd, const float* a, long long lda, const float* b, long long ldb, const float* bias, int M,
                       int N, int K, bool round_b, cudaStream_t st) {
    const int blocks_k = (K + kWarps * kSlice - 1) / (kWarps * kSlice);   // 1 .. 8
    const int slice = ((K + blocks_k * KS - 1) / (blocks_k * KS) + 3) & ~3;
    const int chunk = KS * slice, wpitch = chunk + (chunk % 8 == 0 ? 4 : 0);   // an odd number of 16-byte pieces: lanes read without bank conflicts
    const size_t smem = sizeof(float) * (size_t)(MT * chunk + 32 * wpitch);
    static bool set = false;
    if (!set) { NCC_TRY(cudaFuncSetAttribute(rows_kernel<MT, KS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 208 * 1024)); set = true; }
    launch_clusters((unsigned)blocks_k, rows_kernel<MT, KS>, dim3((unsigned)((N + 31) / 32 * blocks_k), (unsigned)((M + MT - 1) / MT)), kWarps * 32,
                    smem, st, d, ldd, a, lda, b, ldb, bias, M, N, K, slice, wpitch, blocks_k, round_b ? 1 : 0, device_error_word());
    NCC_COUNT_LAUNCH();
    return launch_status("small_rows");
}

int small_rows(float* d, long long ldd, const float* a, long long lda, const float* b, long long ldb, const float* bias, int M, int N,
               int K, bool round_b, cudaStream_t st) {
    // bulk copies want 16-byte pieces; beyond eight blocks of a cluster the sum would need another level
    if (K % 4 == 0 && lda % 4 == 0 && ldb % 4 == 0 && al16(a) && al16(b) && K <= 8 * kWarps * kSlice && (M + 15) / 16 <= 65535) {
        if (M <= 1) return launch_rows<1, 8>(d, ldd, a, lda, b, ldb, bias, M, N, K, round_b, st);
        if (K < 256) return M <= 8 ? launch_rows<8, 1>(d, ldd, a, lda, b, ldb, bias, M, N, K, round_b, st)
                                   : launch_rows<16, 1>(d, ldd, a, lda, b, ldb, bias, M, N, K, round_b, st);
        if (K == 256) return M <= 8 ? launch_rows<8, 4>(d, ldd, a, lda, b, ldb, bias, M, N, K, round_b, st)
                                    : launch_rows<16, 4>(d, ldd, a, lda, b, ldb, bias, M, N, K, round_b, st);
        if (M <= 4) return launch_rows<4, 8>(d, ldd, a, lda, b, ldb, bias, M, N, K, round_b, st);
        if (M <= 8) return launch_rows<8, 8>(d, ldd, a, lda, b, ldb, bias, M, N, K, round_b, st);
        return launch_rows<16, 8>(d, ldd, a, lda, b, ldb, bias, M, N, K, round_b, st);
    }
    const long long row_tiles = (M + 7) / 8, groups = (N + 3) / 4;
    if (row_tiles > 65535) return set_status(NC_CUDA_ERR_UNSUPPORTED, "small_rows: %d rows", M);
    // slices of k inside a block: until about a dozen warps per SM exist, as long as a warp keeps a step
    const int steps = (K + 31) / 32;
    int ks_log2 = 0;
    while (ks_log2 < 3 && ((groups * row_tiles) << ks_log2) < (long long)sm_count() * 12 && (steps >> (ks_log2 + 1)) >= 1) ks_log2++;
    const dim3 grid((unsigned)((groups + (kWarps >> ks_log2) - 1) / (kWarps >> ks_log2)), (unsigned)row_tiles);
    launch(rows_odd_kernel, grid, kWarps * 32, 0, st, d, ldd, a, lda, b, ldb, bias, M, N, K, ks_log2, round_b ? 1 : 0);
    NCC_COUNT_LAUNCH();
    return launch_status("small_rows");
}

static void finish_job(ColumnsJob& j) {
    j.col_tiles = (j.C + 127) / 128;
    const int rows = j.K <= kShortK ? kWarps * kRT : kRT;
    j.blocks = j.d ? (int)((long long)((j.R + rows - 1) / rows) * j.col_tiles) : 0;
    j.vec = j.C % 4 == 0 && j.ldb % 4 == 0 && al16(j.b);
}
int small_columns(ColumnsJob j0, ColumnsJob j1, cudaStream_t st) {
    finish_job(j0);
    finish_job(j1);
    if (j0.blocks + j1.blocks == 0) return NC_CUDA_OK;
    launch(columns_kernel, j0.blocks + j1.blocks, kWarps * 32, 0, st, j0, j1);
    NCC_COUNT_LAUNCH();
    return launch_status("small_columns");
}

}  // namespace ncc
