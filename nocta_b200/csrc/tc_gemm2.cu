// TF32 GEMM on pairs of SMs (tcgen05, cta_group::2), sm_100a: D(M,N) = alpha * A * B^T + beta * D + bias, operands K-major or MN-major.
//
// Large products on one SM per tile (tc_gemm.cu) wait for operands: a 128 x 256 tile loads 48 KB of them per 512 cycles of MMA on
// every SM, and L2 delivers about 46 bytes per cycle and SM (4096 x 1024 outputs, K = 4096: 61 us, 12.9 TB/s).  Here a cluster of two
// CTAs owns a 256 x 256 tile: each loads 128 rows of A and 128 columns of B, 32 KB, and the pair's MMAs read both halves of B.
//
// Roles per CTA (192 threads): warp 0 issues its loads, warp 1 of the leading CTA (rank 0) issues the MMAs of both, warps 2 - 5 store
// the CTA's 128 rows of the accumulator (256 columns, double-buffered in tensor memory) while the next tile is multiplied.
// The loads of both CTAs report to the leader's barriers; the commits release ring slots and accumulators in both (only barrier
// arrivals go to both: every operand byte is loaded by the CTA that uses it).  An MN-major operand arrives as one 3-D box (32-wide
// chunks as the outermost dimension), so one thread keeps up with the issue; that wants an extent of whole chunks.
// Every wait is bounded as in tc_gemm.cu.
#include "tc_gemm.cuh"
#include "tc_ptx.cuh"
#include "../../include/nocta_cuda.h"

namespace tc {
namespace {

constexpr int kRows = 128;                       // rows of A and columns of B per CTA; the tile is twice that each way
constexpr int kHalfBytes = kRows * 32 * 4;       // one operand's part of a stage: 32 of the reduction
constexpr int kStageBytes = 2 * kHalfBytes;
constexpr int kStages = 6;
constexpr int kSmem = kStages * kStageBytes + 1024;
constexpr int kTmemCols = 512;                   // two accumulators of 256 columns
constexpr int kThreads2 = 192;

struct PairParams {
    int M, N, tiles_n, tiles, k_tiles;
    float* D;
    long long ldd;
    const float* bias;
    float alpha, beta;
    unsigned int* err;
};

__device__ __forceinline__ uint32_t on_rank(uint32_t local, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
__device__ __forceinline__ void arrive_remote(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// loads into this CTA's shared memory that report to a barrier of either CTA of the pair
__device__ __forceinline__ void pair_tma_2d(uint32_t dst, const CUtensorMap* tm, int c0, int c1, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tm)), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
__device__ __forceinline__ void pair_tma_3d(uint32_t dst, const CUtensorMap* tm, int c0, int c1, int c2, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tm)), "r"(c0), "r"(c1), "r"(c2), "r"(bar) : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate, uint32_t elected) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(elected) : "memory");
}
// arrival on the barrier at this offset in both CTAs once the MMAs issued so far are done
__device__ __forceinline__ void pair_commit(uint32_t bar, uint32_t elected) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t.reg .b16 m;\n\t"
        "setp.ne.b32 q, %1, 0;\n\t"
        "mov.b16 m, 3;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], m;\n\t}"
        ::"r"(bar), "r"(elected) : "memory");
}

template <bool A_MN, bool B_MN>
__global__ void __launch_bounds__(kThreads2, 1)
pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ PairParams p) {
    extern __shared__ uint8_t dyn_smem[];
    __shared__ __align__(8) uint64_t bar_full[kStages];     // used in the leader: both CTAs' halves of a stage have landed
    __shared__ __align__(8) uint64_t bar_empty[kStages];
    __shared__ __align__(8) uint64_t bar_acc_full[2];
    __shared__ __align__(8) uint64_t bar_acc_empty[2];      // used in the leader: one arrival per epilogue warp of the pair
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    __shared__ __align__(16) float turn[4][32][36];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = ncc::cluster_rank();
    const uint32_t base = (smem_u32(dyn_smem) + 1023u) & ~1023u;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; s++) { mbar_init(smem_u32(&bar_full[s]), 1); mbar_init(smem_u32(&bar_empty[s]), 1); }
        for (int b = 0; b < 2; b++) { mbar_init(smem_u32(&bar_acc_full[b]), 1); mbar_init(smem_u32(&bar_acc_empty[b]), 8); }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"((uint32_t)kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    __syncwarp();
    ncc::cluster_sync();   // the pair's barriers exist before either CTA reports to them
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    ncc::pdl_wait();
    volatile int* abortp = &abort_flag;
    const int first = blockIdx.x >> 1, step = gridDim.x >> 1;

    if (warp == 0) {
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int t = first; t < p.tiles && ok; t += step) {
                const int m0 = (t / p.tiles_n) * 2 * kRows + (int)rank * kRows, n0 = (t % p.tiles_n) * 2 * kRows + (int)rank * kRows;
                for (int kt = 0; kt < p.k_tiles; kt++) {
                    if (!mbar_wait(smem_u32(&bar_empty[s]), ph ^ 1u, p.err, 0x100u + s, abortp)) { ok = false; break; }
                    const uint32_t full = on_rank(smem_u32(&bar_full[s]), 0);
                    if (rank == 0) mbar_expect_tx(smem_u32(&bar_full[s]), 2u * kStageBytes);
                    const uint32_t a = base + (uint32_t)(s * kStageBytes), b = a + kHalfBytes;
                    if (A_MN) pair_tma_3d(a, &tmA, 0, kt * 32, m0 >> 5, full);
                    else pair_tma_2d(a, &tmA, kt * 32, m0, full);
                    if (B_MN) pair_tma_3d(b, &tmB, 0, kt * 32, n0 >> 5, full);
                    else pair_tma_2d(b, &tmB, kt * 32, n0, full);
                    if (++s == kStages) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            // the whole warp runs the loop (descriptors stay in uniform registers), lane 0 issues
            const uint32_t elected = lane == 0 ? 1u : 0u;
            const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((A_MN ? 1u : 0u) << 15) | ((B_MN ? 1u : 0u) << 16) |
                                   ((uint32_t)(2 * kRows >> 3) << 17) | ((uint32_t)(2 * kRows >> 4) << 24);
            // layouts as in tc_gemm.cu; each CTA's half lies at the same offset in its own shared memory
            const uint64_t da0 = smem_desc(base, A_MN ? 4096u : 16u, A_MN ? 512u : 1024u, A_MN ? 1u : 2u);
            const uint64_t db0 = smem_desc(base + kHalfBytes, B_MN ? 4096u : 16u, B_MN ? 512u : 1024u, B_MN ? 1u : 2u);
            const uint32_t ka = (A_MN ? 1024u : 32u) >> 4, kb = (B_MN ? 1024u : 32u) >> 4;
            int s = 0;
            uint32_t ph = 0, iter = 0;
            bool ok = true;
            for (int t = first; t < p.tiles && ok; t += step, iter++) {
                const uint32_t ab = iter & 1u;
                ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_acc_empty[ab]), ((iter >> 1) & 1u) ^ 1u, p.err, 0x500u + ab, abortp));
                if (!ok) break;
                tc_fence_after();
                for (int kt = 0; kt < p.k_tiles; kt++) {
                    ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_full[s]), ph, p.err, 0x200u + s, abortp));
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t off = (uint64_t)((uint32_t)(s * kStageBytes) >> 4);
#pragma unroll
                    for (int ks = 0; ks < 4; ks++)
                        pair_mma(tmem + ab * 256u, da0 + off + (uint64_t)(ks * ka), db0 + off + (uint64_t)(ks * kb), idesc, (uint32_t)(kt != 0 || ks != 0), elected);
                    pair_commit(smem_u32(&bar_empty[s]), elected);
                    if (++s == kStages) { s = 0; ph ^= 1u; }
                }
                if (ok) pair_commit(smem_u32(&bar_acc_full[ab]), elected);
            }
        }
    } else {
        const int q = warp & 3;   // TMEM lane quadrant this warp may read
        uint32_t iter = 0;
        bool ok = true;
        float (*blk)[36] = turn[q];
        const bool vec_ok = ((reinterpret_cast<uintptr_t>(p.D) & 15u) == 0) && (p.ldd & 3) == 0;
        for (int t = first; t < p.tiles && ok; t += step, iter++) {
            const int m0 = (t / p.tiles_n) * 2 * kRows + (int)rank * kRows + q * 32, n0 = (t % p.tiles_n) * 2 * kRows;
            const uint32_t ab = iter & 1u;
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_acc_full[ab]), (iter >> 1) & 1u, p.err, 0x400u + ab, abortp));
            if (!ok) break;
            tc_fence_after();
            const uint32_t acc = tmem + ab * 256u + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
            for (int c0 = 0; c0 < 2 * kRows; c0 += 32) {
                if (n0 + c0 >= p.N) break;
                uint32_t v[32];
                tmem_ld32(acc + (uint32_t)c0, v);
                tmem_ld_wait();
                // turned through shared memory: eight lanes store the 128 bytes of one row
#pragma unroll
                for (int j = 0; j < 32; j += 4)
                    *reinterpret_cast<float4*>(&blk[lane][j]) = make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]),
                                                                            __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
                __syncwarp();
                const int ncols = (p.N - (n0 + c0)) < 32 ? (p.N - (n0 + c0)) : 32;
                if (vec_ok && ncols == 32) {
                    const int cl = (lane & 7) * 4;
                    float4 b4 = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (p.bias) { const float* bp = p.bias + n0 + c0 + cl; b4 = make_float4(bp[0], bp[1], bp[2], bp[3]); }
#pragma unroll
                    for (int it = 0; it < 8; it++) {
                        const int row = it * 4 + (lane >> 3);
                        float4 o = *reinterpret_cast<const float4*>(&blk[row][cl]);
                        if (m0 + row >= p.M) continue;
                        float4* dst = reinterpret_cast<float4*>(p.D + (long long)(m0 + row) * p.ldd + n0 + c0 + cl);
                        o.x *= p.alpha; o.y *= p.alpha; o.z *= p.alpha; o.w *= p.alpha;
                        if (p.beta != 0.f) {
                            const float4 old = *dst;
                            o.x += p.beta * old.x; o.y += p.beta * old.y; o.z += p.beta * old.z; o.w += p.beta * old.w;
                        }
                        if (p.bias) { o.x += b4.x; o.y += b4.y; o.z += b4.z; o.w += b4.w; }
                        *dst = o;
                    }
                } else {
                    const float b1 = (p.bias && lane < ncols) ? p.bias[n0 + c0 + lane] : 0.f;
#pragma unroll 4
                    for (int row = 0; row < 32; row++) {
                        if (m0 + row >= p.M || lane >= ncols) continue;
                        float* dst = p.D + (long long)(m0 + row) * p.ldd + n0 + c0 + lane;
                        float o = p.alpha * blk[row][lane];
                        if (p.beta != 0.f) o += p.beta * *dst;
                        if (p.bias) o += b1;
                        *dst = o;
                    }
                }
                __syncwarp();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_remote(on_rank(smem_u32(&bar_acc_empty[ab]), 0));
        }
    }

    tc_fence_before();
    __syncthreads();
    if (abort_flag) {
        // a wait expired: copies in flight land before shared memory is given back
        const unsigned long long t0 = global_ns();
        while (global_ns() - t0 < 2000000ull) { }
    }
    __syncwarp();
    ncc::cluster_sync();   // neither CTA leaves while the other may still report to its barriers or read its operands
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)kTmemCols) : "memory");
    }
}

template <bool A_MN, bool B_MN>
int launch_pair(const CUtensorMap& ta, const CUtensorMap& tb, const PairParams& p, double flops, cudaStream_t st) {
    static bool set = false;
    if (!set) { NCC_TRY(cudaFuncSetAttribute(pair_kernel<A_MN, B_MN>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem)); set = true; }
    const int pairs = ncc::sm_count() / 2;
    {
        ncc::ProfScope prof(ncc::prof_role(), flops, st, true);
        ncc::launch_clusters(2, pair_kernel<A_MN, B_MN>, dim3((unsigned)(2 * (p.tiles < pairs ? p.tiles : pairs))), kThreads2, kSmem, st, ta, tb, p);
    }
    NCC_COUNT_LAUNCH();
    return ncc::launch_status("pair_kernel");
}

// 128 rows x 32 of the reduction per box
bool pair_map(CUtensorMap* tm, const float* X, int ld, bool mn, int outer, int K) {
    if (!mn) {
        unsigned long long dims[2] = {(unsigned long long)K, (unsigned long long)outer}, str[1] = {(unsigned long long)ld};
        unsigned box[2] = {32, kRows};
        return make_map(tm, X, 2, dims, str, box, false);
    }
    unsigned long long dims[3] = {32, (unsigned long long)K, (unsigned long long)(outer / 32)}, str[2] = {(unsigned long long)ld, 32};
    unsigned box[3] = {32, 32, kRows / 32};
    return make_map(tm, X, 3, dims, str, box, true);
}

}  // namespace

int gemm_pair(float* D, int ldd, const float* A, int lda, bool a_mn, const float* B, int ldb, bool b_mn, int M, int N, int K,
              const float* bias, float alpha, float beta, cudaStream_t st) {
    if ((a_mn && (M & 31)) || (b_mn && (N & 31))) return NC_CUDA_ERR_UNSUPPORTED;
    const long long tiles_m = (M + 2 * kRows - 1) / (2 * kRows), tiles_n = (N + 2 * kRows - 1) / (2 * kRows), tiles = tiles_m * tiles_n;
    if (tiles > 0x3fffffff) return NC_CUDA_ERR_UNSUPPORTED;
    CUtensorMap ta, tb;
    if (!pair_map(&ta, A, lda, a_mn, M, K) || !pair_map(&tb, B, ldb, b_mn, N, K)) return NC_CUDA_ERR_UNSUPPORTED;
    PairParams p = {};
    p.M = M; p.N = N; p.tiles_n = (int)tiles_n; p.tiles = (int)tiles; p.k_tiles = (K + 31) / 32;
    p.D = D; p.ldd = ldd; p.bias = bias; p.alpha = alpha; p.beta = beta;
    p.err = ncc::device_error_word();
    const double flops = 2.0 * M * (double)N * K;
    if (!a_mn && !b_mn) return launch_pair<false, false>(ta, tb, p, flops, st);
    if (!a_mn) return launch_pair<false, true>(ta, tb, p, flops, st);
    if (!b_mn) return launch_pair<true, false>(ta, tb, p, flops, st);
    return launch_pair<true, true>(ta, tb, p, flops, st);
}

}  // namespace tc
