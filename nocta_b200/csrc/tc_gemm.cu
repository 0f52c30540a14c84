// Tensor-core contractions for sm_100a: TMA-fed tcgen05.mma (kind::tf32) with the accumulator in
// tensor memory, written with inline PTX.  tc_kernel serves four problem kinds; the halo-resident convolution and
// weight-gradient kernels, which take the stride-1 filters up to 3 x 3, live in tc_conv.cu.
//
//   GEMM   D(M,N) = A * B^T        either operand K-major or MN-major in memory
//   CONV   channels-last implicit GEMM, stride 1: rows = 128 output pixels (a w x h x n box),
//          cols = output channels, reduction = (kh, kw, 32-channel chunk).  The activation tile of
//          one reduction step is ONE 4-D TMA box at shifted (w, h) coordinates; out-of-bounds
//          elements are zero-filled by TMA, which is the padding.  Used for forward and, with
//          flipped / channel-transposed weights, for dX.
//   CONVT  the same convolution with the operand roles swapped: rows = 128 output channels (the weight
//          tile is the A operand), cols = 256 output pixels (one 4-D TMA box is the B operand).  A
//          tcgen05.mma (kind::tf32, one CTA) takes max(N / 2, operand bytes / 128, about 46) cycles
//          whatever M is, so M = 128 with N >= 128 is the full-rate shape; with pixels on N that holds
//          for any channel count >= 128, while few channels on N (N = 64: 48 cycles) would not.
//          Strided layers: the forward box is a TMA box with traversal stride; the input gradient is one
//          stride-1 convolution per residue class of the input coordinates (ConvClass), all in one launch.
//   DW     weight gradient: rows = output channels, cols = (kh, kw, ci), reduction = 32-pixel
//          boxes; both operands MN-major; split over the reduction with an ordered second stage.
//
// The kernel multiplies TF32 operands as they lie in memory.  The accuracy modes are prepared in memory: operands rounded to
// nearest TF32, or for 3xTF32 split into two planes hi and lo (split_operand); a stage then holds both planes of both operands
// (read once for three products: with one product per stage the loads from L2, not the tensor cores, set the pace; VGG step at batch
// 64 2724 -> 2393 us together with the faster reduction below) and every k-step is lo * hi, hi * lo, hi * hi.  The tensor core's own
// accumulation, which truncates, is the largest error left in that mode (5e-8 of the result per addition of eight products when all
// have one sign: 1e-5 over K = 4096), so a segment is two reduction tiles long, and the epilogue warps add the segments in
// registers, rounding to nearest, while the next one is multiplied: 5e-7 for any K.
//
// CTA = 6 warps (kernels with an MN-major operand add up to five more TMA-issuing warps): warp 0 issues TMA, warp 1
// allocates TMEM and issues MMAs (one lane), warps 2-5 run the epilogue (tcgen05.ld -> registers -> global).
// Every mbarrier wait is bounded: on expiry the kernel records a code in the device error word,
// drains, frees its TMEM and returns.
//
// No cluster launch and no multicast anywhere: each CTA loads its own tiles.
#include "tc_gemm.cuh"
#include "tc_ptx.cuh"
#include "../../include/nocta_cuda.h"

namespace tc {

enum { KIND_GEMM = 0, KIND_CONV = 1, KIND_DW = 2, KIND_CONVT = 3 };

// One stride-1 convolution of a CONVT launch: taps, paddings, where its weights start, its output extent and where that lies
// in the output tensor (stride and offset per axis).
struct ConvClass {
    int kH, kW, pad_h, pad_w;
    int wrow0;               // first row of its packed weights
    int Ho, Wo, tiles_w, tiles_h;
    int oh0, ow0;            // output pixel (h, w) of the class = (oh0 + os * h, ow0 + os * w) of the tensor
    int tile0;               // first pixel tile
};
constexpr int kMaxClasses = 4;

struct TcParams {
    int kind;
    int M, N;              // logical output extent (store masks)
    int planes;            // 1, or 2 for split operands
    int segment;           // reduction tiles per segment (all of them unless SPLIT)
    int a_plane, b_plane;  // coordinate distance of the lo plane of A and B (rows, or images)
    int num_k_tiles;       // reduction tiles in total
    int k_tiles_per_split; // reduction tiles per blockIdx.z
    float* D;
    long long ldd;
    const float* bias;
    float alpha, beta;
    float* partial;        // non-null: raw accumulators go to partial[z][M][N]
    // pixel-box geometry (CONV: 128-pixel output box; DW: 32-pixel reduction box)
    int bw, bh, bn;
    int tiles_w, tiles_h;
    int Ho, Wo, Nimg;
    int kW, pad;
    int stride;            // CONVT, DW: pixel stride of the input box
    int cchunks;           // CONV: 32-channel chunks of the reduction channels
    int wrows;             // CONV: rows per (kh,kw) block of the packed weights (= output channels)
    int Cin;               // DW: input channels, padded to whole chunks (column index -> (shift, ci))
    int lbw, lbh;                  // CONVT: log2 of the pixel box width / height
    int tiles_m, tiles_n, splits;  // persistent tile walk
    int stages;                    // operand ring depth
    // CONVT
    int classes, os, Hout, Wout;   // residue classes; output pixel stride and tensor extent
    ConvClass cls[kMaxClasses];
    double* stat;                  // CONVT, non-null: per CTA and channel (sum, sum of squares) of the output it wrote, [gridDim.x][M][2]
    unsigned int* err;
    double flops;                  // host only: algorithmic FLOPs of the launch, for the profiling scope
};

// ------------------------------------------------------------------------------------------
// The kernel
// ------------------------------------------------------------------------------------------
constexpr int BM = 128;
constexpr int BK = 32;                 // 32 floats = one 128-byte swizzle row
constexpr int A_BYTES = BM * BK * 4;   // 16 KB
constexpr int CHUNK_BYTES = 32 * BK * 4;  // one 32 x 32 MN-major chunk: 4 KB
constexpr int kMaxStages = 8;
constexpr int kSmemBudget = 196 * 1024;  // one persistent CTA per SM

constexpr int kSegment = 2;             // reduction tiles per segment of a 3xTF32 product

template <int BN, bool SPLIT>
struct TileCfg {
    static constexpr int PLANES = SPLIT ? 2 : 1;
    static constexpr int B_BYTES = BN * BK * 4;
    static constexpr int B_AT = PLANES * A_BYTES;   // stage: the planes (hi, lo) of A, then those of B
    static constexpr int STAGE_BYTES = PLANES * (A_BYTES + B_BYTES);
    static constexpr int STAGES_RAW = kSmemBudget / STAGE_BYTES;
    static constexpr int STAGES = STAGES_RAW > kMaxStages ? kMaxStages : STAGES_RAW;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024;  // + alignment slack
    static constexpr int ACC_COLS = BN <= 64 ? 64 : (BN <= 128 ? 128 : 256);
    static constexpr int NBUF = 2;   // the epilogue of one tile (or segment) overlaps the MMAs of the next
    static constexpr int TMEM_COLS = ACC_COLS * NBUF;
    static_assert(TMEM_COLS <= 512, "tensor memory");
};

// MN-major operands arrive as one copy per 32-wide chunk (up to 12 per stage) and a thread spends on the
// order of a hundred cycles per copy it issues, so those kernels run extra producer warps (warps 6..,
// lane 0 each): up to two producers share the A chunks and up to four the B chunks, round-robin.  Every
// producer waits for the ring slot itself and arms the stage barrier with its own byte count.
template <bool A_MN, bool B_MN, int BN>
struct ProdCfg {
    static constexpr bool MULTI = A_MN || B_MN;
    static constexpr int NA_OWNERS = !MULTI ? 1 : (A_MN ? 2 : 1);
    static constexpr int NB_OWNERS = !MULTI ? 0 : (B_MN ? (BN / 32 < 4 ? BN / 32 : 4) : 1);
    static constexpr int NPROD = MULTI ? NA_OWNERS + NB_OWNERS : 1;
    static constexpr int THREADS = 192 + 32 * (NPROD - 1);
};

// What a CTA does for tile t of its walk
struct Tile {
    int m0, n_tile, z, kt_begin, kt_end, cls, px;   // cls, px: CONVT residue class and pixel tile within it
};
__device__ __forceinline__ Tile tile_of(const TcParams& p, int t) {
    Tile o;
    o.n_tile = t % p.tiles_n;
    const int r = t / p.tiles_n;
    o.m0 = (r % p.tiles_m) * BM;
    o.z = r / p.tiles_m;
    o.kt_begin = o.z * p.k_tiles_per_split;
    o.kt_end = o.kt_begin + p.k_tiles_per_split;
    if (o.kt_end > p.num_k_tiles) o.kt_end = p.num_k_tiles;
    o.cls = 0;
    o.px = o.n_tile;
    if (p.kind == KIND_CONVT) {
        while (o.cls + 1 < p.classes && o.n_tile >= p.cls[o.cls + 1].tile0) o.cls++;
        o.px = o.n_tile - p.cls[o.cls].tile0;
        o.kt_end = p.cls[o.cls].kH * p.cls[o.cls].kW * p.cchunks;   // never split
    }
    return o;
}

// reduction tiles of the segment that starts at kt
__device__ __forceinline__ int segment_tiles(const TcParams& p, const Tile& T, int kt) {
    return (T.kt_end - kt) < p.segment ? (T.kt_end - kt) : p.segment;
}

// SPLIT: operands in two planes, segments added in registers (3xTF32)
template <int BN, bool A_MN, bool B_MN, bool SPLIT>
__global__ void __launch_bounds__(ProdCfg<A_MN, B_MN, BN>::THREADS, 1)
tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ TcParams p) {
    using Cfg = TileCfg<BN, SPLIT>;
    constexpr int NBUF = Cfg::NBUF;
    const int STAGES = p.stages;
    extern __shared__ uint8_t dyn_smem[];
    __shared__ __align__(8) uint64_t bar_full[kMaxStages];
    __shared__ __align__(8) uint64_t bar_empty[kMaxStages];
    __shared__ __align__(8) uint64_t bar_acc_full[2];
    __shared__ __align__(8) uint64_t bar_acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    __shared__ __align__(16) float turn[4][32][36];   // per epilogue warp: a 32 x 32 block between accumulator and store

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t tiles_base = (smem_u32(dyn_smem) + 1023u) & ~1023u;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) {
            mbar_init(smem_u32(&bar_full[s]), (uint32_t)ProdCfg<A_MN, B_MN, BN>::NPROD);
            mbar_init(smem_u32(&bar_empty[s]), 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(smem_u32(&bar_acc_full[b]), 1);
            mbar_init(smem_u32(&bar_acc_empty[b]), 128);
        }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"((uint32_t)Cfg::TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot;
    ncc::pdl_wait();   // barriers and tensor memory are set up while the preceding kernel ends
    volatile int* abortp = &abort_flag;

    // Persistent CTA: walks output tiles t = blockIdx.x, blockIdx.x + gridDim.x, ...
    // t -> (n_tile fastest, then m_tile, then reduction split z).
    const int total_tiles = p.tiles_m * p.tiles_n * p.splits;

    if (ProdCfg<A_MN, B_MN, BN>::MULTI && (warp == 0 || warp >= 6)) {
        // ------------------------------ TMA producers (MN-major operands) ------------------------------
        if (lane == 0) {
            using PC = ProdCfg<A_MN, B_MN, BN>;
            const int me = warp == 0 ? 0 : warp - 5;  // producer index
            const bool forA = me < PC::NA_OWNERS;
            const int own = forA ? me : me - PC::NA_OWNERS;         // first chunk this producer owns
            const int step = forA ? PC::NA_OWNERS : PC::NB_OWNERS;  // and the stride to its next one
            constexpr int NACH = A_MN ? BM / 32 : 1;  // copies of operand A per stage
            constexpr int NBCH = B_MN ? BN / 32 : 1;  // copies of operand B per stage
            // 32-wide chunks that lie entirely beyond the matrix edge (rows >= M, columns >= N) are not copied at
            // all: their accumulator rows / columns are never stored, and skipping them saves issue slots and
            // shared-memory writes (Cout = 64 fills only two of the four A chunks).
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
                const Tile T = tile_of(p, t);
                const int m0 = T.m0, n0 = T.n_tile * BN;
                const int edge = forA ? p.M - m0 : p.N - n0;  // chunks starting at or beyond it are skipped
                int my_n = 0;                                 // copies this producer issues per stage of this tile
                for (int c = own; c < (forA ? NACH : NBCH); c += step) my_n += (32 * c < edge) ? 1 : 0;
                const bool chunked = forA ? A_MN : B_MN;
                const uint32_t my_bytes = Cfg::PLANES * (chunked ? (uint32_t)my_n * CHUNK_BYTES : (forA ? (uint32_t)A_BYTES : (uint32_t)Cfg::B_BYTES));
                int dtw = 0, dth = 0, dtn = 0;
                // DW: (first channel, tap) of this producer's B chunks
                int ci0[4] = {0, 0, 0, 0}, dkh[4] = {0, 0, 0, 0}, dkw[4] = {0, 0, 0, 0};
                if (p.kind == KIND_DW) {
                    dtw = T.kt_begin % p.tiles_w;
                    const int tt = T.kt_begin / p.tiles_w;
                    dth = tt % p.tiles_h; dtn = tt / p.tiles_h;
                    if (!forA) {
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const int col = n0 + 32 * (own + i * step);
                            const int sh = col / p.Cin;
                            ci0[i] = col - sh * p.Cin;
                            dkh[i] = sh / p.kW; dkw[i] = sh - dkh[i] * p.kW;
                        }
                    }
                }
                for (int kt = T.kt_begin; kt < T.kt_end; kt++) {
                    if (!mbar_wait(smem_u32(&bar_empty[s]), ph ^ 1u, p.err, 0x100u + s, abortp)) { ok = false; break; }
                    const uint32_t full = smem_u32(&bar_full[s]);
                    if (my_bytes == 0) {
                        mbar_arrive(full);
                    } else {
                        mbar_expect_tx(full, my_bytes);
#pragma unroll
                        for (int pl = 0; pl < Cfg::PLANES; pl++) {
                            const uint32_t a_dst = tiles_base + (uint32_t)s * Cfg::STAGE_BYTES + (uint32_t)(pl * A_BYTES);
                            const uint32_t b_dst = tiles_base + (uint32_t)s * Cfg::STAGE_BYTES + (uint32_t)(Cfg::B_AT + pl * Cfg::B_BYTES);
                            const int off = pl * (forA ? p.a_plane : p.b_plane);
                            if (p.kind == KIND_GEMM) {
                                const int k0 = kt * BK;
                                if (forA) {
                                    if (!A_MN) tma_2d(a_dst, &tmA, k0, m0 + off, full);
                                    else {
#pragma unroll
                                        for (int i = 0; i < 4; i++) {
                                            const int c = own + i * step;
                                            if (c < NACH && 32 * c < edge) tma_2d(a_dst + c * CHUNK_BYTES, &tmA, m0 + 32 * c, k0 + off, full);
                                        }
                                    }
                                } else if (!B_MN) {
                                    tma_2d(b_dst, &tmB, k0, n0 + off, full);
                                } else {
#pragma unroll
                                    for (int i = 0; i < 4; i++) {
                                        const int c = own + i * step;
                                        if (c < NBCH && 32 * c < edge) tma_2d(b_dst + c * CHUNK_BYTES, &tmB, n0 + 32 * c, k0 + off, full);
                                    }
                                }
                            } else {  // KIND_DW (both operands MN-major)
                                const int w0 = dtw * p.bw, h0 = dth * p.bh, nn0 = dtn * p.bn + off;
                                if (forA) {
#pragma unroll
                                    for (int i = 0; i < 4; i++) {
                                        const int c = own + i * step;
                                        if (c < NACH && 32 * c < edge) tma_4d(a_dst + c * CHUNK_BYTES, &tmA, m0 + 32 * c, w0, h0, nn0, full);
                                    }
                                } else {
#pragma unroll
                                    for (int i = 0; i < 4; i++) {
                                        const int c = own + i * step;
                                        if (c < NBCH && 32 * c < edge)
                                            tma_4d(b_dst + c * CHUNK_BYTES, &tmB, ci0[i], w0 * p.stride + dkw[i] - p.pad, h0 * p.stride + dkh[i] - p.pad, nn0, full);
                                    }
                                }
                            }
                        }
                    }
                    if (p.kind == KIND_DW) {
                        if (++dtw == p.tiles_w) { dtw = 0; if (++dth == p.tiles_h) { dth = 0; dtn++; } }
                    }
                    if (++s == STAGES) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 0) {
        // ------------------------------ TMA producer ------------------------------
        if (lane == 0) {
            // One thread feeds the whole CTA, so its loop is kept free of divisions and runtime modulo:
            // ring slot / phase, filter tap and channel chunk are running counters.
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
                const Tile T = tile_of(p, t);
                const int m0 = T.m0, n0 = T.n_tile * BN;
                // pixel box of this tile (CONV: the m tile, CONVT: the n tile), running (tap, chunk)
                int pw0 = 0, ph0 = 0, pn0 = 0, cc = 0, kh = 0, kw = 0, shift = 0, kWc = p.kW, wrow0 = 0;
                if (p.kind == KIND_CONV) {
                    const int pt = m0 / BM, tw = pt % p.tiles_w, tt = pt / p.tiles_w;
                    pw0 = tw * p.bw - p.pad; ph0 = (tt % p.tiles_h) * p.bh - p.pad; pn0 = (tt / p.tiles_h) * p.bn;
                } else if (p.kind == KIND_CONVT) {
                    const ConvClass& c = p.cls[T.cls];
                    const int tw = T.px % c.tiles_w, tt = T.px / c.tiles_w;
                    pw0 = tw * p.bw * p.stride - c.pad_w; ph0 = (tt % c.tiles_h) * p.bh * p.stride - c.pad_h; pn0 = (tt / c.tiles_h) * p.bn;
                    kWc = c.kW; wrow0 = c.wrow0;
                }
                for (int kt = T.kt_begin; kt < T.kt_end; kt++) {
                    if (!mbar_wait(smem_u32(&bar_empty[s]), ph ^ 1u, p.err, 0x100u + s, abortp)) { ok = false; break; }
                    const uint32_t full = smem_u32(&bar_full[s]);
                    mbar_expect_tx(full, (uint32_t)Cfg::STAGE_BYTES);
#pragma unroll
                    for (int pl = 0; pl < Cfg::PLANES; pl++) {
                        const uint32_t a_dst = tiles_base + (uint32_t)s * Cfg::STAGE_BYTES + (uint32_t)(pl * A_BYTES);
                        const uint32_t b_dst = tiles_base + (uint32_t)s * Cfg::STAGE_BYTES + (uint32_t)(Cfg::B_AT + pl * Cfg::B_BYTES);
                        const int offA = pl * p.a_plane, offB = pl * p.b_plane;
                        if (p.kind == KIND_GEMM) {
                            tma_2d(a_dst, &tmA, kt * BK, m0 + offA, full);
                            tma_2d(b_dst, &tmB, kt * BK, n0 + offB, full);
                        } else if (p.kind == KIND_CONV) {
                            tma_4d(a_dst, &tmA, cc * 32, pw0 + kw, ph0 + kh, pn0 + offA, full);
                            tma_2d(b_dst, &tmB, cc * 32, shift * p.wrows + n0 + offB, full);
                        } else {
                            tma_2d(a_dst, &tmA, cc * 32, wrow0 + shift * p.wrows + m0 + offA, full);
                            tma_4d(b_dst, &tmB, cc * 32, pw0 + kw, ph0 + kh, pn0 + offB, full);
                        }
                    }
                    if (p.kind != KIND_GEMM && ++cc == p.cchunks) {
                        cc = 0; shift++;
                        if (++kw == kWc) { kw = 0; kh++; }
                    }
                    if (++s == STAGES) { s = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer ------------------------------
        if (lane == 0) {
            // instruction descriptor: D = f32, A = B = tf32, majors, N, M = 128
            const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((A_MN ? 1u : 0u) << 15) | ((B_MN ? 1u : 0u) << 16) |
                                   ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
            // K-major: 8-row groups 1024 B apart (SBO); a k-step of 8 floats advances 32 B inside the swizzle row.
            // MN-major: rows are reduction indices, 128 B (32 elements of M/N) each; the swizzle atom is
            // 4 rows (SBO = 512 B between atoms along k), 32-element chunks are CHUNK_BYTES apart (LBO);
            // a k-step of 8 rows advances 1024 B.
            const uint32_t lbo_a = A_MN ? CHUNK_BYTES : 16u, sbo_a = A_MN ? 512u : 1024u;
            const uint32_t lbo_b = B_MN ? CHUNK_BYTES : 16u, sbo_b = B_MN ? 512u : 1024u;
            const uint32_t lay_a = A_MN ? 1u : 2u, lay_b = B_MN ? 1u : 2u;
            const uint32_t kstep_a = A_MN ? 1024u : 32u, kstep_b = B_MN ? 1024u : 32u;
            // descriptors are built once; a ring slot or k-step only moves the 14-bit start-address field
            const uint64_t da0 = smem_desc(tiles_base, lbo_a, sbo_a, lay_a);
            const uint64_t db0 = smem_desc(tiles_base + Cfg::B_AT, lbo_b, sbo_b, lay_b);
            int s = 0;
            uint32_t ph = 0, tile_iter = 0;
            bool ok = true;
            // A barrier test takes this thread well over a hundred cycles before its result can be used, about as long as
            // issuing two MMAs.  The state of the NEXT stage's barrier is therefore requested before this stage's MMAs
            // are issued and only looked at afterwards: with the producers ahead it is already set, and the wait at
            // the top of the next round is skipped.
            bool known_ready = false;
            for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
                const Tile T = tile_of(p, t);
                int kt = T.kt_begin;
                do {   // once also for a tile without reduction
                    const int nk = segment_tiles(p, T, kt);
                    const uint32_t ab = tile_iter % NBUF;
                    // wait until the epilogue has drained this accumulator buffer (first use passes at once)
                    if (!mbar_wait(smem_u32(&bar_acc_empty[ab]), ((tile_iter / NBUF) & 1u) ^ 1u, p.err, 0x500u + ab, abortp)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t acc = tmem_base + ab * (uint32_t)Cfg::ACC_COLS;
                    for (int i = 0; i < nk; i++) {
                        if (!known_ready && !mbar_wait(smem_u32(&bar_full[s]), ph, p.err, 0x200u + s, abortp)) { ok = false; break; }
                        tc_fence_after();
                        {
                            const int s1 = (s + 1 == STAGES) ? 0 : s + 1;
                            const uint32_t ph1 = (s + 1 == STAGES) ? (ph ^ 1u) : ph;
                            known_ready = mbar_test(smem_u32(&bar_full[s1]), ph1);
                        }
                        const uint64_t soff = (uint64_t)(((uint32_t)s * (uint32_t)Cfg::STAGE_BYTES) >> 4);
#pragma unroll
                        for (int ks = 0; ks < BK / 8; ks++) {
                            const uint64_t da = da0 + soff + (uint64_t)((ks * kstep_a) >> 4);
                            const uint64_t db = db0 + soff + (uint64_t)((ks * kstep_b) >> 4);
                            if (SPLIT) {
                                umma_tf32(acc, da + (uint64_t)(A_BYTES >> 4), db, idesc, (uint32_t)(i != 0 || ks != 0));
                                umma_tf32(acc, da, db + (uint64_t)(Cfg::B_BYTES >> 4), idesc, 1u);
                            }
                            umma_tf32(acc, da, db, idesc, (uint32_t)(SPLIT || i != 0 || ks != 0));
                        }
                        umma_commit(smem_u32(&bar_empty[s]));
                        if (++s == STAGES) { s = 0; ph ^= 1u; }
                    }
                    if (!ok) break;
                    umma_commit(smem_u32(&bar_acc_full[ab]));
                    tile_iter++;
                    kt += p.segment;
                } while (kt < T.kt_end);
            }
        }
    } else if (warp < 6) {
        // ------------------------------ epilogue warps ------------------------------
        const int q = warp & 3;           // TMEM lane quadrant this warp may read
        const int r = q * 32 + lane;
        uint32_t tile_iter = 0;
        bool ok = true;
        // CONVT output statistics: one running pair per channel tile, written once per CTA (see convh_kernel)
        double ssum = 0.0, ssq = 0.0;
        int stat_m0 = -1;
        if (p.kind == KIND_CONVT && p.stat)
            for (int mt = 0; mt < p.tiles_m; mt++)
                if (mt * BM + r < p.M) {
                    double* sd = p.stat + ((size_t)blockIdx.x * p.M + mt * BM + r) * 2;
                    sd[0] = 0.0; sd[1] = 0.0;
                }
        for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
            const Tile T = tile_of(p, t);
            const int m0 = T.m0, n0 = T.n_tile * BN;
            if (p.kind == KIND_CONVT && p.stat && m0 != stat_m0) {
                if (stat_m0 >= 0 && stat_m0 + r < p.M) {
                    double* sd = p.stat + ((size_t)blockIdx.x * p.M + stat_m0 + r) * 2;
                    sd[0] = ssum; sd[1] = ssq;
                }
                ssum = 0.0; ssq = 0.0; stat_m0 = m0;
            }
            constexpr int kChunks = SPLIT ? BN / 32 : 1;
            float sum[kChunks][32];
#pragma unroll
            for (int c = 0; c < kChunks; c++)
#pragma unroll
                for (int j = 0; j < 32; j++) sum[c][j] = 0.f;
            uint32_t acc_base = 0, ab = 0;
            int kt = T.kt_begin;
            do {
                ab = tile_iter % NBUF;
                ok = mbar_wait(smem_u32(&bar_acc_full[ab]), (tile_iter / NBUF) & 1u, p.err, 0x400u + ab, abortp);
                // all 32 lanes of a warp must agree before the aligned tcgen05.ld
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                acc_base = tmem_base + ab * (uint32_t)Cfg::ACC_COLS + ((uint32_t)(q * 32) << 16);
                tile_iter++;
                if (SPLIT) {
#pragma unroll
                    for (int c = 0; c < kChunks; c++) {
                        uint32_t u[32];
                        tmem_ld32(acc_base + (uint32_t)(c * 32), u);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 32; j++) sum[c][j] += __uint_as_float(u[j]);
                    }
                    tc_fence_before();
                    mbar_arrive(smem_u32(&bar_acc_empty[ab]));
                }
                kt += p.segment;
            } while (kt < T.kt_end);
            if (!ok) break;
            // 32 accumulator columns of this warp's rows; after the last chunk the buffer may be overwritten by the tile after next
            auto read_chunk = [&](int c0, bool last, uint32_t (&v)[32]) {
                if (SPLIT) {
#pragma unroll
                    for (int j = 0; j < 32; j++) {   // chunks are asked for in order and move up: registers want constant indexes
                        v[j] = __float_as_uint(sum[0][j]);
#pragma unroll
                        for (int c = 0; c + 1 < kChunks; c++) sum[c][j] = sum[c + 1][j];
                    }
                    return;
                }
                tmem_ld32(acc_base + (uint32_t)c0, v);
                tmem_ld_wait();
                if (last) {
                    tc_fence_before();
                    mbar_arrive(smem_u32(&bar_acc_empty[ab]));
                }
            };
            if (p.kind == KIND_CONVT) {
                // lane = output channel, column = pixel of the box; channels-last store: for one column the
                // 32 lanes of a warp write 32 consecutive floats
                const ConvClass& c = p.cls[T.cls];
                const int co = m0 + r;
                const bool co_ok = co < p.M;
                const float bv = (co_ok && p.bias) ? p.bias[co] : 0.f;
                const int tw = T.px % c.tiles_w, tt = T.px / c.tiles_w;
                const int pw0 = tw * p.bw, ph0 = (tt % c.tiles_h) * p.bh, pn0 = (tt / c.tiles_h) * p.bn;
                const bool none = T.kt_end == T.kt_begin;   // a residue class no tap reaches: zeros
                const int wstep = p.os * (int)p.ldd;        // between the class's neighbouring pixels of a row
#pragma unroll 1
                for (int c0 = 0; c0 < BN; c0 += 32) {
                    float fs = 0.f, fq = 0.f;  // output statistics over the pixels of this chunk that exist
                    uint32_t v[32];
                    read_chunk(c0, c0 + 32 >= BN, v);
                    if (none)
#pragma unroll
                        for (int j = 0; j < 32; j++) v[j] = 0u;
                    // the 32 columns of a chunk are runs of consecutive w inside one image row (a box is at least 8 wide): the
                    // 64-bit address is formed once per run, each store then adds a small constant multiple of the step
#pragma unroll
                    for (int j0 = 0; j0 < 32; j0 += 8) {
                        const int pj = c0 + j0;
                        const int w = pw0 + (pj & (p.bw - 1));
                        const int h = ph0 + ((pj >> p.lbw) & (p.bh - 1));
                        const int n = pn0 + (pj >> (p.lbw + p.lbh));
                        if (co_ok && h < c.Ho && n < p.Nimg) {
                            float* dst = p.D + (((long long)n * p.Hout + c.oh0 + p.os * h) * p.Wout + c.ow0 + p.os * w) * p.ldd + co;
                            const int lim = c.Wo - w;  // columns j < lim are inside the image
#pragma unroll
                            for (int j = 0; j < 8; j++)
                                if (j < lim) {
                                    const float o = __uint_as_float(v[j0 + j]) + bv;
                                    dst[j * wstep] = o;
                                    if (p.stat) { fs += o; fq = fmaf(o, o, fq); }
                                }
                        }
                    }
                    ssum += (double)fs;
                    ssq += (double)fq;
                }
                continue;
            }
            // where does this row go?
            long long row_off = -1;
            if (p.kind == KIND_CONV) {
                const int m_tile = m0 / BM, tw = m_tile % p.tiles_w, tt = m_tile / p.tiles_w;
                const int cw0 = tw * p.bw, ch0 = (tt % p.tiles_h) * p.bh, cn0 = (tt / p.tiles_h) * p.bn;
                const int iw = r % p.bw, t2 = r / p.bw, ih = t2 % p.bh, in_ = t2 / p.bh;
                const int w = cw0 + iw, h = ch0 + ih, n = cn0 + in_;
                if (w < p.Wo && h < p.Ho && n < p.Nimg) row_off = (((long long)n * p.Ho + h) * p.Wo + w) * p.ldd;
            } else {
                const int m = m0 + r;
                if (m < p.M) row_off = p.partial ? ((long long)T.z * p.M + m) * p.N : (long long)m * p.ldd;
            }
            float* base = p.partial ? p.partial : p.D;
            const bool vec_ok = ((reinterpret_cast<uintptr_t>(base) & 15u) == 0) &&
                                (((p.partial ? (long long)p.N : p.ldd) & 3) == 0);
            // A thread holds 32 columns of ONE row, and storing them as they are would make every store instruction touch 32
            // different lines: the block is turned through shared memory so that eight lanes store one row's 128 bytes.
            float (*blk)[36] = turn[q];
            const float alpha = p.partial ? 1.f : p.alpha, beta = p.partial ? 0.f : p.beta;
            const float* biasv = p.partial ? nullptr : p.bias;
#pragma unroll 1
            for (int c0 = 0; c0 < BN; c0 += 32) {
                if (n0 + c0 >= p.N) break;  // uniform across the CTA
                uint32_t v[32];
                read_chunk(c0, c0 + 32 >= BN || n0 + c0 + 32 >= p.N, v);
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 32; j += 4)
                    *reinterpret_cast<float4*>(&blk[lane][j]) = make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]),
                                                                            __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
                __syncwarp();
                const int ncols = (p.N - (n0 + c0)) < 32 ? (p.N - (n0 + c0)) : 32;
                if (vec_ok && ncols == 32) {
                    const int cl = (lane & 7) * 4;
                    float4 b4 = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (biasv) { const float* bp = biasv + n0 + c0 + cl; b4 = make_float4(bp[0], bp[1], bp[2], bp[3]); }
#pragma unroll
                    for (int it = 0; it < 8; it++) {
                        const int row = it * 4 + (lane >> 3);
                        const long long ro = __shfl_sync(0xffffffffu, row_off, row);
                        float4 o = *reinterpret_cast<const float4*>(&blk[row][cl]);
                        if (ro < 0) continue;
                        float4* dst = reinterpret_cast<float4*>(base + ro + n0 + c0 + cl);
                        o.x *= alpha; o.y *= alpha; o.z *= alpha; o.w *= alpha;
                        if (beta != 0.f) {
                            const float4 old = *dst;
                            o.x += beta * old.x; o.y += beta * old.y; o.z += beta * old.z; o.w += beta * old.w;
                        }
                        if (biasv) { o.x += b4.x; o.y += b4.y; o.z += b4.z; o.w += b4.w; }
                        *dst = o;
                    }
                } else {
                    const float b1 = (biasv && lane < ncols) ? biasv[n0 + c0 + lane] : 0.f;
#pragma unroll 4
                    for (int row = 0; row < 32; row++) {
                        const long long ro = __shfl_sync(0xffffffffu, row_off, row);
                        if (ro < 0 || lane >= ncols) continue;
                        float* dst = base + ro + n0 + c0 + lane;
                        float o = alpha * blk[row][lane];
                        if (beta != 0.f) o += beta * *dst;
                        if (biasv) o += b1;
                        *dst = o;
                    }
                }
            }
        }
        if (p.kind == KIND_CONVT && p.stat && stat_m0 >= 0 && stat_m0 + r < p.M) {
            double* sd = p.stat + ((size_t)blockIdx.x * p.M + stat_m0 + r) * 2;
            sd[0] = ssum; sd[1] = ssq;
        }
    }

    // ------------------------------ teardown ------------------------------
    tc_fence_before();
    __syncthreads();
    if (abort_flag) {
        // A wait expired somewhere: give copies still in flight time to land before the CTA's
        // shared memory is released.
        const unsigned long long t0 = global_ns();
        while (global_ns() - t0 < 2000000ull) { }
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)Cfg::TMEM_COLS) : "memory");
    }
}

// ------------------------------------------------------------------------------------------
// Operand preparation, second stages and weight packing
// ------------------------------------------------------------------------------------------
// dst plane 0 = src rounded to nearest TF32; plane 1 (when there are two) = the rounded remainder.  Rows of ld_dst floats (a multiple
// of four, 16-byte aligned), zeros where dst is larger than src: also turns operands TMA cannot describe (odd leading dimensions,
// misaligned bases) into ones it can.
template <bool VEC>
__global__ void __launch_bounds__(256) split_operand_kernel(float* __restrict__ dst, const float* __restrict__ src, size_t rows, int cols,
                                                            size_t ld_src, size_t rows_dst, int ld_dst, int planes) {
    ncc::pdl_wait();
    const int q4 = ld_dst >> 2;
    const size_t total = rows_dst * q4, plane = rows_dst * (size_t)ld_dst, stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const size_t r = i / q4;
        const int c = (int)(i - r * q4) * 4;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (r < rows) {
            const float* s = src + r * ld_src + c;
            if (VEC && c + 4 <= cols) {
                const float4 t = *reinterpret_cast<const float4*>(s);
                v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
            } else {
#pragma unroll
                for (int e = 0; e < 4; e++) if (c + e < cols) v[e] = s[e];
            }
        }
        float h[4];
#pragma unroll
        for (int e = 0; e < 4; e++) h[e] = ncc::round_tf32(v[e]);
        *reinterpret_cast<float4*>(dst + r * ld_dst + c) = make_float4(h[0], h[1], h[2], h[3]);
        if (planes == 2)
            *reinterpret_cast<float4*>(dst + plane + r * ld_dst + c) =
                make_float4(ncc::round_tf32(v[0] - h[0]), ncc::round_tf32(v[1] - h[1]), ncc::round_tf32(v[2] - h[2]), ncc::round_tf32(v[3] - h[3]));
    }
}
// scratch copy of an operand; rows_dst >= rows.  nullptr: no memory (status set)
static float* split_operand(int slot, const float* src, size_t rows, int cols, size_t ld_src, size_t rows_dst, int ld_dst, int planes,
                            cudaStream_t st) {
    float* dst = (float*)ncc::scratch(slot, sizeof(float) * rows_dst * ld_dst * planes, st);
    if (!dst) return nullptr;
    const bool vec = ld_src % 4 == 0 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0;
    const int grid = ncc::grid_for((long long)(rows_dst * (ld_dst / 4)), 256);
    if (vec) ncc::launch(split_operand_kernel<true>, grid, 256, 0, st, dst, src, rows, cols, ld_src, rows_dst, ld_dst, planes);
    else ncc::launch(split_operand_kernel<false>, grid, 256, 0, st, dst, src, rows, cols, ld_src, rows_dst, ld_dst, planes);
    NCC_COUNT_LAUNCH();
    return ncc::launch_status("split_operand") == NC_CUDA_OK ? dst : nullptr;
}
constexpr int kSlotA = 10, kSlotB = 11;
int mode_planes(int mode) { return mode == NC_CUDA_MATH_3XTF32 ? 2 : 1; }
// a dense channels-last activation as the math mode wants it: itself (TF32), rounded (RNA), hi and lo planes N images apart (3xTF32)
static const float* split_pixels(int slot, const float* x, size_t pixels, int C, int mode, cudaStream_t st) {
    return mode == NC_CUDA_MATH_TF32 ? x : split_operand(slot, x, pixels, C, (size_t)C, pixels, C, mode_planes(mode), st);
}

// Sum of element i over the planes of `partial`, `plane` floats apart: in double, in order.  Eight loads are requested before the
// first one is added.
__device__ __forceinline__ double sum_planes(const float* __restrict__ p, int splits, size_t plane) {
    double acc = 0.0;
    int z = 0;
    for (; z + 8 <= splits; z += 8) {
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = p[(size_t)(z + k) * plane];
#pragma unroll
        for (int k = 0; k < 8; k++) acc += (double)v[k];
    }
    for (; z < splits; z++) acc += (double)p[(size_t)z * plane];
    return acc;
}
__global__ void __launch_bounds__(256) splitk_reduce_kernel(float* __restrict__ D, long long ldd, const float* __restrict__ partial,
                                                            int splits, int M, int N, const float* __restrict__ bias,
                                                            float alpha, float beta) {
    ncc::pdl_wait();
    const size_t total = (size_t)M * N, stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const double acc = sum_planes(partial + i, splits, total);
        size_t m; int n;
        if (total <= 0xffffffffu) { const uint32_t q = (uint32_t)i / (uint32_t)N; m = q; n = (int)((uint32_t)i - q * (uint32_t)N); }   // a 64-bit division is ten times the work
        else { m = i / N; n = (int)(i % N); }
        float* d = D + m * ldd + n;
        float o = alpha * (float)acc;
        if (beta != 0.f) o += beta * *d;
        if (bias) o += bias[n];
        *d = o;
    }
}

// partial[z][co][(kh*kW+kw)*Cp + ci]  ->  dW[co][ci][kh][kw], Cp = Cin padded to whole 32-channel chunks.  A warp takes 32 elements of
// one run of planes, so reads are whole 128-byte lines of every plane; G warps share the planes of their elements in equal runs, added
// in order.  G = 8 from 64 planes on, where few weights leave the chip idle otherwise (64 -> 64 channels, 592 planes: one element per
// thread left 144 blocks, 50 us); with fewer planes a warp has too little to do between the barriers (256 -> 256 channels, 12 planes:
// 20 us with eight warps, 9 with one).  Only the single write per element is scattered.
template <int G>
__global__ void __launch_bounds__(256) dw_reduce_kernel(float* __restrict__ dW, const float* __restrict__ partial, int splits,
                                                        int Cout, int Cin, int Cp, int T) {
    ncc::pdl_wait();
    __shared__ double part[G][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = warp % G;
    const size_t total = (size_t)Cout * Cp * T;   // a multiple of 32
    const int per = (splits + G - 1) / G, z0 = g * per < splits ? g * per : splits, zn = (splits - z0) < per ? (splits - z0) : per;
    constexpr size_t kBlock = 32 * 8 / G;         // elements of a block
    for (size_t base = blockIdx.x * kBlock; base < total; base += gridDim.x * kBlock) {
        const size_t at = base + (size_t)(warp / G) * 32;
        double acc = at < total ? sum_planes(partial + (size_t)z0 * total + at + lane, zn, total) : 0.0;
        if (G > 1) {
            part[g][lane] = acc;
            __syncthreads();
            if (g == 0) {
                acc = 0.0;
#pragma unroll
                for (int w = 0; w < G; w++) acc += part[w][lane];
            }
        }
        const size_t r = at / (unsigned)Cp, co = r / (unsigned)T;
        const int ci = (int)(at - r * Cp) + lane, tap = (int)(r - co * T);
        if (g == 0 && at < total && ci < Cin) dW[(co * Cin + ci) * T + tap] = (float)acc;
        if (G > 1) __syncthreads();
    }
}

// dst[plane][tap][out][in], `in` the channels of the reduction.  DX: out = ci, in = co.  Tap t takes filter position t, counted from
// the end for DX; for strided layers (at most 64 taps) position at[t].
struct TapOrder { int listed; unsigned char at[64]; };
template <bool DX>
__global__ void __launch_bounds__(256) pack_weights_kernel(float* __restrict__ wp, const float* __restrict__ w, int Cout, int Cin,
                                                           int T, const __grid_constant__ TapOrder order, int round, int planes) {
    ncc::pdl_wait();
    const size_t total = (size_t)Cout * Cin * T, stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        size_t r = i;
        int co, ci;
        if (!DX) { ci = r % Cin; r /= Cin; co = r % Cout; r /= Cout; }
        else { co = r % Cout; r /= Cout; ci = r % Cin; r /= Cin; }
        const int tap = order.listed ? order.at[r] : (DX ? T - 1 - (int)r : (int)r);
        const float v = w[((size_t)co * Cin + ci) * T + tap];
        const float h = round ? ncc::round_tf32(v) : v;
        wp[i] = h;
        if (planes == 2) wp[total + i] = ncc::round_tf32(v - h);
    }
}

// ------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------
template <int BN, bool A_MN, bool B_MN, bool SPLIT>
static int launch_one(const CUtensorMap& ta, const CUtensorMap& tb, const TcParams& p_in, dim3 tiles, cudaStream_t st) {
    using Cfg = TileCfg<BN, SPLIT>;
    TcParams p = p_in;
    p.segment = SPLIT ? kSegment : 0x40000000;
    p.tiles_n = (int)tiles.x; p.tiles_m = (int)tiles.y; p.splits = (int)tiles.z;
    p.stages = Cfg::STAGES;
    const long long total = (long long)tiles.x * tiles.y * tiles.z;
    const int sms = ncc::sm_count();
    dim3 grid((unsigned)(total < sms ? total : sms), 1, 1);
    static bool attr_set = false;
    auto kern = tc_kernel<BN, A_MN, B_MN, SPLIT>;
    if (!attr_set) {
        NCC_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
        attr_set = true;
    }
    {
        ncc::ProfScope prof(ncc::prof_role(), p.flops, st, true);
        ncc::launch(kern, grid, ProdCfg<A_MN, B_MN, BN>::THREADS, Cfg::SMEM_BYTES, st, ta, tb, p);
    }
    NCC_COUNT_LAUNCH();
    return ncc::launch_status("tc_kernel");
}

template <bool A_MN, bool B_MN>
static int launch_bn(int bn, const CUtensorMap& ta, const CUtensorMap& tb, const TcParams& p, dim3 grid, cudaStream_t st) {
    const bool split = p.planes == 2;
    switch (bn) {
        case 64: return split ? launch_one<64, A_MN, B_MN, true>(ta, tb, p, grid, st) : launch_one<64, A_MN, B_MN, false>(ta, tb, p, grid, st);
        case 128: return split ? launch_one<128, A_MN, B_MN, true>(ta, tb, p, grid, st) : launch_one<128, A_MN, B_MN, false>(ta, tb, p, grid, st);
        case 256: return launch_one<256, A_MN, B_MN, false>(ta, tb, p, grid, st);
    }
    return ncc::set_status(NC_CUDA_ERR_ARG, "tc: unsupported tile width %d", bn);
}

// sums kept in registers fit for up to 128 columns
static int pick_bn(int N, bool split) { return N <= 64 ? 64 : ((N <= 128 || split) ? 128 : 256); }

// splits over the reduction so that about one wave of CTAs exists; each split keeps >= 4 tiles
static void pick_splits(int tiles, int nk, int* splits, int* kps) {
    int s = 1;
    const int sms = ncc::sm_count();
    if (tiles * 2 <= sms && nk >= 8) {
        s = sms / tiles;
        if (s > nk / 4) s = nk / 4;
        if (s < 1) s = 1;
    }
    int per = (nk + s - 1) / s;
    *kps = per;
    *splits = (nk + per - 1) / per;
}

// cycles of one reduction tile with bn columns: four k-steps of MMA (max(N / 2, operand bytes / 128, 46) cycles each, three of them for
// split operands), or its loads at the 70 bytes per cycle that an SM gets of L2 when all of them load
static double tile_cycles(int bn, int planes) {
    const double mma = 4.0 * (bn / 2 > (BM + bn) / 4 ? bn / 2 : ((BM + bn) / 4 > 46 ? (BM + bn) / 4 : 46)) * (planes == 2 ? 3 : 1);
    const double load = (BM + bn) * 128.0 * planes / 70.0;
    return mma > load ? mma : load;
}
// Columns per tile and splits of a product.  Wide tiles split until about one wave of CTAs exists are right where the reduction is
// long; otherwise the second kernel of a split costs more (about 5000 cycles and the partial sums' traffic) than narrower tiles lose.
// They are taken where the estimate is at least 15 % lower: 1001 x 1250 outputs, K = 310: two splits of 40 tiles -> 80 tiles of 128
// columns; 1001 x 310, K = 1250: nine splits -> three of 64 columns.
static void pick_tile(int M, int N, int nk, int planes, int* bn, int* splits, int* kps) {
    const int sms = ncc::sm_count(), rows = (M + BM - 1) / BM;
    auto cost = [&](int b, int s, int per) {
        const long long ctas = (long long)rows * ((N + b - 1) / b) * s, waves = (ctas + sms - 1) / sms;
        return (double)waves * (per * tile_cycles(b, planes) + 600.0) + 2000.0 + 8.0 * b + (s > 1 ? 5000.0 + (double)s * M * N * 8.0 / 3500.0 : 0.0);
    };
    *bn = pick_bn(N, planes == 2);
    pick_splits(rows * ((N + *bn - 1) / *bn), nk, splits, kps);
    double best = 0.85 * cost(*bn, *splits, *kps);
    for (int b = *bn; b >= 64; b /= 2) {
        int s, per;
        pick_splits(rows * ((N + b - 1) / b), nk, &s, &per);
        if (cost(b, s, per) < best) { best = cost(b, s, per); *bn = b; *splits = s; *kps = per; }
        if (s > 1 && cost(b, 1, nk) < best) { best = cost(b, 1, nk); *bn = b; *splits = 1; *kps = nk; }
    }
}

// Rows beyond M inside the 128-row tile are zero-filled by TMA and never stored; small products stay on CUDA cores.  Operands whose
// rows are no whole 16-byte pieces cost a copy each first: from 2^24 multiply-adds on.
bool gemm_eligible(int M, int N, int K, bool aligned) {
    return M >= 32 && N >= 16 && K >= 32 && (long long)M * N * K >= (aligned ? 1ll << 22 : 1ll << 24);
}

// Whether a product that fills the chip without splitting its reduction runs on pairs of SMs (tc_gemm2.cu): as long as tiles twice the
// height take no more waves.  Residual MLP step at batch 4096 (24 products of 34 GFLOP) 2350 -> 2196 us, 500 -> 560 TFLOP/s a product;
// the sustained TF32 rate of the chip, half of bf16's, is 683.
static bool pair_wins(int M, int N, int K) {
    const long long sms = ncc::sm_count();
    const long long one = ((M + BM - 1) / BM) * (long long)((N + 255) / 256), two = ((M + 255) / 256) * (long long)((N + 255) / 256);
    const long long waves1 = (one + sms - 1) / sms, waves2 = (two + sms / 2 - 1) / (sms / 2);
    return K >= 128 && waves2 <= waves1;
}

int gemm(float* D, int ldd, const float* A, int lda, bool a_mn, const float* B, int ldb, bool b_mn, int M, int N, int K,
         const float* bias, float alpha, float beta, int mode, cudaStream_t st) {
    const bool a_ok = !(lda & 3) && !(reinterpret_cast<uintptr_t>(A) & 15u), b_ok = !(ldb & 3) && !(reinterpret_cast<uintptr_t>(B) & 15u);
    if (!gemm_eligible(M, N, K, a_ok && b_ok)) return NC_CUDA_ERR_UNSUPPORTED;
    const int planes = mode_planes(mode), k_rows = planes == 2 ? (K + BK - 1) / BK * BK : K;
    // the reduction ends at K: along a row the tensor map's extent says so, along the rows of a split MN-major operand zeros do
    auto prepare = [&](int slot, const float*& X, int& ld, bool mn, int outer, bool ok) {
        if (mode == NC_CUDA_MATH_TF32 && ok) return true;
        const int rows = mn ? K : outer, cols = mn ? outer : K, ldp = (cols + 3) & ~3;
        const float* c = split_operand(slot, X, (size_t)rows, cols, (size_t)ld, (size_t)(mn ? k_rows : outer), ldp, planes, st);
        if (!c) return false;
        X = c; ld = ldp;
        return true;
    };
    if (!prepare(kSlotA, A, lda, a_mn, M, a_ok) || !prepare(kSlotB, B, ldb, b_mn, N, b_ok)) return NC_CUDA_ERR_RUNTIME;
    int bn, splits, kps;
    pick_tile(M, N, (K + BK - 1) / BK, planes, &bn, &splits, &kps);
    CUtensorMap ta, tb;
    {
        unsigned long long dims[2], str[1];
        unsigned box[2];
        if (!a_mn) { dims[0] = K; dims[1] = (unsigned long long)M * planes; str[0] = lda; box[0] = 32; box[1] = 128; }
        else       { dims[0] = M; dims[1] = (unsigned long long)k_rows * planes; str[0] = lda; box[0] = 32; box[1] = 32; }
        if (!make_map(&ta, A, 2, dims, str, box, a_mn)) return NC_CUDA_ERR_UNSUPPORTED;
        if (!b_mn) { dims[0] = K; dims[1] = (unsigned long long)N * planes; str[0] = ldb; box[0] = 32; box[1] = (unsigned)bn; }
        else       { dims[0] = N; dims[1] = (unsigned long long)k_rows * planes; str[0] = ldb; box[0] = 32; box[1] = 32; }
        if (!make_map(&tb, B, 2, dims, str, box, b_mn)) return NC_CUDA_ERR_UNSUPPORTED;
    }
    TcParams p = {};
    p.kind = KIND_GEMM;
    p.M = M; p.N = N;
    p.planes = planes;
    p.num_k_tiles = (K + BK - 1) / BK;
    p.a_plane = a_mn ? k_rows : M; p.b_plane = b_mn ? k_rows : N;
    p.D = D; p.ldd = ldd; p.bias = bias; p.alpha = alpha; p.beta = beta;
    p.err = ncc::device_error_word();
    const int tiles_m = (M + BM - 1) / BM, tiles_n = (N + bn - 1) / bn;
    if (planes == 1 && splits == 1 && bn == 256 && pair_wins(M, N, K)) {
        const int rc = gemm_pair(D, ldd, A, lda, a_mn, B, ldb, b_mn, M, N, K, bias, alpha, beta, st);
        if (rc != NC_CUDA_ERR_UNSUPPORTED) return rc;
    }
    p.k_tiles_per_split = kps;
    if (splits > 1) {
        p.partial = (float*)ncc::scratch(2, sizeof(float) * (size_t)splits * M * N, st);
        if (!p.partial) return NC_CUDA_ERR_RUNTIME;
    }
    dim3 grid(tiles_n, tiles_m, splits);
    p.flops = 2.0 * M * (double)N * K;
    int rc;
    if (!a_mn && !b_mn) rc = launch_bn<false, false>(bn, ta, tb, p, grid, st);
    else if (!a_mn && b_mn) rc = launch_bn<false, true>(bn, ta, tb, p, grid, st);
    else if (a_mn && !b_mn) rc = launch_bn<true, false>(bn, ta, tb, p, grid, st);
    else rc = launch_bn<true, true>(bn, ta, tb, p, grid, st);
    if (rc) return rc;
    if (splits > 1) {
        ncc::launch(splitk_reduce_kernel, ncc::grid_for((long long)M * N, 256), 256, 0, st, D, ldd, p.partial, splits, M, N, bias, alpha, beta);
        NCC_COUNT_LAUNCH();
        return ncc::launch_status("splitk_reduce");
    }
    return NC_CUDA_OK;
}

// Pixel box (bw, bh, bn) with bw*bh*bn == pixels that wastes the fewest rows for this image size.
static void pick_box(int pixels, int Wd, int Hd, int Nd, int* bw, int* bh, int* bn, int min_w = 1, int max_side = 256, bool whole_images = false) {
    long long best = -1;
    for (int w = min_w; w <= pixels; w *= 2)
        for (int h = 1; w * h <= pixels; h *= 2) {
            int n = pixels / (w * h);
            if (w * h * n != pixels || w > max_side || h > max_side || n > 256 || (whole_images && Nd % n)) continue;
            long long cover = (long long)((Wd + w - 1) / w) * w * ((Hd + h - 1) / h) * h * ((Nd + n - 1) / n) * n;
            // prefer less waste, then wider rows (longer contiguous runs), then fewer images per box
            if (best < 0 || cover < best || (cover == best && (w > *bw || (w == *bw && n < *bn)))) {
                best = cover; *bw = w; *bh = h; *bn = n;
            }
        }
}

bool conv_eligible(int Cin, int Cout, long long pixels) {
    return !(Cin & 3) && !(Cout & 3) && Cin >= 16 && Cout >= 16 && pixels >= 128;
}

// CONVT launch: the given classes over x (N,H,W,Cin) with input pixel stride `stride`, into y (N,Hout,Wout,Cout) with output pixel
// stride `os`.  xs: x as split_pixels made it.
static int convt_launch(float* y, int Hout, int Wout, int os, const float* xs, const float* wpacked, long long wrows_total, const float* bias,
                        int N, int H, int W, int Cin, int Cout, int stride, ConvClass* cls, int classes, int mode, bool want_stats,
                        double flops, cudaStream_t st) {
    const int planes = mode_planes(mode);
    int mh = 0, mw = 0;
    for (int i = 0; i < classes; i++) { mh = cls[i].Ho > mh ? cls[i].Ho : mh; mw = cls[i].Wo > mw ? cls[i].Wo : mw; }
    int bw = 1, bh = 1, bnn = 1;
    // Pixels per tile: 128 where twice the tiles are done sooner, as for the low images at the end of a network (37 images of 22 x 22:
    // 60 tiles of 256 on 148 SMs, 27 us), else 256, but for 3xTF32, which keeps its sums in registers.
    auto waves = [&](int px) {
        pick_box(px, mw, mh, N, &bw, &bh, &bnn, 8, 256 / stride);
        long long t = 0;
        for (int i = 0; i < classes; i++) t += (long long)((cls[i].Wo + bw - 1) / bw) * ((cls[i].Ho + bh - 1) / bh) * ((N + bnn - 1) / bnn);
        t *= (Cout + BM - 1) / BM;
        return (double)((t + ncc::sm_count() - 1) / ncc::sm_count());
    };
    const int px = planes == 2 || waves(128) * tile_cycles(128, 1) < waves(256) * tile_cycles(256, 1) ? 128 : 256;
    pick_box(px, mw, mh, N, &bw, &bh, &bnn, 8, 256 / stride);
    CUtensorMap ta, tb;
    unsigned long long wd[2] = {(unsigned long long)Cin, (unsigned long long)wrows_total * planes};
    unsigned long long ws[1] = {(unsigned long long)Cin};
    unsigned wb[2] = {32, 128};
    if (!make_map(&ta, wpacked, 2, wd, ws, wb, false)) return NC_CUDA_ERR_UNSUPPORTED;
    unsigned long long dims[4] = {(unsigned long long)Cin, (unsigned long long)W, (unsigned long long)H, (unsigned long long)N * planes};
    unsigned long long str[3] = {(unsigned long long)Cin, (unsigned long long)W * Cin, (unsigned long long)H * W * Cin};
    unsigned box[4] = {32, (unsigned)bw, (unsigned)bh, (unsigned)bnn};
    if (!make_map(&tb, xs, 4, dims, str, box, false, stride)) return NC_CUDA_ERR_UNSUPPORTED;
    TcParams p = {};
    p.kind = KIND_CONVT;
    p.M = Cout;
    p.cchunks = (Cin + 31) / 32;
    p.planes = planes;
    p.a_plane = (int)wrows_total; p.b_plane = N;
    p.D = y; p.ldd = Cout; p.bias = bias; p.alpha = 1.f; p.beta = 0.f;
    p.bw = bw; p.bh = bh; p.bn = bnn;
    for (p.lbw = 0; (1 << p.lbw) < bw; p.lbw++) {}
    for (p.lbh = 0; (1 << p.lbh) < bh; p.lbh++) {}
    p.Nimg = N;
    p.stride = stride; p.wrows = Cout;
    p.classes = classes; p.os = os; p.Hout = Hout; p.Wout = Wout;
    p.err = ncc::device_error_word();
    long long tiles_px = 0;
    for (int i = 0; i < classes; i++) {
        cls[i].tiles_w = (cls[i].Wo + bw - 1) / bw; cls[i].tiles_h = (cls[i].Ho + bh - 1) / bh;
        cls[i].tile0 = (int)tiles_px;
        tiles_px += (long long)cls[i].tiles_w * cls[i].tiles_h * ((N + bnn - 1) / bnn);
        p.cls[i] = cls[i];
    }
    if (tiles_px > (1ll << 30)) return NC_CUDA_ERR_UNSUPPORTED;
    p.N = 0x7fffffff;
    p.k_tiles_per_split = p.num_k_tiles = 1;   // per class, see tile_of
    dim3 tiles((unsigned)tiles_px, (unsigned)((Cout + BM - 1) / BM), 1);
    p.flops = flops;
    // launch_one uses min(tiles, SMs) persistent CTAs: one statistics slab per CTA
    const long long total_tiles = (long long)tiles.x * tiles.y;
    const int n_ctas = (int)(total_tiles < ncc::sm_count() ? total_tiles : ncc::sm_count());
    if (want_stats) p.stat = ncc::conv_stats_buffer((size_t)n_ctas, Cout, st);
    const int rc = launch_bn<false, false>(px, ta, tb, p, tiles, st);
    if (rc == NC_CUDA_OK && p.stat) ncc::conv_stats_publish(y, Cout, (long long)N * Hout * Wout, n_ctas, p.stat);
    return rc;
}

int conv_nhwc(float* y, const float* x, const float* wpacked, const float* bias, int N, int H, int W, int Cin, int Cout,
              int kH, int kW, int pad, int mode, cudaStream_t st) {
    const int Ho = H + 2 * pad - kH + 1, Wo = W + 2 * pad - kW + 1;
    if (Ho <= 0 || Wo <= 0) return NC_CUDA_ERR_UNSUPPORTED;
    if (!conv_eligible(Cin, Cout, (long long)N * Ho * Wo)) return NC_CUDA_ERR_UNSUPPORTED;
    const float* xs = split_pixels(kSlotA, x, (size_t)N * H * W, Cin, mode, st);
    if (!xs) return NC_CUDA_ERR_RUNTIME;
    const int planes = mode_planes(mode);
    {
        const int rc = conv_halo_nhwc(y, xs, wpacked, bias, N, H, W, Cin, Cout, kH, kW, pad, planes, st);
        if (rc != NC_CUDA_ERR_UNSUPPORTED) return rc;
    }
    const double flops = 2.0 * N * Ho * Wo * (double)Cout * Cin * kH * kW;
    if ((long long)N * Ho * Wo >= 1024 && kH * kW * Cout >= 128) {
        // pixels on the N side (256 per tile), channels on the M side
        ConvClass c = {};
        c.kH = kH; c.kW = kW; c.pad_h = c.pad_w = pad; c.Ho = Ho; c.Wo = Wo;
        return convt_launch(y, Ho, Wo, 1, xs, wpacked, (long long)kH * kW * Cout, bias, N, H, W, Cin, Cout, 1, &c, 1, mode, ncc::conv_stats_wanted(), flops, st);
    }
    const int bn_cols = pick_bn(Cout, planes == 2);
    int bw = 1, bh = 1, bnn = 1;
    pick_box(128, Wo, Ho, N, &bw, &bh, &bnn);
    CUtensorMap ta, tb;
    {
        unsigned long long dims[4] = {(unsigned long long)Cin, (unsigned long long)W, (unsigned long long)H, (unsigned long long)N * planes};
        unsigned long long str[3] = {(unsigned long long)Cin, (unsigned long long)W * Cin, (unsigned long long)H * W * Cin};
        unsigned box[4] = {32, (unsigned)bw, (unsigned)bh, (unsigned)bnn};
        if (!make_map(&ta, xs, 4, dims, str, box, false)) return NC_CUDA_ERR_UNSUPPORTED;
        unsigned long long wd[2] = {(unsigned long long)Cin, (unsigned long long)kH * kW * Cout * planes};
        unsigned long long ws[1] = {(unsigned long long)Cin};
        unsigned wb[2] = {32, (unsigned)bn_cols};
        if (!make_map(&tb, wpacked, 2, wd, ws, wb, false)) return NC_CUDA_ERR_UNSUPPORTED;
    }
    TcParams p = {};
    p.kind = KIND_CONV;
    p.M = N * Ho * Wo; p.N = Cout;
    p.cchunks = (Cin + 31) / 32;
    p.planes = planes;
    p.a_plane = N; p.b_plane = kH * kW * Cout;
    p.num_k_tiles = kH * kW * p.cchunks;
    p.k_tiles_per_split = p.num_k_tiles;
    p.D = y; p.ldd = Cout; p.bias = bias; p.alpha = 1.f; p.beta = 0.f;
    p.bw = bw; p.bh = bh; p.bn = bnn;
    p.tiles_w = (Wo + bw - 1) / bw; p.tiles_h = (Ho + bh - 1) / bh;
    p.Ho = Ho; p.Wo = Wo; p.Nimg = N;
    p.kW = kW; p.pad = pad; p.wrows = Cout;
    p.err = ncc::device_error_word();
    const long long tiles_m = (long long)p.tiles_w * p.tiles_h * ((N + bnn - 1) / bnn);
    dim3 grid((Cout + bn_cols - 1) / bn_cols, (unsigned)tiles_m, 1);
    p.flops = flops;
    return launch_bn<false, false>(bn_cols, ta, tb, p, grid, st);
}

int conv_strided_nhwc(float* y, const float* x, const float* wpacked, const float* bias, int N, int H, int W, int Cin, int Cout,
                      int kH, int kW, int stride, int pad, int mode, cudaStream_t st) {
    const int Ho = (H + 2 * pad - kH) / stride + 1, Wo = (W + 2 * pad - kW) / stride + 1;
    if (!conv_strided_eligible(Cin, Cout, (long long)N * Ho * Wo, kH, kW, stride)) return NC_CUDA_ERR_UNSUPPORTED;
    const float* xs = split_pixels(kSlotA, x, (size_t)N * H * W, Cin, mode, st);
    if (!xs) return NC_CUDA_ERR_RUNTIME;
    ConvClass c = {};
    c.kH = kH; c.kW = kW; c.pad_h = c.pad_w = pad; c.Ho = Ho; c.Wo = Wo;
    return convt_launch(y, Ho, Wo, 1, xs, wpacked, (long long)kH * kW * Cout, bias, N, H, W, Cin, Cout, stride, &c, 1, mode,
                        ncc::conv_stats_wanted(), 2.0 * N * Ho * Wo * (double)Cout * Cin * kH * kW, st);
}

// Input coordinate h of residue class r is h = s * i + r; filter row kh reaches it from output row (h + pad - kh) / s, so with
// kh0 = (r + pad) mod s only the taps kh0, kh0 + s, ... count, and output row = i + (r + pad - kh0) / s - t for the t-th of them.
// Reversed, they are an ordinary stride-1 filter over dy with padding taps - 1 - (r + pad - kh0) / s.
static void residue_axis(int r, int k, int s, int pad, int extent, int* kh0, int* taps, int* cpad, int* outs) {
    *kh0 = (r + pad) % s;
    *taps = *kh0 < k ? (k - *kh0 + s - 1) / s : 0;
    *cpad = *taps - 1 - (r + pad - *kh0) / s;
    *outs = r < extent ? (extent - r + s - 1) / s : 0;
}
int conv_dx_strided_nhwc(float* dx, const float* dy, const float* wpacked, int N, int H, int W, int Cin, int Cout, int kH, int kW,
                         int stride, int pad, int mode, cudaStream_t st) {
    const int Ho = (H + 2 * pad - kH) / stride + 1, Wo = (W + 2 * pad - kW) / stride + 1;
    if (!conv_strided_eligible(Cout, Cin, (long long)N * H * W, kH, kW, stride)) return NC_CUDA_ERR_UNSUPPORTED;
    const float* ds = split_pixels(kSlotA, dy, (size_t)N * Ho * Wo, Cout, mode, st);
    if (!ds) return NC_CUDA_ERR_RUNTIME;
    ConvClass cls[kMaxClasses] = {};
    int n = 0, row = 0;
    for (int rh = 0; rh < stride; rh++)
        for (int rw = 0; rw < stride; rw++) {
            ConvClass c = {};
            int a, b;
            residue_axis(rh, kH, stride, pad, H, &a, &c.kH, &c.pad_h, &c.Ho);
            residue_axis(rw, kW, stride, pad, W, &b, &c.kW, &c.pad_w, &c.Wo);
            c.oh0 = rh; c.ow0 = rw;
            c.wrow0 = row * Cin;
            row += c.kH * c.kW;
            if (c.Ho > 0 && c.Wo > 0) cls[n++] = c;
        }
    return convt_launch(dx, H, W, stride, ds, wpacked, (long long)kH * kW * Cin, nullptr, N, Ho, Wo, Cout, Cin, 1, cls, n, mode, false,
                        2.0 * N * Ho * Wo * (double)Cout * Cin * kH * kW, st);
}
// the input box of a forward pass is at most 256 pixels wide before its stride; the input gradient has stride^2 classes
bool conv_strided_eligible(int Cin, int Cout, long long pixels, int kH, int kW, int stride) {
    return conv_eligible(Cin, Cout, pixels) && stride == 2 && kH * kW <= 64 && kH <= 16 && kW <= 16;
}

int conv_dw_nhwc(float* dW, const float* dy, const float* x, int N, int H, int W, int Cin, int Cout, int kH, int kW, int stride, int pad,
                 int mode, cudaStream_t st) {
    const int Ho = (H + 2 * pad - kH) / stride + 1, Wo = (W + 2 * pad - kW) / stride + 1;
    if (Ho <= 0 || Wo <= 0 || stride > 2) return NC_CUDA_ERR_UNSUPPORTED;
    if ((Cin & 3) || (Cout & 3) || Cin < 16 || Cout < 16) return NC_CUDA_ERR_UNSUPPORTED;
    const int planes = mode_planes(mode);
    const float* xs = split_pixels(kSlotA, x, (size_t)N * H * W, Cin, mode, st);
    const float* ds = split_pixels(kSlotB, dy, (size_t)N * Ho * Wo, Cout, mode, st);
    if (!xs || !ds) return NC_CUDA_ERR_RUNTIME;
    if (stride == 1) {
        const int rc = conv_dw_halo_nhwc(dW, ds, xs, N, H, W, Cin, Cout, kH, kW, pad, planes, st);
        if (rc != NC_CUDA_ERR_UNSUPPORTED) return rc;
    }
    const int Cp = (Cin + 31) & ~31;   // channels beyond Cin are zero-filled by TMA and dropped in the second stage
    const int Ncols = kH * kW * Cp;
    // column tile: whole filter rows when they fit in 256 columns, else 256 / 128 / 64
    int bn_cols;
    if (planes == 1 && (kW * Cp == 64 || kW * Cp == 128 || kW * Cp == 192 || kW * Cp == 256)) bn_cols = kW * Cp;
    else bn_cols = pick_bn(Ncols, planes == 2);
    int bw = 1, bh = 1, bnn = 1;
    // split operands: a box that hung over the last image of the hi plane would read the lo plane instead of zeros
    pick_box(32, Wo, Ho, N, &bw, &bh, &bnn, 1, 256 / stride, planes == 2);
    CUtensorMap ta, tb;
    {
        unsigned long long dims[4] = {(unsigned long long)Cout, (unsigned long long)Wo, (unsigned long long)Ho, (unsigned long long)N * planes};
        unsigned long long str[3] = {(unsigned long long)Cout, (unsigned long long)Wo * Cout, (unsigned long long)Ho * Wo * Cout};
        unsigned box[4] = {32, (unsigned)bw, (unsigned)bh, (unsigned)bnn};
        if (!make_map(&ta, ds, 4, dims, str, box, true)) return NC_CUDA_ERR_UNSUPPORTED;
        unsigned long long xd[4] = {(unsigned long long)Cin, (unsigned long long)W, (unsigned long long)H, (unsigned long long)N * planes};
        unsigned long long xst[3] = {(unsigned long long)Cin, (unsigned long long)W * Cin, (unsigned long long)H * W * Cin};
        if (!make_map(&tb, xs, 4, xd, xst, box, true, stride)) return NC_CUDA_ERR_UNSUPPORTED;
    }
    TcParams p = {};
    p.kind = KIND_DW;
    p.M = Cout; p.N = Ncols;
    p.bw = bw; p.bh = bh; p.bn = bnn;
    p.tiles_w = (Wo + bw - 1) / bw; p.tiles_h = (Ho + bh - 1) / bh;
    p.Ho = Ho; p.Wo = Wo; p.Nimg = N;
    p.kW = kW; p.pad = pad; p.stride = stride; p.Cin = Cp;
    p.planes = planes;
    p.num_k_tiles = p.tiles_w * p.tiles_h * ((N + bnn - 1) / bnn);
    p.a_plane = p.b_plane = N;
    p.alpha = 1.f;
    p.err = ncc::device_error_word();
    const int tiles_m = (Cout + BM - 1) / BM, tiles_n = (Ncols + bn_cols - 1) / bn_cols;
    int splits, kps;
    pick_splits(tiles_m * tiles_n, p.num_k_tiles, &splits, &kps);
    p.k_tiles_per_split = kps;
    p.partial = (float*)ncc::scratch(2, sizeof(float) * (size_t)splits * Cout * Ncols, st);
    if (!p.partial) return NC_CUDA_ERR_RUNTIME;
    dim3 grid(tiles_n, tiles_m, splits);
    p.flops = 2.0 * N * Ho * Wo * (double)Cout * Cin * kH * kW;
    int rc;
    if (bn_cols == 192) rc = launch_one<192, true, true, false>(ta, tb, p, grid, st);
    else rc = launch_bn<true, true>(bn_cols, ta, tb, p, grid, st);
    if (rc) return rc;
    return dw_reduce(dW, p.partial, splits, Cout, Cin, kH, kW, st);
}

int dw_reduce(float* dW, const float* partial, int splits, int Cout, int Cin, int kH, int kW, cudaStream_t st) {
    const int Cp = (Cin + 31) & ~31;
    const long long total = (long long)Cout * Cp * kH * kW;
    if (splits >= 64) ncc::launch(dw_reduce_kernel<8>, ncc::grid_for(total / 32, 1), 256, 0, st, dW, partial, splits, Cout, Cin, Cp, kH * kW);
    else ncc::launch(dw_reduce_kernel<1>, ncc::grid_for(total, 256), 256, 0, st, dW, partial, splits, Cout, Cin, Cp, kH * kW);
    NCC_COUNT_LAUNCH();
    return ncc::launch_status("dw_reduce");
}

// Packed weights: rounded to TF32 in every tensor-core mode, with the remainders as a second plane for 3xTF32.
int pack_weights_fwd(float* wp, const float* w, int Cout, int Cin, int kH, int kW, int planes, cudaStream_t st) {
    const TapOrder o = {};
    ncc::launch(pack_weights_kernel<false>, ncc::grid_for((long long)Cout * Cin * kH * kW, 256), 256, 0, st, wp, w, Cout, Cin, kH * kW, o, 1, planes);
    NCC_COUNT_LAUNCH();
    return ncc::launch_status("pack_weights_fwd");
}
int pack_weights_dx(float* wp, const float* w, int Cout, int Cin, int kH, int kW, int stride, int pad, int planes, cudaStream_t st) {
    TapOrder o = {};
    if (stride > 1) {   // per residue class, taps reversed
        if (kH * kW > 64) return NC_CUDA_ERR_UNSUPPORTED;
        o.listed = 1;
        int t = 0;
        for (int rh = 0; rh < stride; rh++)
            for (int rw = 0; rw < stride; rw++) {
                int a, b, th, tw, unused, outs;
                residue_axis(rh, kH, stride, pad, 1, &a, &th, &unused, &outs);
                residue_axis(rw, kW, stride, pad, 1, &b, &tw, &unused, &outs);
                for (int i = th - 1; i >= 0; i--)
                    for (int j = tw - 1; j >= 0; j--) o.at[t++] = (unsigned char)((a + i * stride) * kW + b + j * stride);
            }
    }
    ncc::launch(pack_weights_kernel<true>, ncc::grid_for((long long)Cout * Cin * kH * kW, 256), 256, 0, st, wp, w, Cout, Cin, kH * kW, o, 1, planes);
    NCC_COUNT_LAUNCH();
    return ncc::launch_status("pack_weights_dx");
}

}  // namespace tc
