// f32-accurate GEMM on the tensor core for the head of the f32 model: C[M,N] = A * B with every f32 operand
// carried as TWO f16 values,
//     x * s  =  hi + lo * 2^-11,     hi = f16(x * s),   lo = f16((x * s - hi) * 2^11)      (s: a power of two),
// and the product expanded into three `tcgen05.mma kind::f16` products with f32 accumulation in TMEM:
//     main += A_hi * B_hi        corr += A_hi * B_lo + A_lo * B_hi        C = (main + corr * 2^-11) * out_scale
// (the lo * lo term is below 2^-22 of the product).  hi and lo have 11 significant bits each, so an operand is
// carried to 2^-22 and a 192- or 50257-term sum comes out closer to the exact value than a sequential f32 sum
// does; the reference computes these products in full f32 (cuBLAS with CUBLAS_COMPUTE_32F,
// src/storage/cuda.rs:1098-1128), not in TF32, and this keeps that accuracy at tensor-core speed.
// It serves `lm_head` of src/models/gpt.rs:351 and the two products of its backward (src/ops.rs:1089-1101):
// 80 % of the FLOPs of a training step of the reference's GPT.
//
// Two kernels.  gemm_f16x3_pair_kernel (described there): pairs of CTAs, the head of a training step.  gemm_f16x3_kernel, for products of few
// tiles: persistent, 128 x 128 output tiles, 64-deep K blocks, 3-stage TMA ring of four operand tiles (A_hi,
// A_lo, B_hi, B_lo: 64 KB per stage, 128-byte swizzle, out-of-range rows / columns read as zero), twelve MMAs
// per K block, two pairs of TMEM accumulators so the epilogue of a tile overlaps the next tile's products.
// Either storage order of A and of B (the operand orders of forward, dgrad and wgrad), as in gemm_f16_sm100.cu.
// Long reductions with few output tiles (the head's input gradient: K = vocabulary) are split along K over the
// work units; every part writes its f32 partial tile, a second kernel adds the parts in index order.
#include "sm100_ptx.cuh"
#include "tma_host.cuh"

#include <cooperative_groups.h>

namespace {
using namespace sm100;

constexpr int XM = 128, XN = 128, XK = 64;
constexpr uint32_t X_TILE = 128 * XK * 2;          // 16 KB: one operand tile of a stage
constexpr uint32_t X_STAGE = 4 * X_TILE;           // A_hi | A_lo | B_hi | B_lo
constexpr int X_STAGES = 3;

constexpr uint32_t X_MN_BLOCK = XK * 128;          // 8 KB: 64 K-rows x 64 columns of an MN-major operand
constexpr float X_LO = 1.0f / 2048.0f;

// warp 0 TMA, warp 1 MMA, then two epilogue warpgroups that each take half of a tile's columns: with one, the
// head's forward product waits on its epilogue (206 MB of logits through 4 warps per SM), not on the tensor pipe
constexpr int X_EPI_WG = 2;
constexpr int X_THREADS = 64 + 128 * X_EPI_WG;

constexpr uint32_t X_TURN = X_STAGES * X_STAGE + 256;              // per epilogue warp: 32 x 32 elements, padded
constexpr int X_TURN_FLOATS = 32 * 33;
constexpr uint32_t X_SMEM = X_TURN + 4 * X_EPI_WG * X_TURN_FLOATS * 4;

enum XBar { X_FULL = 0, X_EMPTY = 3, X_ACC_FULL = 6, X_ACC_EMPTY = 8, X_COUNT = 10 };

struct X3Params {
    float* c;                   // parts == 1: the output; parts > 1: partial tiles [part][M][N] (dense)
    long long ldc;
    int M, N, K;
    int parts, k_chunk;         // K range of part p: [p * k_chunk, min(K, (p + 1) * k_chunk)); k_chunk % 64 == 0
    float out_scale;
    int vec;                    // rows of c start on 16-byte boundaries: 16-byte stores
    unsigned int* err;
};

// The part of the start that needs nothing of global memory (see started()).
__device__ __forceinline__ void gemm_f16x3_prologue(const void* tm_ah, const void* tm_al, const void* tm_bh, const void* tm_bl) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + X_STAGES * X_STAGE);
    uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(bars + X_COUNT);
    if (threadIdx.x == 0) {
        tmem_base_s[1] = 0;                                     // the abort flag
        for (int s = 0; s < X_STAGES; ++s) { mbar_init(&bars[X_FULL + s], 1); mbar_init(&bars[X_EMPTY + s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&bars[X_ACC_FULL + s], 1); mbar_init(&bars[X_ACC_EMPTY + s], 128 * X_EPI_WG); }
        fence_barrier_init();
        tma_prefetch_desc(tm_ah); tma_prefetch_desc(tm_al); tma_prefetch_desc(tm_bh); tma_prefetch_desc(tm_bl);
    }
    if (uniform((int)threadIdx.x / 32) == 1) {
        tmem_alloc(tmem_base_s, 512);
        tmem_relinquish();
    }
}

template <int A_MN, int B_MN>
__global__ void __launch_bounds__(X_THREADS, 1)
gemm_f16x3_kernel(const __grid_constant__ CUtensorMap tm_ah, const __grid_constant__ CUtensorMap tm_al,
                  const __grid_constant__ CUtensorMap tm_bh, const __grid_constant__ CUtensorMap tm_bl, const X3Params p) {
    gemm_f16x3_prologue(&tm_ah, &tm_al, &tm_bh, &tm_bl);
    chain_wait();
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + X_STAGES * X_STAGE);
    uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(bars + X_COUNT);
    volatile uint32_t* abort_s = tmem_base_s + 1;
    uint32_t* skip_s = tmem_base_s + 2;

    const int warp = uniform((int)threadIdx.x / 32), lane = threadIdx.x % 32;
    const int tiles_m = (p.M + XM - 1) / XM, tiles_n = (p.N + XN - 1) / XN;
    const int n_units = tiles_m * tiles_n * p.parts;

    if (!started(smem, skip_s, p.err, DEERS_KERR_GEMM | 0x21)) {
        if (warp == 1) tmem_dealloc(*tmem_base_s, 512);
        return;
    }
    const uint32_t tmem = (uint32_t)uniform((int)*tmem_base_s);
    WaitState ws{abort_s, p.err};

    // unit u -> (tile, part); consecutive units are the parts of one tile, so they run at the same time on
    // neighbouring CTAs and share the B columns in L2
    auto unit = [&](int u, int& tm, int& tn, int& kb0, int& kb1) {
        const int part = u % p.parts, tile = u / p.parts;
        tm = tile % tiles_m; tn = tile / tiles_m;
        const int k0 = part * p.k_chunk;
        const int k1 = min(p.K, k0 + p.k_chunk);
        kb0 = k0 / XK; kb1 = (k1 + XK - 1) / XK;
    };

    if (warp == 0) {
        // ------------------------------ TMA producer ------------------------------
        if (lane == 0) {
            uint32_t g = 0;
            bool ok = true;
            for (int u = blockIdx.x; ok && u < n_units; u += gridDim.x) {
                int tm, tn, kb0, kb1;
                unit(u, tm, tn, kb0, kb1);
                for (int kb = kb0; kb < kb1; ++kb, ++g) {
                    const uint32_t s = g % X_STAGES;
                    if (!mbar_wait(ws, &bars[X_EMPTY + s], ((g / X_STAGES) & 1u) ^ 1u, DEERS_KERR_GEMM | 0x11)) { ok = false; break; }
                    mbar_arrive_expect_tx(&bars[X_FULL + s], X_STAGE);
                    uint8_t* st = smem + s * X_STAGE;
#pragma unroll
                    for (int half = 0; half < 2; ++half) {           // hi, lo
                        const CUtensorMap* ta = half ? &tm_al : &tm_ah;
                        const CUtensorMap* tb = half ? &tm_bl : &tm_bh;
                        uint8_t* a_dst = st + half * X_TILE;
                        uint8_t* b_dst = st + (2 + half) * X_TILE;
                        if (A_MN) {
#pragma unroll
                            for (int blk = 0; blk < XM / 64; ++blk)
                                tma_load_4d(a_dst + blk * X_MN_BLOCK, ta, &bars[X_FULL + s], tm * XM + blk * 64, kb * XK, 0, 0);
                        } else {
                            tma_load_4d(a_dst, ta, &bars[X_FULL + s], kb * XK, tm * XM, 0, 0);
                        }
                        if (B_MN) {
#pragma unroll
                            for (int blk = 0; blk < XN / 64; ++blk)
                                tma_load_4d(b_dst + blk * X_MN_BLOCK, tb, &bars[X_FULL + s], tn * XN + blk * 64, kb * XK, 0, 0);
                        } else {
                            tma_load_4d(b_dst, tb, &bars[X_FULL + s], kb * XK, tn * XN, 0, 0);
                        }
                    }
                }
            }
        }
        __syncwarp();
        chain_next();                                           // all loads are under way: the end is near
    } else if (warp == 1) {
        // ------------------------------ MMA issuer ------------------------------
        // The whole warp runs this; one elected lane issues (see elect_one).
        {
            constexpr uint32_t IDESC = idesc_f16(XM, XN, A_MN, B_MN);
            constexpr uint64_t TILE_STEP = X_TILE >> 4, STAGE_STEP = X_STAGE >> 4;
            const uint32_t s0 = (uint32_t)uniform((int)smem_u32(smem));
            const uint64_t a0 = A_MN ? desc_mnmajor(s0, 0, X_MN_BLOCK) : desc_kmajor(s0, 0, 0);
            const uint64_t b0 = B_MN ? desc_mnmajor(s0 + 2 * X_TILE, 0, X_MN_BLOCK)
                                     : desc_kmajor(s0 + 2 * X_TILE, 0, 0);
            uint32_t g = 0;
            int n = 0;
            bool ok = true;
            for (int u = blockIdx.x; ok && u < n_units; u += gridDim.x, ++n) {
                int tm, tn, kb0, kb1;
                unit(u, tm, tn, kb0, kb1);
                const uint32_t buf = (uint32_t)n & 1u;
                const uint32_t t_main = tmem + buf * 256u, t_corr = tmem + buf * 256u + 128u;
                if (!mbar_wait_warp(ws, &bars[X_ACC_EMPTY + buf], (((uint32_t)n >> 1) & 1u) ^ 1u, DEERS_KERR_GEMM | 0x12)) break;
                for (int kb = kb0; kb < kb1; ++kb, ++g) {
                    const uint32_t s = g % X_STAGES;
                    if (!mbar_wait_warp(ws, &bars[X_FULL + s], (g / X_STAGES) & 1u, DEERS_KERR_GEMM | 0x13)) { ok = false; break; }
                    tc_fence_after_sync();
                    const uint64_t ah = a0 + (uint64_t)s * STAGE_STEP, al = ah + TILE_STEP;
                    const uint64_t bh = b0 + (uint64_t)s * STAGE_STEP, bl = bh + TILE_STEP;
                    if (elect_one()) {
#pragma unroll
                        for (int ks = 0; ks < XK / 16; ++ks) {
                            const uint64_t sa = A_MN ? mnmajor_step(ks) : kmajor_step(ks, 0);
                            const uint64_t sb = B_MN ? mnmajor_step(ks) : kmajor_step(ks, 0);
                            const uint32_t first = (kb > kb0 || ks > 0);
                            umma_ss(t_main, ah + sa, bh + sb, IDESC, first);
                            umma_ss(t_corr, ah + sa, bl + sb, IDESC, first);
                            umma_ss(t_corr, al + sa, bh + sb, IDESC, 1u);
                        }
                        umma_commit(&bars[X_EMPTY + s]);
                        if (kb == kb1 - 1) umma_commit(&bars[X_ACC_FULL + buf]);
                    }
                    __syncwarp();
                }
            }
        }
    } else {
        // ------------------------------ epilogue ------------------------------
        const int lane_base = (warp & 3) * 32;
        const uint32_t t_lane = (uint32_t)lane_base << 16;
        const int ewg = (warp - 2) >> 2;                         // which share of the columns
        constexpr int CHUNKS = XN / 32 / X_EPI_WG;
        int n = 0;
        for (int u = blockIdx.x; u < n_units; u += gridDim.x, ++n) {
            int tm, tn, kb0, kb1;
            unit(u, tm, tn, kb0, kb1);
            const int part = u % p.parts;
            const uint32_t buf = (uint32_t)n & 1u;
            if (!__all_sync(0xffffffffu, mbar_wait(ws, &bars[X_ACC_FULL + buf], ((uint32_t)n >> 1) & 1u, DEERS_KERR_GEMM | 0x14))) break;
            tc_fence_after_sync();
            float* cbase = p.c + (p.parts > 1 ? (long long)part * p.M * p.ldc : 0);
            const int row0 = tm * XM + lane_base + (lane & ~7);
#pragma unroll 1
            for (int chunk = ewg * CHUNKS; chunk < (ewg + 1) * CHUNKS; ++chunk) {      // 32 columns at a time
                uint32_t rm[32], rc[32];
                tmem_ld_x32(tmem + buf * 256u + t_lane + chunk * 32, rm);
                tmem_ld_x32(tmem + buf * 256u + 128u + t_lane + chunk * 32, rc);
                tmem_wait_ld();
                if (chunk == (ewg + 1) * CHUNKS - 1) {           // this warpgroup's share of both accumulators is in registers
                    tc_fence_before_sync();
                    mbar_arrive(&bars[X_ACC_EMPTY + buf]);
                }
                float o[32];
#pragma unroll
                for (int e = 0; e < 32; ++e) o[e] = fmaf(__uint_as_float(rc[e]), X_LO, __uint_as_float(rm[e])) * p.out_scale;
                if (p.vec) {
                    uint4 pc[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        pc[q] = make_uint4(__float_as_uint(o[q * 4]), __float_as_uint(o[q * 4 + 1]), __float_as_uint(o[q * 4 + 2]), __float_as_uint(o[q * 4 + 3]));
                    // 16-byte pieces transposed within 8-lane groups: a store instruction writes 128 contiguous bytes per row
                    transpose_pieces<8>(pc, (uint32_t)lane);
                    const int col = tn * XN + chunk * 32 + (lane & 7) * 4;
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const int row = row0 + c;
                        if (row >= p.M || col >= p.N) continue;
                        float* dst = cbase + (long long)row * p.ldc + col;
                        if (col + 4 <= p.N) {
                            *reinterpret_cast<uint4*>(dst) = pc[c];
                        } else {
                            const uint32_t v[4] = {pc[c].x, pc[c].y, pc[c].z, pc[c].w};
                            for (int e = 0; e < 4 && col + e < p.N; ++e) dst[e] = __uint_as_float(v[e]);
                        }
                    }
                } else {
                    // Rows on any 4-byte boundary (logits of an odd vocabulary, straight into the caller's tensor): 32 x 32 elements
                    // turned round in the warp's own shared memory, a row per store instruction.  100 x 50257 x 192: 16 us, as
                    // with padded rows, and the copy behind those took 11.
                    float* turn = reinterpret_cast<float*>(smem + X_TURN) + (warp - 2) * X_TURN_FLOATS;
#pragma unroll
                    for (int e = 0; e < 32; ++e) turn[lane * 33 + e] = o[e];
                    __syncwarp();
                    const int col = tn * XN + chunk * 32 + lane, first = tm * XM + lane_base;
                    if (col < p.N) {
#pragma unroll 8
                        for (int r = 0; r < 32; ++r)
                            if (first + r < p.M) cbase[(long long)(first + r) * p.ldc + col] = turn[r * 33 + lane];
                    }
                    __syncwarp();
                }
            }
        }
    }
    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

// ---------------------------------------------------------------------------------------------
// Pairs of CTAs on tiles of 256 x TN
// ---------------------------------------------------------------------------------------------
// A CTA alone on 128 x 128 reads 800 MB through L2 for a head product of 1024 tokens (10 TB/s: 75 to 85 us) and moves 213 bytes a cycle through
// its shared memory, which has 128.  A pair (cta_group::2) brings half of B's columns each: of 192 columns 350 to 400 MB and 121 bytes, and 192
// columns are one tile where 128-wide ones compute a quarter for nothing.  Bound now: the gradients by L2 and HBM reads (4.9 and 7 TB/s), the
// logits by their 206 MB and the epilogue that makes them.
//   TN = 128  two pairs of accumulators in TMEM, an epilogue beside the next tile's products
//   TN = 192  one pair of accumulators (384 columns): for long K
//   TURN      rows of C on any 4-byte boundary, turned round in shared memory
//   TRANS     the caller's C is [N][M]: 32 rows of M are one contiguous store (head weight gradient: M is the vocabulary)
//   STATS     also per row and 32 columns (maximum, sum of exponentials relative to it): the cross-entropy then needs no pass of its own
//   resident  (up to P_RES_KB K blocks) A stays in shared memory while the pair walks along N: 150 MB instead of 450 for the logits
constexpr int P_M = 256;
// Shared memory: the ring (stages, or resident A and stages of B) | barriers | TURN: 32 x 32 elements per epilogue warp
__host__ __device__ constexpr uint32_t p_ring(bool turn) { return turn ? 163840 : 196608; }
constexpr int P_RES_KB = 4;                            // K blocks of A that may stay
// Epilogue warpgroups, each with 32 (TN = 128) or 64 columns: four warps per scheduler for the logits.
__host__ __device__ constexpr int p_epi_wg(int tn) { return tn == 128 ? 4 : 3; }
__host__ __device__ constexpr int p_threads(int tn) { return 64 + 128 * p_epi_wg(tn); }
__host__ __device__ constexpr uint32_t p_smem(bool turn) { return p_ring(turn) + 256 + (turn ? 16 * 4096 : 0); }
static_assert(p_smem(false) <= 232448 && p_smem(true) <= 232448, "shared memory");
constexpr int P_MAX_STAGES = 10;
enum PBar { P_FULL = 0, P_EMPTY = P_MAX_STAGES, P_ACC_FULL = 2 * P_MAX_STAGES, P_ACC_EMPTY = P_ACC_FULL + 2, P_A_FULL = P_ACC_EMPTY + 2, P_COUNT };
static_assert(P_COUNT * 8 + 16 <= 256, "barriers");

struct X3PairParams {
    float* c;                   // parts == 1: the output; parts > 1: partial tiles [part][M][N] (dense)
    long long ldc;
    int M, N, K;
    int parts, k_chunk;
    float out_scale;
    int resident;               // K blocks of A that stay (0: A travels with B); needs parts == 1
    float2* stats;              // STATS: [4 * tiles along N][M]
    unsigned int* err;
};

__device__ __forceinline__ float x3_ex2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float x3_max_nan(float a, float b) { float y; asm("max.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b)); return y; }

// exp(o - ref) of 32 values, summed.  y log2(e) is rounded to z, exp2(z) corrected by the first order of what the rounding lost.
__device__ __forceinline__ float x3_exp_sum(const float (&o)[32], float ref) {
    constexpr float LH = 1.44269502162933349609f, LL = 1.92596299112661746887e-8f, LN2 = 0.693147180559945309417f;    // LH + LL = log2(e)
    uint64_t s2 = 0;
    const uint64_t nref = pack_f32x2(-ref, -ref), lh = pack_f32x2(LH, LH), ll = pack_f32x2(LL, LL), ln2 = pack_f32x2(LN2, LN2);
#pragma unroll
    for (int e = 0; e < 32; e += 2) {
        float a, b, z0, z1;
        unpack_f32x2(add2(pack_f32x2(o[e], o[e + 1]), nref), a, b);
        const uint64_t y = pack_f32x2(x3_max_nan(a, -160.f), x3_max_nan(b, -160.f));              // (exp(-160) is below any sum's last place)
        const uint64_t z = mul2(y, lh);
        unpack_f32x2(z, z0, z1);
        const uint64_t r = mul2(fma2(y, ll, fma2(y, lh, pack_f32x2(-z0, -z1))), ln2);
        const uint64_t x = pack_f32x2(x3_ex2(z0), x3_ex2(z1));
        s2 = add2(s2, fma2(x, r, x));
    }
    float s, t;
    unpack_f32x2(s2, s, t);
    return s + t;
}

template <int TN, int B_MN, bool TURN>
struct X3PairShape {
    static constexpr uint32_t RING = p_ring(TURN);
    static constexpr int BN = TN / 2;                                                    // columns of B a CTA brings
    static constexpr int B_BLOCKS = (BN + 63) / 64;    // MN order: of 64 columns (half of the second is not used for 192)
    static constexpr uint32_t B_TILE = B_MN ? B_BLOCKS * X_MN_BLOCK : BN * XK * 2u;      // hi or lo of a stage
    static constexpr uint32_t A_STAGE = 2 * X_TILE, B_STAGE = 2 * B_TILE;
    static constexpr int STAGES = RING / (A_STAGE + B_STAGE);
    static constexpr int BUFS = TN == 128 ? 2 : 1;
    static_assert(STAGES <= P_MAX_STAGES && (RING - A_STAGE) / B_STAGE <= P_MAX_STAGES && B_TILE % 1024 == 0, "ring");
};

// The part of the start that needs nothing of global memory (see started()).
template <int TN, bool TURN>
__device__ __forceinline__ void gemm_f16x3_pair_prologue(const void* tm_ah, const void* tm_al, const void* tm_bh, const void* tm_bl) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + p_ring(TURN));
    uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(bars + P_COUNT);
    if (threadIdx.x == 0) {
        tmem_base_s[1] = 0;                                     // the abort flag
        for (int s = 0; s < P_MAX_STAGES; ++s) { mbar_init(&bars[P_FULL + s], 1); mbar_init(&bars[P_EMPTY + s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&bars[P_ACC_FULL + s], 1); mbar_init(&bars[P_ACC_EMPTY + s], 2 * 4 * p_epi_wg(TN)); }
        mbar_init(&bars[P_A_FULL], 1);
        fence_barrier_init();
        tma_prefetch_desc(tm_ah); tma_prefetch_desc(tm_al); tma_prefetch_desc(tm_bh); tma_prefetch_desc(tm_bl);
    }
    if (uniform((int)threadIdx.x / 32) == 1) {
        tmem_alloc_pair(tmem_base_s, 512);
        tmem_relinquish_pair();
    }
}

template <int A_MN, int B_MN, int TN, bool TRANS, bool STATS, bool TURN>
__global__ void __launch_bounds__(p_threads(TN), 1)
gemm_f16x3_pair_kernel(const __grid_constant__ CUtensorMap tm_ah, const __grid_constant__ CUtensorMap tm_al,
                       const __grid_constant__ CUtensorMap tm_bh, const __grid_constant__ CUtensorMap tm_bl, const X3PairParams p) {
    gemm_f16x3_pair_prologue<TN, TURN>(&tm_ah, &tm_al, &tm_bh, &tm_bl);
    chain_wait();
    namespace cg = cooperative_groups;
    using S = X3PairShape<TN, B_MN, TURN>;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + p_ring(TURN));
    uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(bars + P_COUNT);
    volatile uint32_t* abort_s = tmem_base_s + 1;
    uint32_t* skip_s = tmem_base_s + 2;

    const int warp = uniform((int)threadIdx.x / 32), lane = threadIdx.x % 32;
    const int half = (int)cg::this_cluster().block_rank();
    const int tiles_m = (p.M + P_M - 1) / P_M, tiles_n = (p.N + TN - 1) / TN;
    const int n_units = tiles_m * tiles_n * p.parts;
    const int pairs = (int)gridDim.x / 2, pair = (int)blockIdx.x / 2;

    bool skip = !started(smem, skip_s, p.err, DEERS_KERR_GEMM | 0x41);
    cg::this_cluster().sync();                                  // both have their barriers, and both go on or neither
    skip = skip || *cg::this_cluster().map_shared_rank(skip_s, half ^ 1) != 0;
    const uint32_t tmem = (uint32_t)uniform((int)*tmem_base_s);
    WaitState ws{abort_s, p.err};

    // This pair's units, neighbouring pairs on neighbouring units: what runs at the same time shares what it reads in L2 and writes
    // neighbouring pieces of rows.  With a resident A a pair keeps to one row of tiles, every rows-th unit.
    const bool res = p.resident != 0;
    const int u_first = pair, u_end = n_units, u_step = res ? pairs / tiles_m * tiles_m : pairs;
    const int stages = res ? min(P_MAX_STAGES, (int)((S::RING - p.resident * S::A_STAGE) / S::B_STAGE)) : S::STAGES;
    const uint32_t ring = res ? p.resident * S::A_STAGE : 0u, stage_bytes = res ? S::B_STAGE : S::A_STAGE + S::B_STAGE;
    auto unit = [&](int u, int& tm, int& tn, int& kb0, int& kb1) {
        const int part = u % p.parts, tile = u / p.parts;
        tm = tile % tiles_m; tn = tile / tiles_m;
        const int k0 = part * p.k_chunk, k1 = min(p.K, k0 + p.k_chunk);
        kb0 = k0 / XK; kb1 = (k1 + XK - 1) / XK;
    };

    if (skip) {
    } else if (warp == 0) {
        // ------------------------------ TMA producer ------------------------------
        if (lane == 0) {
            uint32_t s = 0, turn = 0;                               // place in the ring, times round it
            bool have_a = false;
            bool ok = true;
            // hi and lo of the CTA's half of a K block
            auto load_a = [&](uint8_t* dst, int tm, int kb, uint32_t bar) {
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    const CUtensorMap* t = w ? &tm_al : &tm_ah;
                    const int m0 = tm * P_M + half * XM;
                    if (A_MN) {
#pragma unroll
                        for (int blk = 0; blk < XM / 64; ++blk)
                            tma_load_4d_pair(dst + w * X_TILE + blk * X_MN_BLOCK, t, bar, m0 + blk * 64, kb * XK, 0, 0);
                    } else {
                        tma_load_4d_pair(dst + w * X_TILE, t, bar, kb * XK, m0, 0, 0);
                    }
                }
            };
            auto load_b = [&](uint8_t* dst, int tn, int kb, uint32_t bar) {
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    const CUtensorMap* t = w ? &tm_bl : &tm_bh;
                    const int n0 = tn * TN + half * S::BN;
                    if (B_MN) {
#pragma unroll
                        for (int blk = 0; blk < S::B_BLOCKS; ++blk)
                            tma_load_4d_pair(dst + w * S::B_TILE + blk * X_MN_BLOCK, t, bar, n0 + blk * 64, kb * XK, 0, 0);
                    } else {
                        tma_load_4d_pair(dst + w * S::B_TILE, t, bar, kb * XK, n0, 0, 0);
                    }
                }
            };
            for (int u = u_first; ok && u < u_end; u += u_step) {
                int tm, tn, kb0, kb1;
                unit(u, tm, tn, kb0, kb1);
                if (res && !have_a) {
                    if (half == 0) mbar_arrive_expect_tx(&bars[P_A_FULL], 2u * p.resident * S::A_STAGE);
                    for (int kb = 0; kb < p.resident; ++kb) load_a(smem + kb * S::A_STAGE, tm, kb, cluster_addr(&bars[P_A_FULL], 0));
                    have_a = true;
                }
                for (int kb = kb0; kb < kb1; ++kb) {
                    if (!mbar_wait(ws, &bars[P_EMPTY + s], (turn & 1u) ^ 1u, DEERS_KERR_GEMM | 0x42)) { ok = false; break; }
                    if (half == 0) mbar_arrive_expect_tx(&bars[P_FULL + s], 2u * stage_bytes);
                    uint8_t* st = smem + ring + s * stage_bytes;
                    const uint32_t bar = cluster_addr(&bars[P_FULL + s], 0);
                    if (!res) { load_a(st, tm, kb, bar); st += S::A_STAGE; }
                    load_b(st, tn, kb, bar);
                    if (++s == (uint32_t)stages) { s = 0; ++turn; }
                }
            }
        }
        __syncwarp();
        chain_next();                                           // all loads are under way: the end is near
    } else if (warp == 1) {
        // ------------------------------ MMA issuer (the pair's first CTA) ------------------------------
        if (half == 0) {
            constexpr uint32_t IDESC = idesc_f16(P_M, TN, A_MN, B_MN);
            const uint32_t s0 = (uint32_t)uniform((int)smem_u32(smem));
            const uint64_t a0 = A_MN ? desc_mnmajor(s0, 0, X_MN_BLOCK) : desc_kmajor(s0, 0, 0);
            const uint64_t b0 = B_MN ? desc_mnmajor(s0, 0, X_MN_BLOCK) : desc_kmajor(s0, 0, 0);
            uint32_t s = 0, turn = 0;
            int n = 0;
            bool ok = true;
            for (int u = u_first; ok && u < u_end; u += u_step, ++n) {
                int tm, tn, kb0, kb1;
                unit(u, tm, tn, kb0, kb1);
                const uint32_t buf = S::BUFS == 2 ? (uint32_t)n & 1u : 0u, t_main = tmem + buf * 256u, t_corr = t_main + TN;
                const uint32_t use = S::BUFS == 2 ? (uint32_t)n >> 1 : (uint32_t)n;
                if (!mbar_wait_warp(ws, &bars[P_ACC_EMPTY + buf], (use & 1u) ^ 1u, DEERS_KERR_GEMM | 0x43)) break;
                tc_fence_after_sync();
                if (res && n == 0 && !mbar_wait_warp(ws, &bars[P_A_FULL], 0u, DEERS_KERR_GEMM | 0x46)) break;
                for (int kb = kb0; kb < kb1; ++kb) {
                    if (!mbar_wait_warp(ws, &bars[P_FULL + s], turn & 1u, DEERS_KERR_GEMM | 0x44)) { ok = false; break; }
                    tc_fence_after_sync();
                    const uint32_t at = ring + s * stage_bytes;
                    const uint64_t ah = a0 + (uint64_t)((res ? (uint32_t)kb * S::A_STAGE : at) >> 4), al = ah + (X_TILE >> 4);
                    const uint64_t bh = b0 + (uint64_t)((res ? at : at + S::A_STAGE) >> 4), bl = bh + (S::B_TILE >> 4);
                    if (elect_one()) {
#pragma unroll
                        for (int ks = 0; ks < XK / 16; ++ks) {
                            const uint64_t sa = A_MN ? mnmajor_step(ks) : kmajor_step(ks, 0);
                            const uint64_t sb = B_MN ? mnmajor_step(ks) : kmajor_step(ks, 0);
                            const uint32_t first = (kb > kb0 || ks > 0);
                            umma_ss_pair(t_main, ah + sa, bh + sb, IDESC, first);
                            umma_ss_pair(t_corr, ah + sa, bl + sb, IDESC, first);
                            umma_ss_pair(t_corr, al + sa, bh + sb, IDESC, 1u);
                        }
                        umma_commit_pair(&bars[P_EMPTY + s], 3u);
                        if (kb == kb1 - 1) umma_commit_pair(&bars[P_ACC_FULL + buf], 3u);
                    }
                    __syncwarp();
                    if (++s == (uint32_t)stages) { s = 0; ++turn; }
                }
            }
        }
    } else {
        // ------------------------------ epilogue ------------------------------
        const int lane_base = (warp & 3) * 32;
        const uint32_t t_lane = (uint32_t)lane_base << 16;
        const int ewg = (warp - 2) >> 2;                         // which share of the columns
        constexpr int CHUNKS = TN / 32 / p_epi_wg(TN);
        int n = 0;
        for (int u = u_first; u < u_end; u += u_step, ++n) {
            int tm, tn, kb0, kb1;
            unit(u, tm, tn, kb0, kb1);
            const int part = u % p.parts;
            const uint32_t buf = S::BUFS == 2 ? (uint32_t)n & 1u : 0u, use = S::BUFS == 2 ? (uint32_t)n >> 1 : (uint32_t)n;
            if (!__all_sync(0xffffffffu, mbar_wait(ws, &bars[P_ACC_FULL + buf], use & 1u, DEERS_KERR_GEMM | 0x47))) break;
            tc_fence_after_sync();
            float* cbase = p.c + (p.parts > 1 ? (long long)part * p.M * p.ldc : 0);
            const int first = tm * P_M + half * XM + lane_base, row0 = first + (lane & ~7);
            float st_m = -INFINITY, st_s = 0.f;
#pragma unroll 1
            for (int chunk = ewg * CHUNKS; chunk < (ewg + 1) * CHUNKS; ++chunk) {      // 32 columns at a time
                uint32_t rm[32], rc[32];
                tmem_ld_x32(tmem + buf * 256u + t_lane + chunk * 32, rm);
                tmem_ld_x32(tmem + buf * 256u + TN + t_lane + chunk * 32, rc);
                tmem_wait_ld();
                if (chunk == (ewg + 1) * CHUNKS - 1) {           // this warp's share of both accumulators is in registers
                    tc_fence_before_sync();
                    mbar_arrive_cluster_warp(cluster_addr(&bars[P_ACC_EMPTY + buf], 0));
                }
                float o[32];
#pragma unroll
                for (int e = 0; e < 32; ++e) o[e] = fmaf(__uint_as_float(rc[e]), X_LO, __uint_as_float(rm[e])) * p.out_scale;
                const int c0 = tn * TN + chunk * 32;
                if constexpr (TRANS) {
                    if (first + lane < p.M) {
                        float* dst = cbase + (long long)c0 * p.ldc + first + lane;
#pragma unroll
                        for (int e = 0; e < 32; ++e, dst += p.ldc)
                            if (c0 + e < p.N) *dst = o[e];
                    }
                } else if constexpr (!TURN) {
                    uint4 pc[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        pc[q] = make_uint4(__float_as_uint(o[q * 4]), __float_as_uint(o[q * 4 + 1]), __float_as_uint(o[q * 4 + 2]), __float_as_uint(o[q * 4 + 3]));
                    // 16-byte pieces transposed within 8-lane groups: a store instruction writes 128 contiguous bytes per row
                    transpose_pieces<8>(pc, (uint32_t)lane);
                    const int col = c0 + (lane & 7) * 4;
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const int row = row0 + c;
                        if (row >= p.M || col >= p.N) continue;
                        float* dst = cbase + (long long)row * p.ldc + col;
                        if (col + 4 <= p.N) {
                            *reinterpret_cast<uint4*>(dst) = pc[c];
                        } else {
                            const uint32_t v[4] = {pc[c].x, pc[c].y, pc[c].z, pc[c].w};
                            for (int e = 0; e < 4 && col + e < p.N; ++e) dst[e] = __uint_as_float(v[e]);
                        }
                    }
                } else {
                    // turned round in the warp's own 4 KB, a row per store instruction
                    float* turned = reinterpret_cast<float*>(smem + S::RING + 256) + (warp - 2) * 1024;
#pragma unroll
                    for (int e = 0; e < 32; ++e) turned[lane * 32 + (e ^ lane)] = o[e];
                    __syncwarp();
                    if (c0 + lane < p.N) {
#pragma unroll 8
                        for (int r = 0; r < 32; ++r)
                            if (first + r < p.M) cbase[(long long)(first + r) * p.ldc + c0 + lane] = turned[r * 32 + (lane ^ r)];
                    }
                    __syncwarp();
                }
                if constexpr (STATS) {
                    if (c0 + 32 > p.N) {
#pragma unroll
                        for (int e = 0; e < 32; ++e)
                            if (c0 + e >= p.N) o[e] = -INFINITY;
                    }
                    float m = o[0];
#pragma unroll
                    for (int e = 1; e < 32; ++e) m = fmaxf(m, o[e]);
                    const float both = fmaxf(st_m, m), ref = both == -INFINITY ? 0.f : both;       // (nothing but -inf: sums of zeros)
                    st_s = st_s * expf(st_m - ref) + x3_exp_sum(o, ref);
                    st_m = both;
                }
            }
            if constexpr (STATS)
                if (first + lane < p.M) p.stats[(long long)(tn * p_epi_wg(TN) + ewg) * p.M + first + lane] = make_float2(st_m, st_s);
        }
    }
    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    cg::this_cluster().sync();                                  // nobody leaves while its peer's loads or products still reach its memory
    if (warp == 1) tmem_dealloc_pair(tmem, 512);
}

// c[m][n] = sum over parts (in index order) of partial[part][m][n]; four at a time (N and ldc multiples of 4, 16-byte bases) or one by one, eight
// parts' loads on their way together (18 parts of 1024 x 192 take 5 us, as 9 did one by one).
template <typename V>
__global__ void __launch_bounds__(256) x3_reduce_kernel(const float* partial, int parts, long long MN,
                                                        int N, float* __restrict__ c, long long ldc) {
    chain_begin();
    constexpr int W = sizeof(V) / 4;
    for (long long i = ((long long)blockIdx.x * 256 + threadIdx.x) * W; i < MN; i += (long long)gridDim.x * 256 * W) {
        float acc[W];
#pragma unroll
        for (int e = 0; e < W; ++e) acc[e] = 0.f;
        for (int p0 = 0; p0 < parts; p0 += 8) {
            V v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (p0 + q < parts) v[q] = *reinterpret_cast<const V*>(partial + (long long)(p0 + q) * MN + i);
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (p0 + q < parts)
#pragma unroll
                    for (int e = 0; e < W; ++e) {
                        const float x = reinterpret_cast<const float*>(&v[q])[e];
                        acc[e] = p0 + q ? acc[e] + x : x;
                    }
        }
        V o;
#pragma unroll
        for (int e = 0; e < W; ++e) reinterpret_cast<float*>(&o)[e] = acc[e];
        *reinterpret_cast<V*>(c + (i / N) * ldc + (i % N)) = o;
    }
}

// hi = f16(x * s), lo = f16((x * s - hi) * 2^11); 8 elements per thread (16-byte loads and stores when aligned)
__global__ void __launch_bounds__(256) x3_split_kernel(const float* src, long long ld_src, long long rows, int cols,
                                                       float scale, __half* __restrict__ hi, __half* __restrict__ lo,
                                                       long long ld_dst, int vec) {
    chain_begin();
    const int per_row = (cols + 7) / 8;
    const long long total = rows * per_row;
    for (long long t = (long long)blockIdx.x * 256 + threadIdx.x; t < total; t += (long long)gridDim.x * 256) {
        const long long r = t / per_row;
        const int c0 = (int)(t % per_row) * 8;
        const float* s = src + r * ld_src + c0;
        float x[8];
        if (vec && c0 + 8 <= cols) {
            const float4 a = *reinterpret_cast<const float4*>(s), b = *reinterpret_cast<const float4*>(s + 4);
            x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = (c0 + e < cols) ? s[e] : 0.f;
        }
        __half h[8], l[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float v = x[e] * scale;
            h[e] = __float2half_rn(v);
            l[e] = __float2half_rn((v - __half2float(h[e])) * 2048.0f);
        }
        __half* dh = hi + r * ld_dst + c0;
        __half* dl = lo + r * ld_dst + c0;
        if (vec && c0 + 8 <= cols) {
            *reinterpret_cast<uint4*>(dh) = *reinterpret_cast<const uint4*>(h);
            *reinterpret_cast<uint4*>(dl) = *reinterpret_cast<const uint4*>(l);
        } else {
            for (int e = 0; e < 8 && c0 + e < cols; ++e) { dh[e] = h[e]; dl[e] = l[e]; }
        }
    }
}

// Tensor map over a row-major f16 matrix [rows][inner] with leading dimension ld (a multiple of 8 elements), as
// a 4-D map {inner, rows, 1, 1} with box {64, box_rows, 1, 1}, 128-byte swizzle, out-of-range elements read as zero.
int make_tmap_x3(deers_ctx* ctx, CUtensorMap* out, const void* base, long long rows, long long inner, long long ld, int box_rows) {
    if (!ctx->encode_tiled) {
        snprintf(ctx->last_error, sizeof(ctx->last_error), "cuTensorMapEncodeTiled not available");
        return DEERS_ERR_CUDA;
    }
    const cuuint64_t dims[4] = {(cuuint64_t)inner, (cuuint64_t)rows, 1, 1};
    const cuuint64_t row_bytes = (cuuint64_t)ld * 2;
    const cuuint64_t gstr[3] = {row_bytes, row_bytes * (cuuint64_t)rows, row_bytes * (cuuint64_t)rows};
    const cuuint32_t box[4] = {64u, (cuuint32_t)box_rows, 1u, 1u};
    const cuuint32_t estr[4] = {1u, 1u, 1u, 1u};
    const CUresult r = ((PFN_encodeTiled)ctx->encode_tiled)(
        out, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void*>(base), dims, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        snprintf(ctx->last_error, sizeof(ctx->last_error), "cuTensorMapEncodeTiled failed with CUresult %d (rows %lld, inner %lld, ld %lld)",
                 (int)r, rows, inner, ld);
        return DEERS_ERR_LAYOUT;
    }
    return DEERS_OK;
}

struct X3Plan {
    int parts, k_chunk;
    bool pair;                  // the rest: of pairs
    int tn;
    bool trans;
    int resident;
};

// K split for `tiles` tiles on `room` CTAs or pairs: all (tile, part) units in one wave, at least `least` K blocks per part.
void x3_split(X3Plan& pl, long long tiles, int K, int room, int least) {
    const int kblocks = (K + XK - 1) / XK;
    pl.parts = 1;
    pl.k_chunk = kblocks * XK;
    if (tiles >= room) return;
    int parts = (int)(room / tiles);
    const int max_parts = kblocks / least > 1 ? kblocks / least : 1;
    if (parts > max_parts) parts = max_parts;
    if (parts > 64) parts = 64;
    const int chunk_blocks = (kblocks + parts - 1) / parts;
    pl.k_chunk = chunk_blocks * XK;
    pl.parts = (kblocks + chunk_blocks - 1) / chunk_blocks;
}

// Single CTAs on 128 x 128, or pairs: for logits of many waves (1024 x 50257 x 192 77 -> 61 us, in the model with the row statistics 77 and no
// pass of 42 for them; 300 x 12000 x 320, two waves, 11.2 and 15.3), input gradients with long parts of K (1024 x 192 x 50257 87 -> 57) and weight
// gradients of many tokens (192 x 50257 x 1024 76 -> 56; of 300 tokens 11.2 and 14.7: one pair of accumulators, nothing beside its epilogue;
// 128 columns never leave fewer waves than single CTAs have).
X3Plan x3_plan(int M, int N, int K, int a_mn, int b_mn, int sm_count, int pairs) {
    X3Plan pl{};
    const int kblocks = (K + XK - 1) / XK;
    const long long tiles = (long long)((M + XM - 1) / XM) * ((N + XN - 1) / XN);
    x3_split(pl, tiles, K, sm_count, 8);                              // at least eight K blocks per part
    if (pairs < 1 || (a_mn && !b_mn)) return pl;
    const int m = a_mn ? N : M, n = a_mn ? M : N;                     // rows and columns of the pair's tiles
    const int wide = (n + 191) / 192 * 192, narrow = (n + 127) / 128 * 128, tn = !a_mn && b_mn ? 128 : wide <= narrow ? 192 : 128;
    const int rows = (m + P_M - 1) / P_M;
    const long long pair_tiles = (long long)rows * ((n + tn - 1) / tn);
    const long long waves = (tiles + sm_count - 1) / sm_count, pair_waves = (pair_tiles + pairs - 1) / pairs;
    if (m <= XM) return pl;                                           // one CTA of a pair would have nothing to do
    const bool by_pairs = a_mn   ? K >= 512 && tn == 192 && pair_waves < waves
                          : b_mn ? waves >= 6 && pair_waves <= waves
                                 : pl.k_chunk >= 16 * XK && N % 4 == 0;
    if (!by_pairs) return pl;
    pl = X3Plan{};
    pl.pair = true;
    pl.trans = a_mn != 0;
    pl.tn = tn;
    if (pl.trans) { pl.parts = 1; pl.k_chunk = kblocks * XK; }
    else x3_split(pl, pair_tiles, K, pairs, 8);
    // a pair keeps to one row of tiles: where that leaves more than one in twenty pairs idle A travels with B
    if (!a_mn && b_mn && pl.parts == 1 && kblocks <= P_RES_KB && rows <= pairs && pairs % rows * 20 <= pairs) pl.resident = kblocks;
    return pl;
}

size_t x3_partials(const X3Plan& pl, int M, int N) { return pl.parts > 1 ? (size_t)pl.parts * M * N * sizeof(float) : 0; }

// The plan of a call.  Input gradients by pairs store 16 bytes at a time; and the workspace may be one for single CTAs.
int x3_choose(deers_ctx* ctx, int M, int N, int K, int a_mn, int b_mn, bool rows16, size_t ws_bytes, int* pairs, X3Plan* pl) {
    const int rc = gemm_f16_pairs(ctx, pairs);
    if (rc) return rc;
    *pl = x3_plan(M, N, K, a_mn, b_mn, ctx->sm_count, *pairs);
    if (pl->pair && ((!a_mn && !b_mn && !rows16 && pl->parts == 1) || ws_bytes < x3_partials(*pl, M, N)))
        *pl = x3_plan(M, N, K, a_mn, b_mn, ctx->sm_count, 0);
    return DEERS_OK;
}

template <int A_MN, int B_MN>
int x3_launch(deers_ctx* ctx, const CUtensorMap* t, const X3Params& p, unsigned grid) {
    DEERS_SMEM_ONCE(ctx, (gemm_f16x3_kernel<A_MN, B_MN>), X_SMEM);
    {
        KernelTimerScope ts(ctx, DEERS_K_GEMM_X3);
        DEERS_CUDA_TRY(ctx, launch_chained(ctx, gemm_f16x3_kernel<A_MN, B_MN>, grid, X_THREADS, X_SMEM, 1, t[0], t[1], t[2], t[3], p));
    }
    ctx->launches += 1;
    DEERS_CUDA_TRY(ctx, cudaGetLastError());
    return DEERS_OK;
}

template <int A_MN, int B_MN, int TN, bool TRANS, bool STATS, bool TURN>
int x3_launch_pair(deers_ctx* ctx, const CUtensorMap* t, const X3PairParams& p, int pairs) {
    const auto kernel = gemm_f16x3_pair_kernel<A_MN, B_MN, TN, TRANS, STATS, TURN>;
    DEERS_SMEM_ONCE(ctx, (gemm_f16x3_pair_kernel<A_MN, B_MN, TN, TRANS, STATS, TURN>), p_smem(TURN));
    const long long units = (long long)((p.M + P_M - 1) / P_M) * ((p.N + TN - 1) / TN) * p.parts;
    const long long most = p.resident ? pairs / ((p.M + P_M - 1) / P_M) * ((p.M + P_M - 1) / P_M) : pairs;
    const unsigned grid = 2u * (unsigned)(units < most ? units : most);
    {
        KernelTimerScope ts(ctx, DEERS_K_GEMM_X3);
        DEERS_CUDA_TRY(ctx, launch_chained(ctx, kernel, grid, p_threads(TN), p_smem(TURN), 2, t[0], t[1], t[2], t[3], p));
    }
    ctx->launches += 1;
    return DEERS_OK;
}

int x3_reduce(deers_ctx* ctx, const float* partial, int parts, int M, int N, float* c, long long ldc) {
    const long long MN = (long long)M * N;
    const bool four = N % 4 == 0 && ldc % 4 == 0 && (((uintptr_t)c | (uintptr_t)partial) & 15u) == 0;
    const long long want = (MN / (four ? 4 : 1) + 255) / 256, cap = 8LL * ctx->sm_count;
    const auto kernel = four ? x3_reduce_kernel<float4> : x3_reduce_kernel<float>;
    {
        KernelTimerScope ts(ctx, DEERS_K_GEMM_X3);
        DEERS_CUDA_TRY(ctx, launch_chained(ctx, kernel, (unsigned)(want < cap ? want : cap), 256, 0, 1, partial, parts, MN, N, c, ldc));
    }
    ctx->launches += 1;
    return DEERS_OK;
}

}  // namespace

size_t gemm_f16x3_workspace_bytes(const deers_ctx* ctx, int M, int N, int K) {
    const int sms = ctx ? ctx->sm_count : 148;
    size_t most = 0;
    for (int pairs : {0, sms / 2})                                      // whichever of the two the product takes
        for (int b_mn = 0; b_mn <= 1; ++b_mn) {
            const X3Plan pl = x3_plan(M, N, K, 0, b_mn, sms, pairs);
            if (x3_partials(pl, M, N) > most) most = x3_partials(pl, M, N);
        }
    return most;
}

int route_gemm_f16x3(deers_ctx* ctx, int M, int N, int K, int a_mn, int b_mn, int rows16, deers_product_route* r) {
    X3Plan pl;
    int pairs = 0;
    const int rc = x3_choose(ctx, M, N, K, a_mn, b_mn, rows16 != 0, gemm_f16x3_workspace_bytes(ctx, M, N, K), &pairs, &pl);
    if (rc) return rc;
    r->tile_m = !pl.pair ? XM : pl.trans ? pl.tn : P_M; r->tile_n = !pl.pair ? XN : pl.trans ? P_M : pl.tn;
    r->parts = pl.parts; r->tensor_core = 1; r->pair = pl.pair; r->resident = pl.resident;
    return DEERS_OK;
}

int launch_split_f16x3(deers_ctx* ctx, long long rows, int cols, const float* src, long long ld_src, float scale,
                       void* hi, void* lo, long long ld_dst) {
    if (rows == 0 || cols == 0) return DEERS_OK;
    const int vec = (((uintptr_t)src | (uintptr_t)hi | (uintptr_t)lo) & 15u) == 0 && ld_src % 4 == 0 && ld_dst % 8 == 0;
    const long long total = rows * ((cols + 7) / 8);
    long long want = (total + 255) / 256;
    const long long cap = 16LL * ctx->sm_count;
    {
        KernelTimerScope ts(ctx, DEERS_K_GEMM_X3);
        DEERS_CUDA_TRY(ctx, launch_chained(ctx, x3_split_kernel, (unsigned)(want < cap ? want : cap), 256, 0, 1, src, ld_src, rows, cols, scale, (__half*)hi,
                                                                                      (__half*)lo, ld_dst, vec));
    }
    ctx->launches += 1;
    DEERS_CUDA_TRY(ctx, cudaGetLastError());
    return DEERS_OK;
}

int launch_gemm_f16x3(deers_ctx* ctx, int M, int N, int K, const void* a_hi, const void* a_lo, long long lda, int a_mn,
                      const void* b_hi, const void* b_lo, long long ldb, int b_mn, float* c, long long ldc, float out_scale,
                      void* workspace, size_t ws_bytes, float2* stats, int* stat_parts) {
    if (stat_parts) *stat_parts = 0;
    if (M == 0 || N == 0) return DEERS_OK;
    CUtensorMap t[4];
    X3Plan pl;
    const bool rows16 = ldc % 4 == 0 && ((uintptr_t)c & 15u) == 0;
    int pairs = 0, rc = x3_choose(ctx, M, N, K, a_mn, b_mn, rows16, workspace ? ws_bytes : 0, &pairs, &pl);
    if (rc) return rc;
    const bool split = pl.parts > 1;
    if (split && (!workspace || ws_bytes < x3_partials(pl, M, N) || ((uintptr_t)workspace & 15u))) return DEERS_ERR_WORKSPACE;
    float* out = split ? (float*)workspace : c;
    const long long ldo = split ? N : ldc;
    const int vec = ldo % 4 == 0 && ((uintptr_t)out & 15u) == 0;
    const void* ap[2] = {a_hi, a_lo};
    const void* bp[2] = {b_hi, b_lo};
    if (pl.pair && pl.trans) {                                          // C^T = B^T A: the pair's rows are the caller's columns
        const void* tp[2] = {ap[0], ap[1]};
        for (int h = 0; h < 2; ++h) { ap[h] = bp[h]; bp[h] = tp[h]; }
        const long long tl = lda; lda = ldb; ldb = tl;
    }
    const int m = pl.trans ? N : M, n = pl.trans ? M : N;
    // K-major operand: [rows = M or N][inner = K], boxes of 64 K by the rows a CTA brings; MN-major: [rows = K][inner = M or N], box {64, 64}
    for (int h = 0; h < 2; ++h) {
        if ((rc = a_mn ? make_tmap_x3(ctx, &t[h], ap[h], K, m, lda, XK) : make_tmap_x3(ctx, &t[h], ap[h], m, K, lda, XM))) return rc;
        const int b_rows = pl.pair ? pl.tn / 2 : XN;
        if ((rc = b_mn ? make_tmap_x3(ctx, &t[2 + h], bp[h], K, n, ldb, XK) : make_tmap_x3(ctx, &t[2 + h], bp[h], n, K, ldb, b_rows))) return rc;
    }
    if (pl.pair) {
        X3PairParams p;
        p.c = out; p.ldc = ldo; p.M = m; p.N = n; p.K = K; p.parts = pl.parts; p.k_chunk = pl.k_chunk; p.out_scale = out_scale;
        p.resident = pl.resident; p.stats = stats; p.err = ctx->dev_err;
        if (pl.trans) rc = x3_launch_pair<1, 1, 192, true, false, false>(ctx, t, p, pairs);
        else if (!b_mn) rc = pl.tn == 192 ? x3_launch_pair<0, 0, 192, false, false, false>(ctx, t, p, pairs)
                                          : x3_launch_pair<0, 0, 128, false, false, false>(ctx, t, p, pairs);
        else if (!vec) rc = x3_launch_pair<0, 1, 128, false, false, true>(ctx, t, p, pairs);
        else if (stats && !split) {
            rc = x3_launch_pair<0, 1, 128, false, true, false>(ctx, t, p, pairs);
            *stat_parts = p_epi_wg(128) * ((n + 127) / 128);
        } else rc = x3_launch_pair<0, 1, 128, false, false, false>(ctx, t, p, pairs);
    } else {
        X3Params p;
        p.M = M; p.N = N; p.K = K; p.parts = pl.parts; p.k_chunk = pl.k_chunk; p.err = ctx->dev_err;
        p.c = out; p.ldc = ldo; p.out_scale = out_scale; p.vec = vec;
        const long long units = (long long)((M + XM - 1) / XM) * ((N + XN - 1) / XN) * pl.parts;
        const unsigned grid = (unsigned)(units < ctx->sm_count ? units : ctx->sm_count);
        if (a_mn) rc = b_mn ? x3_launch<1, 1>(ctx, t, p, grid) : x3_launch<1, 0>(ctx, t, p, grid);
        else rc = b_mn ? x3_launch<0, 1>(ctx, t, p, grid) : x3_launch<0, 0>(ctx, t, p, grid);
    }
    if (rc || !split) return rc;
    return x3_reduce(ctx, (const float*)workspace, pl.parts, M, N, c, ldc);
}

extern "C" int deers_b200_split_f16x3(deers_ctx* ctx, int64_t rows, int32_t cols, const float* src, int64_t ld_src, float scale,
                                      void* hi, void* lo, int64_t ld_dst) {
    if (!ctx || !src || !hi || !lo) return DEERS_ERR_NULL;
    if (rows < 0 || cols < 0) return DEERS_ERR_SHAPE;
    if (ld_src < cols || ld_dst < cols || ((uintptr_t)src & 3u) || (((uintptr_t)hi | (uintptr_t)lo) & 1u)) return DEERS_ERR_LAYOUT;
    if (!(scale > 0.f)) return DEERS_ERR_SHAPE;
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    return launch_split_f16x3(ctx, rows, cols, src, ld_src, scale, hi, lo, ld_dst);
}

extern "C" size_t deers_b200_gemm_f16x3_workspace_bytes(deers_ctx* ctx, int32_t M, int32_t N, int32_t K) {
    if (!ctx || M < 0 || N < 0 || K < 0) return 0;
    return gemm_f16x3_workspace_bytes(ctx, M, N, K);
}

extern "C" int deers_b200_gemm_f16x3(deers_ctx* ctx, int32_t M, int32_t N, int32_t K, const void* a_hi, const void* a_lo,
                                     int64_t lda, int32_t a_mn_major, const void* b_hi, const void* b_lo, int64_t ldb,
                                     int32_t b_mn_major, float* c, int64_t ldc, float out_scale, void* workspace,
                                     size_t workspace_bytes) {
    if (!ctx || !a_hi || !a_lo || !b_hi || !b_lo || !c) return DEERS_ERR_NULL;
    if (M < 1 || N < 1 || K < 1) return DEERS_ERR_SHAPE;
    // 16-byte rows for TMA (f16 operands) and for the epilogue's 16-byte stores (f32 output)
    if ((lda % 8) || (ldb % 8) || (ldc % 4) || lda < (a_mn_major ? M : K) || ldb < (b_mn_major ? N : K) || ldc < N)
        return DEERS_ERR_LAYOUT;
    if (((uintptr_t)a_hi | (uintptr_t)a_lo | (uintptr_t)b_hi | (uintptr_t)b_lo | (uintptr_t)c) & 15u) return DEERS_ERR_LAYOUT;
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    return launch_gemm_f16x3(ctx, M, N, K, a_hi, a_lo, lda, a_mn_major, b_hi, b_lo, ldb, b_mn_major, c, ldc, out_scale, workspace,
                             workspace_bytes, nullptr, nullptr);
}
