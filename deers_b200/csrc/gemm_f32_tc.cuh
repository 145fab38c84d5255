// A tile of an f32 GEMM on the tensor core without the loss of f32: every operand value is three bf16,
//     x = h + m 2^-8 + l 2^-16,    h = bf16(x), m = bf16((x - h) 2^8), l = bf16(((x - h) 2^8 - m) 2^8)
// (all 24 bits: the remainders are exact, and the tensor core keeps subnormal bf16, so the parts reach down to f32's 2^-149; unscaled
// ones would end at 2^-133) and a product is the six of their nine products that reach 2^-24:
//     main += Ah Bh          corr1 += Ah Bm + Am Bh          corr2 += Ah Bl + Am Bm + Al Bh          C = main + corr1 2^-8 + corr2 2^-16
// The tensor core rounds its sums towards zero, which a long walk in one accumulator shows (two f16 per value and one accumulator:
// 2-norm error 2.8e-7 at K = 192, all positive 8e-7, where FFMA sums have 1.3e-7 and 7e-8).  So `main` starts anew with every 16 k, in
// columns of its own, and these sums are added in f32, rounded to nearest, by the threads that take them out; the
// corrections are 2^-8 of it and smaller and may run on.  2-norm errors against 64 bits, FFMA kernels and these: normal operands K = 192 1.3e-7
// and 5.8e-8, K = 768 1.4e-7 and 7.0e-8, K = 1024 2.1e-7 and 7.3e-8; all positive K = 192 6.3e-8 and 4.5e-8, K = 768 4.6e-8 and 4.3e-8
// (every 32 k instead: 6.2e-8 and 5.6e-8).
// A block works its tile out again with FFMA sums (plain_tile) where these cannot stand for them:
//   - a sum that is not finite: bf16 has the exponents of f32, but values from 2^128 - 2^119 on round to an infinity, a correction may overflow
//     ahead of its whole, and 0 * inf must not appear where x * y has none.  An h that is not finite makes every sum of its row or column such;
//   - subnormal operands that a result rests on: their h, and below 2^-134 their m, holds few bits or none, and the three products left
//     out, 1.5 2^-151 of the other operand at most, are then not 2^-24 of the result but 4e-6 at 2^-134 and 2e-3 at 2^-146.  Sums of 2^-120
//     times the largest value of either operand or more have them below 2^-24 whatever K, so only smaller ones (not zeros) make the block
//     look for subnormal operands.
//
// A block owns a tile of 128 x 64: 512 threads load, split and store a stage of 64 k (128-byte swizzle, in the operand's own storage
// order) while the products of the stage before run and the one after is on its way.  Blocks of a cluster share a long K and
// meet as those of gemm_f32_kernel do; norm, rotation and epilogues are the same code.
// What bounds it: shared memory, 185 KB a stage stored and read by the products (1470 cycles of its 128 bytes; the products take 900, the
// conversions 700 issue slots), around it launch, first load and the way out;
// 2500 cycles a stage as it is, because the sums of a stage are taken out between its products and the next one's.
// In a graph, FFMA kernels and these (us): 1024 x 768 x 192 10.9 -> 7.7, 1024 x 192 x 768 12.8 -> 9.1, 1024 x 192 x 576 12.2 -> 8.3,
// 4096 x 768 x 192 40 -> 22, 1024 x 1152 x 384 27 -> 12.
#pragma once
#include "gemm_f32_kernel.cuh"
#include "sm100_ptx.cuh"

namespace {
using namespace sm100;

constexpr int TC_M = 128, TC_N = 64, TC_RING = 3;             // a tile; stages of 64 k
constexpr int TC_T = 512;
constexpr uint32_t TC_A = 128 * 128, TC_B = 64 * 128;            // one of the three parts of a stage's A, B: 64 k
constexpr uint32_t TC_STAGE = 3 * (TC_A + TC_B);
constexpr uint32_t TC_BLOCK = 64 * 128;                          // MN order: 64 k by 64 columns
constexpr uint32_t TC_SQ = TC_RING * TC_STAGE;                 // rows' sums of squares
constexpr uint32_t TC_BARS = TC_SQ + 2 * TC_M * 4;               // (and the inverse norms)
constexpr uint32_t TC_SMEM = TC_BARS + 64;                      // a barrier per stage, TMEM base, abort flag
static_assert(TC_M * (TC_N + 4) * 4 <= TC_SQ && TC_SMEM <= 232448, "shared memory");
// TMEM columns: main of a stage's four steps of 16 k | corr1 | corr2
constexpr uint32_t TC_C1 = 4 * TC_N, TC_C2 = TC_C1 + TC_N;
static_assert(TC_C2 + TC_N <= 512, "TMEM");

// Eight consecutive floats of which `valid` exist (p on a 16-byte boundary).
__device__ __forceinline__ void load8(float (&x)[8], const float* p, int valid) {
    if (valid >= 8) {
        const float4 u = *reinterpret_cast<const float4*>(p), v = *reinterpret_cast<const float4*>(p + 4);
        x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w; x[4] = v.x; x[5] = v.y; x[6] = v.z; x[7] = v.w;
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = e < valid ? p[e] : 0.f;
    }
}

__device__ __forceinline__ uint32_t bf16x2(float lo, float hi) {
    uint32_t v;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(v) : "f"(hi), "f"(lo));
    return v;
}

// What two values' parts leave, times 2^8.
__device__ __forceinline__ void remainders(float& a, float& b, float fa, float fb) {
    unpack_f32x2(mul2(fma2(pack_f32x2(fa, fb), pack_f32x2(-1.f, -1.f), pack_f32x2(a, b)), pack_f32x2(256.f, 256.f)), a, b);
}

// What `large` adds up of the h: not finite any more when one of them is 2^25 or more (or several come near).
constexpr float TC_LARGE = 0x1p104f;
// The bits of 2^-95 and 2^8: 2^-120 of values below 2^25, and of any.
constexpr uint32_t TC_SMALL_SUM = (127u - 95u) << 23, TC_SMALL_SUM_OF_LARGE = (127u + 8u) << 23;

// Splits eight values and stores the three parts, `part` bytes apart.
__device__ __forceinline__ void split8(uint8_t* dst, uint32_t part, const float (&x)[8], float& large) {
    uint32_t w[3][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        float a = x[2 * e], b = x[2 * e + 1];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            w[q][e] = bf16x2(a, b);
            if (q == 2) break;
            const float fa = __uint_as_float(w[q][e] << 16), fb = __uint_as_float(w[q][e] & 0xffff0000u);
            if (q == 0) large = fmaf(fa, TC_LARGE, fmaf(fb, TC_LARGE, large));
            remainders(a, b, fa, fb);
        }
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(dst + q * part) = make_uint4(w[q][0], w[q][1], w[q][2], w[q][3]);
}

// The same for two values.
__device__ __forceinline__ void split2(uint8_t* dst, uint32_t part, float a, float b, float& large) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const uint32_t w = bf16x2(a, b);
        *reinterpret_cast<uint32_t*>(dst + q * part) = w;
        const float fa = __uint_as_float(w << 16), fb = __uint_as_float(w & 0xffff0000u);
        if (q == 0) large = fmaf(fa, TC_LARGE, fmaf(fb, TC_LARGE, large));
        remainders(a, b, fa, fb);
    }
}

// How the 512 threads take a stage of one operand, R rows of L floats (rows: m, n in K order, k in MN order) of which rv rows and lv floats
// exist, from global memory and, split, into shared memory.
// Rows on 16-byte boundaries go by eights.  Rows on any boundary go by twos, neighbouring lanes side by side: a warp's load touches 8 sectors
// where single floats of eights would touch 32 (2133 x 769 x 1405 68 us; FFMA kernels 146).
template <int R, int L, bool LOOSE>
struct TcOperand {
    static constexpr int W = LOOSE ? 2 : 8;                        // floats of a piece
    static constexpr int PIECES = R * L / W / TC_T, PER_ROW = L / W, ROW_STEP = TC_T / PER_ROW;
    static_assert(PIECES * TC_T * W == R * L && TC_T % PER_ROW == 0 && ROW_STEP % 8 == 0, "whole pieces, swizzled alike");
    static constexpr int FLOATS = PIECES * W;
    const float* p;
    int row, col;                                                  // of the thread's first piece; the others lie ROW_STEP rows apart
    uint32_t at;                                                   // its place in shared memory
    __device__ __forceinline__ void init(const float* base, long long ld) {
        row = (int)threadIdx.x / PER_ROW; col = (int)threadIdx.x % PER_ROW * W;
        p = base + row * ld + col;
        at = (uint32_t)(col / 64) * TC_BLOCK + sw128_chunk_offset(row, col % 64 / 8) + (uint32_t)(col % 8) * 2u;
    }
    __device__ __forceinline__ void load(float (&x)[FLOATS], long long ld, int rv, int lv) const {
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            const float* q = p + (long long)(i * ROW_STEP) * ld;
            const int valid = row + i * ROW_STEP < rv ? lv - col : 0;
            if constexpr (LOOSE) {
                x[2 * i] = valid > 0 ? q[0] : 0.f;
                x[2 * i + 1] = valid > 1 ? q[1] : 0.f;
            } else {
                load8(reinterpret_cast<float(&)[8]>(x[8 * i]), q, valid);
            }
        }
    }
    __device__ __forceinline__ void store(uint8_t* s, uint32_t part, const float (&x)[FLOATS], float& large) const {
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            if constexpr (LOOSE) {
                split2(s + at + i * ROW_STEP * 128u, part, x[2 * i], x[2 * i + 1], large);
            } else {
                split8(s + at + i * ROW_STEP * 128u, part, reinterpret_cast<const float(&)[8]>(x[8 * i]), large);
            }
        }
    }
};

// Whether this thread's share of a piece of an operand, `rows` rows of `len` floats, holds a subnormal value.
__device__ __forceinline__ bool subnormals(const float* p, long long ld, int rows, int len) {
    bool any = false;
    for (int r = threadIdx.x / 32; r < rows; r += TC_T / 32)
        for (int i = threadIdx.x % 32; i < len; i += 32) {
            const float x = p[r * ld + i];
            any |= x != 0.f && fabsf(x) < 0x1p-126f;
        }
    return any;
}

// The tile's sums by FFMA, four to an element as the FFMA kernels' groups have them.  a, b: the first values; rows, cols: those there are.
template <bool A_MN, bool B_MN>
__device__ __forceinline__ void plain_tile(float* red, const float* a, long long lda, const float* b, long long ldb, int rows, int cols, int klen) {
    for (int i = threadIdx.x; i < TC_M * TC_N; i += TC_T) {
        const int row = i / TC_N, col = i % TC_N;
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        if (row < rows && col < cols) {
            const float* pa = a + (A_MN ? row : row * lda);
            const float* pb = b + (B_MN ? col : col * ldb);
            for (int k = 0; k < klen; k += 4) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (k + e < klen) acc[e] = fmaf(pa[(k + e) * (A_MN ? lda : 1)], pb[(k + e) * (B_MN ? ldb : 1)], acc[e]);
            }
        }
        red[row * (TC_N + 4) + col] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
    }
}

// The part of the start that needs nothing of global memory.
__device__ __forceinline__ void gemm_f32_tc_prologue() {
    extern __shared__ __align__(1024) uint8_t tc_smem[];
    uint64_t* done = reinterpret_cast<uint64_t*>(tc_smem + TC_BARS);
    uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(done + TC_RING);
    if (threadIdx.x == 0) {
        tmem_base_s[1] = 0;                                       // the abort flag
        for (int s = 0; s < TC_RING; ++s) mbar_init(&done[s], 1);
        fence_barrier_init();
    }
    if (uniform((int)threadIdx.x / 32) == 1) {
        tmem_alloc(tmem_base_s, 512);
        tmem_relinquish();
    }
}

template <bool A_MN, bool B_MN, bool FUSED, bool LOOSE>
__device__ __forceinline__ void gemm_f32_tc_tile(const GemmArgs& g, const int tile_m, const int tile_n, const int part, const int parts,
                                                 unsigned int* err) {
    extern __shared__ __align__(1024) uint8_t tc_smem[];
    uint64_t* done = reinterpret_cast<uint64_t*>(tc_smem + TC_BARS);
    uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(done + TC_RING);
    float* sq_s = reinterpret_cast<float*>(tc_smem + TC_SQ);
    const int t = threadIdx.x, warp = uniform(t / 32), lane = t % 32;
    const int m0 = tile_m * TC_M, n0 = tile_n * TC_N;
    const int kbeg = part * g.k_chunk, klen = min(g.K - kbeg, g.k_chunk);      // at least 1
    const int stages = (klen + 63) / 64;

    using OA = TcOperand<A_MN ? 64 : TC_M, A_MN ? TC_M : 64, LOOSE>;
    using OB = TcOperand<B_MN ? 64 : TC_N, B_MN ? TC_N : 64, LOOSE>;
    static_assert(!(FUSED && (A_MN || LOOSE)), "the rows' squares are summed over eight lanes");
    OA oa;
    OB ob;
    oa.init(g.a + (A_MN ? (long long)kbeg * g.lda + m0 : (long long)m0 * g.lda + kbeg), g.lda);
    ob.init(g.b + (B_MN ? (long long)kbeg * g.ldb + n0 : (long long)n0 * g.ldb + kbeg), g.ldb);
    struct Stage { float of_a[OA::FLOATS], of_b[OB::FLOATS]; } x0, x1;   // of two stages: one is split while the next is on its way
    int kl = klen;                                                 // k from the stage to load on
    auto load = [&](Stage& x) {
        oa.load(x.of_a, g.lda, A_MN ? kl : g.M - m0, A_MN ? g.M - m0 : kl);
        ob.load(x.of_b, g.ldb, B_MN ? kl : g.N - n0, B_MN ? g.N - n0 : kl);
        oa.p += A_MN ? 64 * g.lda : 64;
        ob.p += B_MN ? 64 * g.ldb : 64;
        kl -= 64;
    };
    load(x0);
    if (stages > 1) load(x1);
    tc_fence_before_sync();
    __syncthreads();                                               // barrier and tensor memory are there
    tc_fence_after_sync();
    const uint32_t tmem = (uint32_t)uniform((int)*tmem_base_s);

    // Out of tensor memory: a warp takes 32 rows and 16 columns, after each stage the sums of its steps.
    const int out_row = (warp & 3) * 32 + lane, out_col = (warp >> 2) * 16;
    const uint32_t t_out = tmem + ((uint32_t)((warp & 3) * 32) << 16) + out_col;
    WaitState ws{reinterpret_cast<volatile uint32_t*>(tmem_base_s + 1), err};
    float sum[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) sum[e] = 0.f;
    // The sums of the last stage issued.  slot: its place in the ring; phase: of that place's barrier.
    int slot = 0, left = klen;                           // left: k from the present stage on
    uint32_t phase = 0;
    auto drain = [&](int steps, bool last) {
        mbar_wait(ws, &done[slot], phase, DEERS_KERR_GEMM | 0x31);
        __syncwarp();
        tc_fence_after_sync();
        uint32_t u[4][16];
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
            if (ks < steps) {
                tmem_ld_x16(t_out + (uint32_t)ks * TC_N, u[ks]);
            } else {
#pragma unroll
                for (int e = 0; e < 16; ++e) u[ks][e] = 0;
            }
        }
        tmem_wait_ld();
        float v[16];
#pragma unroll
        for (int e = 0; e < 16; ++e)                               // pairs first: fewer roundings at the size of the whole
            v[e] = (__uint_as_float(u[0][e]) + __uint_as_float(u[1][e])) + (__uint_as_float(u[2][e]) + __uint_as_float(u[3][e]));
        if (last) {
            tmem_ld_x16(t_out + TC_C1, u[0]);
            tmem_ld_x16(t_out + TC_C2, u[1]);
            tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = fmaf(fmaf(__uint_as_float(u[1][e]), 0x1p-8f, __uint_as_float(u[0][e])), 0x1p-8f, v[e]);
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) sum[e] += v[e];
        tc_fence_before_sync();
    };

    float large = 0.f, sq[2] = {0.f, 0.f};
    // The place a stage takes is free: the products of the one three before have been waited for (drain).
    auto stage = [&](int s, Stage& x) {
        const int now = s == 0 ? 0 : slot == TC_RING - 1 ? 0 : slot + 1;
        uint8_t* st = tc_smem + now * TC_STAGE;
        oa.store(st, TC_A, x.of_a, large);
        ob.store(st + 3 * TC_A, TC_B, x.of_b, large);
        if constexpr (FUSED) {
#pragma unroll
            for (int e = 0; e < OA::FLOATS; ++e) sq[e / 8] = fmaf(x.of_a[e], x.of_a[e], sq[e / 8]);
        }
        if (s + 2 < stages) load(x);
        fence_proxy_async_smem();
        if (s > 0) {
            drain(4, false);                                       // frees the columns, which this stage uses again
            if (now == 0) phase ^= 1u;
            left -= 64;
        }
        slot = now;
        __syncthreads();
        if (warp == 0) {
            tc_fence_after_sync();
            constexpr uint32_t ID64 = idesc_bf16(TC_M, TC_N, A_MN, B_MN), ID128 = idesc_bf16(TC_M, 2 * TC_N, A_MN, B_MN);
            const uint32_t s0 = (uint32_t)uniform((int)smem_u32(st));
            const uint64_t a = A_MN ? desc_mnmajor(s0, 0, TC_BLOCK) : desc_kmajor(s0, 0, 0);
            const uint64_t b = B_MN ? desc_mnmajor(s0 + 3 * TC_A, 0, TC_BLOCK) : desc_kmajor(s0 + 3 * TC_A, 0, 0);
            const int steps = min(4, (left + 15) / 16);
            if (elect_one()) {
#pragma unroll
                for (int ks = 0; ks < 4; ++ks) {
                    if (ks < steps) {
                        const uint64_t ah = a + (A_MN ? mnmajor_step(ks) : kmajor_step(ks, 0));
                        const uint64_t bh = b + (B_MN ? mnmajor_step(ks) : kmajor_step(ks, 0));
                        const uint64_t am = ah + (TC_A >> 4), al = am + (TC_A >> 4), bm = bh + (TC_B >> 4);
                        umma_ss(tmem + (uint32_t)ks * TC_N, ah, bh, ID64, 0u);
                        umma_ss(tmem + TC_C1, ah, bm, ID128, s + ks > 0);              // h m | h l  (the parts of B follow one another)
                        umma_ss(tmem + TC_C1, am, bh, ID128, 1u);                      // m h | m m
                        umma_ss(tmem + TC_C2, al, bh, ID64, 1u);                       // l h
                    }
                }
                umma_commit(&done[slot]);
            }
            __syncwarp();
        }
    };
    for (int s = 0; s < stages; s += 2) {
        stage(s, x0);
        if (s + 1 < stages) stage(s + 1, x1);
    }
    if constexpr (FUSED) {                                         // eight lanes share a row
#pragma unroll
        for (int i = 0; i < 2; ++i) {
#pragma unroll
            for (int o = 1; o < 8; o *= 2) sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], o);
            if (lane % 8 == 0) sq_s[oa.row + i * OA::ROW_STEP] = sq[i];
        }
    }
    drain(min(4, (left + 15) / 16), true);
    float* red = reinterpret_cast<float*>(tc_smem);                // every product has read its operands
#pragma unroll
    for (int e = 0; e < 16; e += 4)
        *reinterpret_cast<float4*>(red + out_row * (TC_N + 4) + out_col + e) = make_float4(sum[e], sum[e + 1], sum[e + 2], sum[e + 3]);
    float finite = 0.f;
    uint32_t least = 0xffffffffu;                                  // of the sums' magnitudes but zeros: twice the bits less one
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        finite = fmaf(sum[e], 0.f, finite);
        least = min(least, 2u * __float_as_uint(sum[e]) - 1u);
    }
    bool again = !(finite == 0.f);
    const bool of_large = !(fabsf(large) < INFINITY);
    const bool look = __syncthreads_or(again || of_large || least < 2u * TC_SMALL_SUM - 1u) != 0;
    if (warp == 1) tmem_dealloc(tmem, 512);
    if (look) {
        const float* a = g.a + (A_MN ? (long long)kbeg * g.lda + m0 : (long long)m0 * g.lda + kbeg);
        const float* b = g.b + (B_MN ? (long long)kbeg * g.ldb + n0 : (long long)n0 * g.ldb + kbeg);
        const int rows = min(TC_M, g.M - m0), cols = min(TC_N, g.N - n0);
        const uint32_t limit = __syncthreads_or(of_large) ? TC_SMALL_SUM_OF_LARGE : TC_SMALL_SUM;
        if (__syncthreads_or(least < 2u * limit - 1u))
            again |= subnormals(a, g.lda, A_MN ? klen : rows, A_MN ? rows : klen) || subnormals(b, g.ldb, B_MN ? klen : cols, B_MN ? cols : klen);
        if (__syncthreads_or(again)) {
            plain_tile<A_MN, B_MN>(red, a, g.lda, b, g.ldb, rows, cols, klen);
            __syncthreads();
        }
    }
    finish_tile<TC_M, TC_N, 1, TC_T, FUSED>(g, red, sq_s, m0, n0, parts, part);
}

template <bool A_MN, bool B_MN, bool FUSED, bool LOOSE>
__global__ void __launch_bounds__(TC_T, 1) gemm_f32_tc_kernel(const GemmArgs g, unsigned int* err) {
    gemm_f32_tc_prologue();
    chain_wait();
    gemm_f32_tc_tile<A_MN, B_MN, FUSED, LOOSE>(g, blockIdx.y, blockIdx.x, blockIdx.z, gridDim.z, err);
}

template <bool A_MN, bool B_MN, bool FUSED, bool LOOSE>
int launch_tc_order(deers_ctx* ctx, int parts, const GemmArgs& g) {
    const auto kernel = gemm_f32_tc_kernel<A_MN, B_MN, FUSED, LOOSE>;
    DEERS_SMEM_ONCE(ctx, (gemm_f32_tc_kernel<A_MN, B_MN, FUSED, LOOSE>), TC_SMEM);
    const dim3 grid((g.N + TC_N - 1) / TC_N, (g.M + TC_M - 1) / TC_M, parts);
    DEERS_CUDA_TRY(ctx, launch_chained(ctx, kernel, grid, TC_T, TC_SMEM, dim3(1, 1, parts), g, ctx->dev_err));
    return DEERS_OK;
}

template <bool LOOSE>
int launch_tc_orders(deers_ctx* ctx, int parts, const GemmArgs& g, int a_mn, int b_mn) {
    if (a_mn) return b_mn ? launch_tc_order<true, true, false, LOOSE>(ctx, parts, g) : launch_tc_order<true, false, false, LOOSE>(ctx, parts, g);
    return b_mn ? launch_tc_order<false, true, false, LOOSE>(ctx, parts, g) : launch_tc_order<false, false, false, LOOSE>(ctx, parts, g);
}

}  // namespace
