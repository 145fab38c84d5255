// Kernels of the f32 causal attention for sm_100a: FFMA register tiling, no tensor cores and no
// TF32, so that the result holds 1e-4 against the CPU path of the reference
// (src/storage/cpu.rs:688-791 of deers).  Forward is one pass with an online softmax; backward recomputes P
// from the saved lse and has two kinds of blocks in one launch, neither with atomics: key-tile-stationary ones own
// dK/dV, query-tile-stationary ones own dQ.  All take [B,H,T,D] strides, so no compaction copy is needed around them.
//
// What bounds it: at the model's sizes (24 slices of 256 x 32) the arithmetic is 2 us of the chip's FFMA time; the
// rest is the length of one block's walk.  So a block owns few rows (32 or less) and splits its walk: NG groups of two
// warps take every NG-th tile of the other side, each with its own softmax state (or gradient sums) and its own
// tiles in shared memory, and meet once at the end in group order.  A group never waits for another: its two
// warps meet at a named barrier, and the P / dS tile a product reads was written by the same warp.
// Within a group thread (ty, tx) of 8 x 8 owns RM rows RM ty .. and columns tx, tx + 8, ... of an 8 RM x BN score tile
// (4 x 8 or 4 x 4 patches with RM = 4: 12 LDS.128 per 128 FFMA) and the same rows with float4 columns 4 tx + 32 j of the
// accumulators.  RM = 2 and 1, blocks of 16 and 8 rows, are for calls of few blocks: each walks in half or a quarter of the time on SMs
// that would idle, and every row is summed in the same order (B3 H4 T77 D48 forward 6.7 -> 4.6 -> 3.9 us, backward 13.6 -> 8.2; B1 H6 T100 D32
// forward 4.9 -> 3.5 -> 2.9; the rules: attn_f32.cu).  Second products run two to an issue slot (forward, and from 64 wide tiles on backward;
// score products from 96), and lanes lie so that shared-memory reads cost half.  Tiles arrive by cp.async: the next K (or Q) is fetched while
// the current one's scores are turned into the second product, the next V (or dO) while the next scores are computed.  B8 H12 T2048 D64 forward
// 1909 -> 1688 us, backward 5821 -> 5642; B3 H4 T77 D48 forward 10.3 -> 6.8.
#pragma once
#include "common.cuh"
#include "f32_util.cuh"

#include <type_traits>

struct Strides3 { long long b, h, t; };

struct F32Params {
    const float* q; const float* k; const float* v; const float* o; const float* d_o;
    float* out_o; float* lse_out; const float* lse;
    float* dq; float* dk; float* dv;
    Strides3 sq, sk, sv, so, sdo, sdq, sdk, sdv;
    int B, H, T, D;
    int causal;
    int vec;            // 1: every row start of the inputs is 16-byte aligned and D % 4 == 0
    int vec_out;        // the same for the outputs
    float scale;
    const float* cosv; const float* sinv;   // backward: dQ and dK leave rotated back by their position ([T][D / 2]; nullptr: not)
};

// Blocks of 16 or 8 stationary rows (attn_f32_few.cuh), by tile width.
int launch_attn_fwd_f32_few32(deers_ctx* ctx, const F32Params& p, int groups, int stream, int rm);
int launch_attn_bwd_f32_few32(deers_ctx* ctx, const F32Params& p, int groups, int rm);
int launch_attn_fwd_f32_few64(deers_ctx* ctx, const F32Params& p, int groups, int stream, int rm);
int launch_attn_bwd_f32_few64(deers_ctx* ctx, const F32Params& p, int groups, int rm);
int launch_attn_fwd_f32_few96(deers_ctx* ctx, const F32Params& p, int groups, int stream, int rm);
int launch_attn_bwd_f32_few96(deers_ctx* ctx, const F32Params& p, int groups, int rm);
int launch_attn_fwd_f32_few128(deers_ctx* ctx, const F32Params& p, int groups, int stream, int rm);
int launch_attn_bwd_f32_few128(deers_ctx* ctx, const F32Params& p, int groups, int rm);

namespace {

constexpr float LOG2E = 1.4426950408889634f;
constexpr float LN2 = 0.6931471805599453f;

// Place of a thread in its group's 8 x 8 arrangement.  A quarter warp holds two rows and four columns, neighbouring lanes a
// column each: a 16-byte shared-memory read along either side then costs 2.1 cycles (4 with lane % 8 along the columns).
__device__ __forceinline__ int place_y(int t) { return (t / 32) * 4 + (t & 1) + 2 * ((t >> 3) & 1); }
__device__ __forceinline__ int place_x(int t) { return ((t >> 1) & 3) + 4 * ((t >> 4) & 1); }
// The two warps of a group meet (barrier 0 is __syncthreads).
__device__ __forceinline__ void group_sync(int g) { asm volatile("bar.sync %0, 64;" ::"r"(g + 1) : "memory"); }

// Enqueues rows [row0, row0 + ROWS) x [0, DP) of a [T, D] matrix for shared memory (row stride DP + 4), zeros
// beyond T and D; COUNT threads of index t share the pieces.
template <int DP, int ROWS, int COUNT>
__device__ __forceinline__ void fetch_tile(float* __restrict__ dst, const float* __restrict__ src, int row0, int T, int D,
                                           long long st, int vec, int t) {
    constexpr int C4 = DP / 4;
    constexpr int PIECES = ROWS * C4;
#pragma unroll
    for (int i = 0; i < (PIECES + COUNT - 1) / COUNT; ++i) {
        const int idx = t + i * COUNT;
        if (PIECES % COUNT != 0 && idx >= PIECES) break;
        const int r = idx / C4, c = (idx % C4) * 4;
        const bool row_ok = row0 + r < T;
        const float* p = src + (long long)(row0 + r) * st + c;
        float* d = dst + r * (DP + 4) + c;
        if (vec) {
            const bool ok = row_ok && c < D;
            cp16(d, ok ? p : src, ok ? 16 : 0);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const bool ok = row_ok && c + e < D;
                cp4(d + e, ok ? p + e : src, ok ? 4 : 0);
            }
        }
    }
}

// s[r][c] = sum_d A[4 ty + r][d] * B[tx + 8 c][d].  PAIRS: even and odd d side by side, from 96 wide tiles on, where both
// directions have the registers for twice the sums.  Both, because the backward makes the probabilities again from the forward's
// row sums: with pairs in the forward alone the two round the scores differently, and at B4 H6 T256 D32 the gradients were 7 to
// 11 % further from 64 bits (dQ 3.1e-7 -> 3.5e-7) than with the same sums on both sides.
template <int DP, bool PAIRS, int RM, int NC>
__device__ __forceinline__ void tile_nt(const float* __restrict__ A, const float* __restrict__ Bm, int ty, int tx, float (&s)[RM][NC]) {
    constexpr int LD = DP + 4;
    if constexpr (PAIRS) {
        uint64_t s2[RM][NC];
#pragma unroll
        for (int r = 0; r < RM; ++r)
#pragma unroll
            for (int c = 0; c < NC; ++c) s2[r][c] = 0;
#pragma unroll 2
        for (int d = 0; d < DP; d += 4) {
            ulonglong2 a[RM];
#pragma unroll
            for (int r = 0; r < RM; ++r) a[r] = *reinterpret_cast<const ulonglong2*>(A + (ty * RM + r) * LD + d);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(Bm + (tx + 8 * c) * LD + d);
#pragma unroll
                for (int r = 0; r < RM; ++r) s2[r][c] = fma2(a[r].x, b.x, s2[r][c]);
#pragma unroll
                for (int r = 0; r < RM; ++r) s2[r][c] = fma2(a[r].y, b.y, s2[r][c]);
            }
        }
#pragma unroll
        for (int r = 0; r < RM; ++r)
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                float even, odd;
                unpack_f32x2(s2[r][c], even, odd);
                s[r][c] = even + odd;
            }
    } else {
#pragma unroll
        for (int r = 0; r < RM; ++r)
#pragma unroll
            for (int c = 0; c < NC; ++c) s[r][c] = 0.f;
#pragma unroll 2
        for (int d = 0; d < DP; d += 4) {
            float4 a[RM];
#pragma unroll
            for (int r = 0; r < RM; ++r) a[r] = *reinterpret_cast<const float4*>(A + (ty * RM + r) * LD + d);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const float4 b = *reinterpret_cast<const float4*>(Bm + (tx + 8 * c) * LD + d);
#pragma unroll
                for (int r = 0; r < RM; ++r) {
                    s[r][c] = fmaf(a[r].x, b.x, s[r][c]);
                    s[r][c] = fmaf(a[r].y, b.y, s[r][c]);
                    s[r][c] = fmaf(a[r].z, b.z, s[r][c]);
                    s[r][c] = fmaf(a[r].w, b.w, s[r][c]);
                }
            }
        }
    }
}

// A row of an accumulator: DP / 8 floats, as pairs or one by one.
template <int DP, bool PAIRS>
struct Acc {
    using T = typename std::conditional<PAIRS, uint64_t, float>::type;
    T v[PAIRS ? DP / 16 : DP / 8];
    __device__ __forceinline__ T& operator[](int i) { return v[i]; }
    __device__ __forceinline__ const T& operator[](int i) const { return v[i]; }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (auto& x : v) x = 0;
    }
};

// acc[r][2 j], acc[r][2 j + 1] (pairs of columns 4 tx + 32 j ..) += sum_k P[4 ty + r][k] * X[k][..], k < KN (P row stride PLD)
// PAIRS as above: the 32-wide backward has no registers for the doubled P.  (The 64-wide one spills with them, 136 / 208 bytes of stores /
// loads where single products spill 64 / 116, and is 1 to 3 % faster all the same.)
template <int DP, int KN, int PLD, bool PAIRS, int RM>
__device__ __forceinline__ void tile_pv(const float* __restrict__ Ps, const float* __restrict__ X, int ty, int tx, Acc<DP, PAIRS> (&acc)[RM]) {
    constexpr int LD = DP + 4;
#pragma unroll 2
    for (int k = 0; k < KN; k += 4) {
        float4 p[RM];
#pragma unroll
        for (int r = 0; r < RM; ++r) p[r] = *reinterpret_cast<const float4*>(Ps + (ty * RM + r) * PLD + k);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            float pr[RM];
#pragma unroll
            for (int r = 0; r < RM; ++r) pr[r] = kk == 0 ? p[r].x : kk == 1 ? p[r].y : kk == 2 ? p[r].z : p[r].w;
#pragma unroll
            for (int j = 0; j < DP / 32; ++j) {
                const float* q = X + (k + kk) * LD + tx * 4 + 32 * j;
                if constexpr (PAIRS) {
                    const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(q);
#pragma unroll
                    for (int r = 0; r < RM; ++r) acc[r][2 * j] = fma2(pack_f32x2(pr[r], pr[r]), x.x, acc[r][2 * j]);
#pragma unroll
                    for (int r = 0; r < RM; ++r) acc[r][2 * j + 1] = fma2(pack_f32x2(pr[r], pr[r]), x.y, acc[r][2 * j + 1]);
                } else {
                    const float4 x = *reinterpret_cast<const float4*>(q);
#pragma unroll
                    for (int r = 0; r < RM; ++r) {
                        acc[r][4 * j + 0] = fmaf(pr[r], x.x, acc[r][4 * j + 0]);
                        acc[r][4 * j + 1] = fmaf(pr[r], x.y, acc[r][4 * j + 1]);
                        acc[r][4 * j + 2] = fmaf(pr[r], x.z, acc[r][4 * j + 2]);
                        acc[r][4 * j + 3] = fmaf(pr[r], x.w, acc[r][4 * j + 3]);
                    }
                }
            }
        }
    }
}

// Row reductions over the eight threads that share a row.
__device__ __forceinline__ float row_max(float x) {
#pragma unroll
    for (int o = 0; o < 3; ++o) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o == 0 ? 16 : o == 1 ? 4 : 2));    // the bits of place_x
    return x;
}
__device__ __forceinline__ float row_sum(float x) {
#pragma unroll
    for (int o = 0; o < 3; ++o) x += __shfl_xor_sync(0xffffffffu, x, o == 0 ? 16 : o == 1 ? 4 : 2);
    return x;
}

template <int DP, bool PAIRS, int RM>
__device__ __forceinline__ void put_acc(float* dst, int ty, int tx, const Acc<DP, PAIRS> (&acc)[RM]) {
#pragma unroll
    for (int r = 0; r < RM; ++r)
#pragma unroll
        for (int j = 0; j < DP / 32; ++j)
            if constexpr (PAIRS)
                *reinterpret_cast<ulonglong2*>(dst + (ty * RM + r) * (DP + 4) + tx * 4 + 32 * j) = make_ulonglong2(acc[r][2 * j], acc[r][2 * j + 1]);
            else
                *reinterpret_cast<float4*>(dst + (ty * RM + r) * (DP + 4) + tx * 4 + 32 * j) =
                    make_float4(acc[r][4 * j], acc[r][4 * j + 1], acc[r][4 * j + 2], acc[r][4 * j + 3]);
}

// One 16-byte piece of an output row, element by element where alignment or D ask for it.
__device__ __forceinline__ void store4(float* p, float4 v, int valid, int vec) {
    if (vec) { if (valid > 0) *reinterpret_cast<float4*>(p) = v; return; }
    if (valid > 0) p[0] = v.x;
    if (valid > 1) p[1] = v.y;
    if (valid > 2) p[2] = v.z;
    if (valid > 3) p[3] = v.w;
}

// NG: groups of 64 threads per block; FBN: rows of a tile streamed in the forward; RM: stationary rows per thread, an eighth of a block's
template <int DP, int NG = 4, int FBN = 32, int RM = 4>
struct Tile {
    static constexpr int BM = 8 * RM;                           // stationary rows per block
    static constexpr int NT = 64 * NG;
    static constexpr int BN = FBN;
    static constexpr int NC = BN / 8;                           // score columns per thread
    static constexpr int LD = DP + 4;
    static constexpr int ROWS = BM * LD;                        // a stationary tile
    static constexpr int STREAM = BN * LD;                      // a streamed tile
    // forward: Q | per group: K, V, P.  The merge at the end reuses the groups' K (partial O) and P (max, sum).
    static constexpr int FWD_PLD = BN + 4;
    static constexpr int FWD_GROUP = 2 * STREAM + BM * FWD_PLD;
    static constexpr size_t FWD_SMEM = (size_t)(ROWS + NG * FWD_GROUP) * sizeof(float);
    // backward: two stationary tiles | per group: two streamed tiles, half a P / dS tile (32 columns), row statistics
    static constexpr int BWD_PLD = 36;
    static constexpr int BWD_BN = 32;
    static constexpr bool BWD_PAIRS = DP >= 64;                 // pairs of products in the backward's second products
    static constexpr int BWD_STREAM = BWD_BN * LD;
    static constexpr int BWD_GROUP = 2 * BWD_STREAM + BM * BWD_PLD + 2 * BWD_BN;
    static constexpr size_t BWD_SMEM = (size_t)(2 * ROWS + 2 * BM + NG * BWD_GROUP) * sizeof(float);
};

// ---------------------------------------------------------------------------
// Forward: one block per (batch*head, query tile of BM rows); the heaviest (latest) query tiles of all slices first.
// ---------------------------------------------------------------------------
template <int DP, int NG, int FBN, int RM>
__global__ void __launch_bounds__(64 * NG, DP <= 32 && NG == 4 ? 2 : 1) attn_fwd_f32_kernel(const F32Params p) {
    chain_wait();
    using L = Tile<DP, NG, FBN, RM>;
    constexpr int BM = L::BM, NT = L::NT, BN = L::BN, NC = L::NC, LD = L::LD, PLD = L::FWD_PLD;
    extern __shared__ __align__(16) float smem[];
    const int g = threadIdx.x / 64, t = threadIdx.x % 64;
    const int ty = place_y(t), tx = place_x(t);
    float* Qs = smem;
    float* Ks = Qs + L::ROWS + g * L::FWD_GROUP;
    float* Vs = Ks + L::STREAM;
    float* Ps = Vs + L::STREAM;

    const int nq = (p.T + BM - 1) / BM;
    const int q0 = (nq - 1 - (int)blockIdx.y) * BM;
    const int bh = blockIdx.x;
    const int b = bh / p.H, h = bh % p.H;
    const float* kb = p.k + b * p.sk.b + h * p.sk.h;
    const float* vb = p.v + b * p.sv.b + h * p.sv.h;
    const int keys = p.causal ? min(p.T, q0 + BM) : p.T;
    const int ntiles = (keys + BN - 1) / BN;

    fetch_tile<DP, BM, NT>(Qs, p.q + b * p.sq.b + h * p.sq.h, q0, p.T, p.D, p.sq.t, p.vec, threadIdx.x);
    if (g < ntiles) fetch_tile<DP, BN, 64>(Ks, kb, g * BN, p.T, p.D, p.sk.t, p.vec, t);
    cp_commit();
    if (g < ntiles) fetch_tile<DP, BN, 64>(Vs, vb, g * BN, p.T, p.D, p.sv.t, p.vec, t);
    cp_commit();
    cp_wait<1>();
    __syncthreads();                                            // Q is shared by the groups

    float m[RM], l[RM];
    Acc<DP, true> acc[RM];
#pragma unroll
    for (int r = 0; r < RM; ++r) {
        m[r] = -INFINITY; l[r] = 0.f;
        acc[r].clear();
    }
    const float sl2 = p.scale * LOG2E;

    for (int j = g; j < ntiles; j += NG) {
        const int k0 = j * BN;
        if (j != g) { cp_wait<1>(); group_sync(g); }            // this K tile has landed for both warps
        float s[RM][NC];
        tile_nt<DP, (DP >= 96)>(Qs, Ks, ty, tx, s);
        group_sync(g);                                          // K is consumed: the next one may land
        if (j + NG < ntiles) fetch_tile<DP, BN, 64>(Ks, kb, k0 + NG * BN, p.T, p.D, p.sk.t, p.vec, t);
        cp_commit();
        const bool edge = k0 + BN > p.T || (p.causal && k0 + BN - 1 > q0);
#pragma unroll
        for (int r = 0; r < RM; ++r) {
            const int row = q0 + ty * RM + r;
            float mx = -INFINITY;
            if (edge) {
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const int col = k0 + tx + 8 * c;
                    s[r][c] = (col >= p.T || (p.causal && col > row)) ? -INFINITY : s[r][c] * sl2;
                    mx = fmaxf(mx, s[r][c]);
                }
            } else {
#pragma unroll
                for (int c = 0; c < NC; ++c) { s[r][c] *= sl2; mx = fmaxf(mx, s[r][c]); }
            }
            const float m_new = fmaxf(m[r], row_max(mx));
            const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
            const float alpha = exp2f(m[r] - m_use);
            float rs = 0.f;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const float e = exp2f(s[r][c] - m_use);
                rs += e;
                Ps[(ty * RM + r) * PLD + tx + 8 * c] = e;
            }
            l[r] = l[r] * alpha + row_sum(rs);
            m[r] = m_new;
#pragma unroll
            for (int c = 0; c < DP / 16; ++c) acc[r][c] = mul2(acc[r][c], pack_f32x2(alpha, alpha));
        }
        cp_wait<1>();
        group_sync(g);                                          // V has landed (and this warp's P rows are visible)
        tile_pv<DP, BN, PLD, true>(Ps, Vs, ty, tx, acc);
        group_sync(g);                                          // V is consumed
        if (j + NG < ntiles) fetch_tile<DP, BN, 64>(Vs, vb, k0 + NG * BN, p.T, p.D, p.sv.t, p.vec, t);
        cp_commit();
    }
    cp_wait<0>();
    // Where a block fills its SM, successors set up in front of its last stores take the idle SMs unevenly (forward and backward
    // in turn, B4 H6 T256 D32: 31.0 us, with the call at the end 29.3).
    if (NG == 4) chain_next();

    // The groups meet: O = sum_g 2^(m_g - M) O_g / sum_g 2^(m_g - M) l_g, in group order.
    put_acc(Ks, ty, tx, acc);
    if (tx == 0) {
#pragma unroll
        for (int r = 0; r < RM; ++r) { Ps[ty * RM + r] = m[r]; Ps[BM + ty * RM + r] = l[r]; }
    }
    __syncthreads();
    float* ob = p.out_o + b * p.so.b + h * p.so.h;
    constexpr int C4 = DP / 4;
    for (int idx = threadIdx.x; idx < BM * C4; idx += NT) {
        const int r = idx / C4, c = (idx % C4) * 4, row = q0 + r;
        if (row >= p.T || c >= p.D) continue;
        const float* grp = smem + L::ROWS;
        float mg[NG], M = -INFINITY, sum = 0.f;
#pragma unroll
        for (int z = 0; z < NG; ++z) { mg[z] = grp[z * L::FWD_GROUP + 2 * L::STREAM + r]; M = fmaxf(M, mg[z]); }
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int z = 0; z < NG; ++z) {
            const float w = exp2f(mg[z] - M);                   // a group without keys has m = -inf: weight 0
            const float4 x = *reinterpret_cast<const float4*>(grp + z * L::FWD_GROUP + r * LD + c);
            sum += w * grp[z * L::FWD_GROUP + 2 * L::STREAM + BM + r];
            v.x = fmaf(w, x.x, v.x); v.y = fmaf(w, x.y, v.y); v.z = fmaf(w, x.z, v.z); v.w = fmaf(w, x.w, v.w);
        }
        const float inv = 1.f / sum;
        store4(ob + (long long)row * p.so.t + c, make_float4(v.x * inv, v.y * inv, v.z * inv, v.w * inv), p.D - c, p.vec_out);
        if (c == 0) p.lse_out[(long long)bh * p.T + row] = (M + log2f(sum)) * LN2;
    }
    if (NG != 4) chain_next();
}

// ---------------------------------------------------------------------------
// Backward
// ---------------------------------------------------------------------------
// delta = rowsum(dO * O) (= rowsum(dP * P)), LPR lanes per row: dO from its shared tile, O from global memory.  load() may
// run long before dot(), so that the walk does not wait for global memory (head dims up to 32: 16 registers).
template <int DP, int LPR>
struct RowDelta {
    static constexpr int N = DP / 4 / LPR;
    static constexpr bool EARLY = N <= 4;
    float4 o[EARLY ? N : 1];
    __device__ __forceinline__ static float4 piece(const F32Params& p, const float* orow, int c) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p.vec) {
            if (c < p.D) v = *reinterpret_cast<const float4*>(orow + c);
        } else {
            if (c + 0 < p.D) v.x = orow[c + 0];
            if (c + 1 < p.D) v.y = orow[c + 1];
            if (c + 2 < p.D) v.z = orow[c + 2];
            if (c + 3 < p.D) v.w = orow[c + 3];
        }
        return v;
    }
    __device__ __forceinline__ void load(const F32Params& p, const float* ob, int row, int part) {
        if constexpr (EARLY) {
#pragma unroll
            for (int i = 0; i < N; ++i) o[i] = row < p.T ? piece(p, ob + (long long)row * p.so.t, (part + LPR * i) * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    __device__ __forceinline__ float dot(const F32Params& p, const float* ob, const float* g_row, int row, int part) {
        float d = 0.f;
        if (row < p.T) {
#pragma unroll 4
            for (int i = 0; i < N; ++i) {
                const int c = (part + LPR * i) * 4;
                float4 x;
                if constexpr (EARLY) x = o[i]; else x = piece(p, ob + (long long)row * p.so.t, c);
                const float4 y = *reinterpret_cast<const float4*>(g_row + c);
                d = fmaf(x.x, y.x, d); d = fmaf(x.y, y.y, d); d = fmaf(x.z, y.z, d); d = fmaf(x.w, y.w, d);
            }
        }
#pragma unroll
        for (int off = LPR / 2; off >= 1; off >>= 1) d += __shfl_xor_sync(0xffffffffu, d, off);
        return d;
    }
};

// Adds the groups' partial gradients (each parked in its first streamed tile) and stores the block's rows.
template <int DP, int NG, int BM>
__device__ __forceinline__ void merge_store(const F32Params& p, const float* parts, int stride, float* dst, long long st, int row0, bool rotate) {
    constexpr int C4 = DP / 4, NT = 64 * NG;
    if (rotate) {                                               // D % 8 == 0: a thread takes four columns of both halves
        const int half = p.D / 2, h4 = half / 4;
        for (int idx = threadIdx.x; idx < BM * h4; idx += NT) {
            const int r = idx / h4, c = (idx % h4) * 4, row = row0 + r;
            if (row >= p.T) continue;
            float a[4] = {0.f, 0.f, 0.f, 0.f}, b[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int z = 0; z < NG; ++z) {
                const float* q = parts + z * stride + r * (DP + 4) + c;
#pragma unroll
                for (int e = 0; e < 4; ++e) { a[e] += q[e]; b[e] += q[half + e]; }
            }
            const long long at = (long long)row * half + c;
            const float4 c4 = *reinterpret_cast<const float4*>(p.cosv + at), s4 = *reinterpret_cast<const float4*>(p.sinv + at);
            const float cs[4] = {c4.x, c4.y, c4.z, c4.w}, sn[4] = {-s4.x, -s4.y, -s4.z, -s4.w};
            float o1[4], o2[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {                       // rounded as the rotary pack does
                o1[e] = __fadd_rn(__fmul_rn(a[e], cs[e]), __fmul_rn(b[e], sn[e]));
                o2[e] = __fadd_rn(__fmul_rn(a[e], -sn[e]), __fmul_rn(b[e], cs[e]));
            }
            float* o = dst + (long long)row * st + c;
            store4(o, make_float4(o1[0], o1[1], o1[2], o1[3]), 4, p.vec_out);
            store4(o + half, make_float4(o2[0], o2[1], o2[2], o2[3]), 4, p.vec_out);
        }
        return;
    }
    for (int idx = threadIdx.x; idx < BM * C4; idx += NT) {
        const int r = idx / C4, c = (idx % C4) * 4, row = row0 + r;
        if (row >= p.T || c >= p.D) continue;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int z = 0; z < NG; ++z) {
            const float4 x = *reinterpret_cast<const float4*>(parts + z * stride + r * (DP + 4) + c);
            v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
        }
        store4(dst + (long long)row * st + c, v, p.D - c, p.vec_out);
    }
}

// Scores to P in place: rows are query rows (ROWS_ARE_Q) or key rows of the BM x BN tile; l2 / dl hold lse * log2e and delta
// of the tile's query rows.
template <bool ROWS_ARE_Q, int RM, int NC>
__device__ __forceinline__ void probabilities(const F32Params& p, float (&s)[RM][NC], const float* l2, int row0, int col0, int ty, int tx) {
    const float sl2 = p.scale * LOG2E;
#pragma unroll
    for (int r = 0; r < RM; ++r) {
        const int row = row0 + ty * RM + r;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int col = col0 + tx + 8 * c;
            const bool masked = row >= p.T || col >= p.T || (p.causal && (ROWS_ARE_Q ? col > row : row > col));
            const float lq = ROWS_ARE_Q ? l2[ty * RM + r] : l2[tx + 8 * c];
            s[r][c] = masked ? 0.f : exp2f(fmaf(s[r][c], sl2, -lq));
        }
    }
}

// acc += tile * X with the BM x BN tile handed through shared memory 32 columns at a time (rows stay inside a warp).
template <int DP, int RM, int NC>
__device__ __forceinline__ void staged_product(float* stage, const float (&v)[RM][NC], const float* X, int ty, int tx,
                                               Acc<DP, Tile<DP>::BWD_PAIRS> (&acc)[RM]) {
    constexpr int PLD = Tile<DP>::BWD_PLD;
#pragma unroll
    for (int half = 0; half < NC / 4; ++half) {
        __syncwarp();
#pragma unroll
        for (int r = 0; r < RM; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) stage[(ty * RM + r) * PLD + tx + 8 * c] = v[r][half * 4 + c];
        __syncwarp();
        tile_pv<DP, 32, PLD, Tile<DP>::BWD_PAIRS>(stage, X + half * 32 * (DP + 4), ty, tx, acc);
    }
}

// dK / dV of BM key rows: the groups walk the query tiles at or below the diagonal.
template <int DP, int NG, int RM>
__device__ __forceinline__ void bwd_dkdv(const F32Params& p, float* smem, int kt, int bh) {
    using L = Tile<DP, NG, 32, RM>;
    constexpr int BM = L::BM, NT = L::NT, BN = L::BWD_BN, NC = BN / 8, LD = L::LD;
    const int g = threadIdx.x / 64, t = threadIdx.x % 64;
    const int ty = DP <= 32 ? t / 8 : place_y(t), tx = DP <= 32 ? t % 8 : place_x(t);     // (DP 32: plain, it spills less)
    float* Ks = smem;
    float* Vs = Ks + L::ROWS;
    float* grp0 = smem + 2 * L::ROWS + 2 * BM;
    float* Qs = grp0 + g * L::BWD_GROUP;
    float* Gs = Qs + L::BWD_STREAM;
    float* stage = Gs + L::BWD_STREAM;
    float* l2 = stage + BM * L::BWD_PLD;
    float* dl = l2 + BN;

    const int b = bh / p.H, h = bh % p.H;
    const int k0 = kt * BM;
    const float* qb = p.q + b * p.sq.b + h * p.sq.h;
    const float* gb = p.d_o + b * p.sdo.b + h * p.sdo.h;
    const float* ob = p.o + b * p.so.b + h * p.so.h;
    const int first = p.causal ? k0 / BN : 0, ntiles = (p.T + BN - 1) / BN;
    const int i0 = first + g;

    fetch_tile<DP, BM, NT>(Ks, p.k + b * p.sk.b + h * p.sk.h, k0, p.T, p.D, p.sk.t, p.vec, threadIdx.x);
    if (i0 < ntiles) fetch_tile<DP, BN, 64>(Qs, qb, i0 * BN, p.T, p.D, p.sq.t, p.vec, t);
    cp_commit();
    fetch_tile<DP, BM, NT>(Vs, p.v + b * p.sv.b + h * p.sv.h, k0, p.T, p.D, p.sv.t, p.vec, threadIdx.x);
    if (i0 < ntiles) fetch_tile<DP, BN, 64>(Gs, gb, i0 * BN, p.T, p.D, p.sdo.t, p.vec, t);
    cp_commit();
    cp_wait<0>();
    __syncthreads();                                            // K and V are shared by the groups

    Acc<DP, L::BWD_PAIRS> dk[RM], dv[RM];
#pragma unroll
    for (int r = 0; r < RM; ++r) { dk[r].clear(); dv[r].clear(); }

    RowDelta<DP, 2> rd;                                         // two threads per row of the streamed tile
    float lse_next = 0.f;
    auto stats_ahead = [&](int q0) {
        const int row = q0 + t / 2;
        rd.load(p, ob, row, t % 2);
        lse_next = row < p.T ? p.lse[(long long)bh * p.T + row] * LOG2E : 0.f;
    };
    static_assert(BN == 32, "two threads per row");
    if (i0 < ntiles) stats_ahead(i0 * BN);
    for (int i = i0; i < ntiles; i += NG) {
        const int q0 = i * BN;
        if (i != i0) { cp_wait<1>(); group_sync(g); }           // this Q tile has landed for both warps
        float pp[RM][NC], ds[RM][NC];
        tile_nt<DP, (DP >= 96)>(Ks, Qs, ty, tx, pp);                    // S^T
        if (i != i0) { cp_wait<0>(); group_sync(g); }           // and so has dO
        {
            const float d = rd.dot(p, ob, Gs + (t / 2) * LD, q0 + t / 2, t % 2);
            if (t % 2 == 0) { l2[t / 2] = lse_next; dl[t / 2] = d; }
        }
        tile_nt<DP, (DP >= 96)>(Vs, Gs, ty, tx, ds);                    // dP^T
        group_sync(g);                                          // statistics are visible
        probabilities<false>(p, pp, l2, k0, q0, ty, tx);
#pragma unroll
        for (int r = 0; r < RM; ++r)
#pragma unroll
            for (int c = 0; c < NC; ++c) ds[r][c] = pp[r][c] * (ds[r][c] - dl[tx + 8 * c]) * p.scale;
        staged_product<DP>(stage, ds, Qs, ty, tx, dk);      // dK += dS^T Q
        group_sync(g);                                          // Q is consumed
        if (i + NG < ntiles) fetch_tile<DP, BN, 64>(Qs, qb, q0 + NG * BN, p.T, p.D, p.sq.t, p.vec, t);
        cp_commit();
        if (i + NG < ntiles) stats_ahead(q0 + NG * BN);
        staged_product<DP>(stage, pp, Gs, ty, tx, dv);      // dV += P^T dO
        group_sync(g);
        if (i + NG < ntiles) fetch_tile<DP, BN, 64>(Gs, gb, q0 + NG * BN, p.T, p.D, p.sdo.t, p.vec, t);
        cp_commit();
    }
    cp_wait<0>();
    chain_next();
    put_acc(Qs, ty, tx, dk);
    put_acc(Gs, ty, tx, dv);
    __syncthreads();
    merge_store<DP, NG, BM>(p, grp0, L::BWD_GROUP, p.dk + b * p.sdk.b + h * p.sdk.h, p.sdk.t, k0, p.cosv != nullptr);
    merge_store<DP, NG, BM>(p, grp0 + L::BWD_STREAM, L::BWD_GROUP, p.dv + b * p.sdv.b + h * p.sdv.h, p.sdv.t, k0, false);
}

// dQ of BM query rows: the groups walk the key tiles at or left of the diagonal.
template <int DP, int NG, int RM>
__device__ __forceinline__ void bwd_dq(const F32Params& p, float* smem, int qt, int bh) {
    using L = Tile<DP, NG, 32, RM>;
    constexpr int BM = L::BM, NT = L::NT, BN = L::BWD_BN, NC = BN / 8, LD = L::LD;
    const int g = threadIdx.x / 64, t = threadIdx.x % 64;
    const int ty = DP <= 32 ? t / 8 : place_y(t), tx = DP <= 32 ? t % 8 : place_x(t);     // (DP 32: plain, it spills less)
    float* Qs = smem;
    float* Gs = Qs + L::ROWS;
    float* l2 = smem + 2 * L::ROWS;
    float* dl = l2 + BM;
    float* grp0 = dl + BM;
    float* Ks = grp0 + g * L::BWD_GROUP;
    float* Vs = Ks + L::BWD_STREAM;
    float* stage = Vs + L::BWD_STREAM;

    const int b = bh / p.H, h = bh % p.H;
    const int q0 = qt * BM;
    const float* kb = p.k + b * p.sk.b + h * p.sk.h;
    const float* vb = p.v + b * p.sv.b + h * p.sv.h;
    const int keys = p.causal ? min(p.T, q0 + BM) : p.T;
    const int ntiles = (keys + BN - 1) / BN;

    fetch_tile<DP, BM, NT>(Qs, p.q + b * p.sq.b + h * p.sq.h, q0, p.T, p.D, p.sq.t, p.vec, threadIdx.x);
    if (g < ntiles) fetch_tile<DP, BN, 64>(Ks, kb, g * BN, p.T, p.D, p.sk.t, p.vec, t);
    fetch_tile<DP, BM, NT>(Gs, p.d_o + b * p.sdo.b + h * p.sdo.h, q0, p.T, p.D, p.sdo.t, p.vec, threadIdx.x);
    if (g < ntiles) fetch_tile<DP, BN, 64>(Vs, vb, g * BN, p.T, p.D, p.sv.t, p.vec, t);
    cp_commit();
    cp_wait<0>();
    __syncthreads();                                            // Q and dO are shared by the groups
    RowDelta<DP, 8> rd;
    if (threadIdx.x < 8 * BM) {
        const int r = threadIdx.x / 8, row = q0 + r;            // eight threads per row
        const float* ob = p.o + b * p.so.b + h * p.so.h;
        rd.load(p, ob, row, threadIdx.x % 8);
        const float d = rd.dot(p, ob, Gs + r * LD, row, threadIdx.x % 8);
        if (threadIdx.x % 8 == 0) { l2[r] = row < p.T ? p.lse[(long long)bh * p.T + row] * LOG2E : 0.f; dl[r] = d; }
    }

    Acc<DP, L::BWD_PAIRS> dq[RM];
#pragma unroll
    for (int r = 0; r < RM; ++r) dq[r].clear();
    float pp[RM][NC], ds[RM][NC];
    if (g < ntiles) tile_nt<DP, (DP >= 96)>(Qs, Ks, ty, tx, pp);        // the first S while the statistics are made
    __syncthreads();

    for (int j = g; j < ntiles; j += NG) {
        const int k0 = j * BN;
        if (j != g) {
            cp_wait<0>();
            group_sync(g);
            tile_nt<DP, (DP >= 96)>(Qs, Ks, ty, tx, pp);
        }
        tile_nt<DP, (DP >= 96)>(Gs, Vs, ty, tx, ds);                    // dP
        group_sync(g);                                          // V is consumed
        if (j + NG < ntiles) fetch_tile<DP, BN, 64>(Vs, vb, k0 + NG * BN, p.T, p.D, p.sv.t, p.vec, t);
        cp_commit();
        probabilities<true>(p, pp, l2, q0, k0, ty, tx);
#pragma unroll
        for (int r = 0; r < RM; ++r)
#pragma unroll
            for (int c = 0; c < NC; ++c) ds[r][c] = pp[r][c] * (ds[r][c] - dl[ty * RM + r]) * p.scale;
        staged_product<DP>(stage, ds, Ks, ty, tx, dq);      // dQ += dS K
        group_sync(g);
        if (j + NG < ntiles) {
            fetch_tile<DP, BN, 64>(Ks, kb, k0 + NG * BN, p.T, p.D, p.sk.t, p.vec, t);
        }
        cp_commit();
    }
    cp_wait<0>();
    chain_next();
    put_acc(Ks, ty, tx, dq);
    __syncthreads();
    merge_store<DP, NG, BM>(p, grp0, L::BWD_GROUP, p.dq + b * p.sdq.b + h * p.sdq.h, p.sdq.t, q0, p.cosv != nullptr);
}

// Both roles in one launch: row n of the grid holds every slice's n-th heaviest key tile, then every slice's n-th heaviest query
// tile (gridDim.y ends at 65535; the longest sequence, 2^20, has 32768 tiles of a kind, and comes with too many blocks for smaller ones).
template <int DP, int NG, int RM>
__global__ void __launch_bounds__(64 * NG, DP <= 64 && NG == 4 ? 2 : 1) attn_bwd_f32_kernel(const F32Params p) {
    chain_wait();
    extern __shared__ __align__(16) float smem[];
    const int n = blockIdx.y, slices = p.B * p.H, x = blockIdx.x;
    if (x < slices) bwd_dkdv<DP, NG, RM>(p, smem, n, x);
    else bwd_dq<DP, NG, RM>(p, smem, (int)gridDim.y - 1 - n, x - slices);
}

Strides3 s3(const int64_t* s) { return Strides3{(long long)s[0], (long long)s[1], (long long)s[2]}; }

bool rows_vec_ok(const void* ptr, const int64_t* s) {
    return (((uintptr_t)ptr) & 15u) == 0 && (s[0] & 3) == 0 && (s[1] & 3) == 0 && (s[2] & 3) == 0;
}

template <int DP, int NG, int FBN, int RM>
int fwd_launch_f32(deers_ctx* ctx, const F32Params& p) {
    using L = Tile<DP, NG, FBN, RM>;
    DEERS_SMEM_ONCE(ctx, (attn_fwd_f32_kernel<DP, NG, FBN, RM>), L::FWD_SMEM);
    const dim3 grid(p.B * p.H, (p.T + L::BM - 1) / L::BM);
    const auto kernel = attn_fwd_f32_kernel<DP, NG, FBN, RM>;
    {
        KernelTimerScope ts(ctx, DEERS_K_FWD);
        DEERS_CUDA_TRY(ctx, launch_chained(ctx, kernel, grid, L::NT, L::FWD_SMEM, 1, p));
    }
    ctx->launches += 1;
    DEERS_CUDA_TRY(ctx, cudaGetLastError());
    return DEERS_OK;
}

template <int DP, int NG, int RM>
int bwd_launch_f32(deers_ctx* ctx, const F32Params& p) {
    using L = Tile<DP, NG, 32, RM>;
    DEERS_SMEM_ONCE(ctx, (attn_bwd_f32_kernel<DP, NG, RM>), L::BWD_SMEM);
    const dim3 grid(2 * p.B * p.H, (p.T + L::BM - 1) / L::BM);
    const auto kernel = attn_bwd_f32_kernel<DP, NG, RM>;
    {
        KernelTimerScope ts(ctx, DEERS_K_BWD_MAIN);
        DEERS_CUDA_TRY(ctx, launch_chained(ctx, kernel, grid, L::NT, L::BWD_SMEM, 1, p));
    }
    DEERS_CUDA_TRY(ctx, cudaGetLastError());
    ctx->launches += 1;
    return DEERS_OK;
}

}  // namespace
