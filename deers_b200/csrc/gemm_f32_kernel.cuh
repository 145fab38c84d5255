// f32 GEMM on the FFMA pipe (no TF32) for the projections of the f32 model: Linear::forward
// (src/nn.rs:184-190, weight stored [in, out]) and the two products of the matmul backward
// (src/ops.rs:1089-1101).  The reference sends these to cublasGemmStridedBatchedEx with
// CUBLAS_COMPUTE_32F (src/storage/cuda.rs:1098-1128), i.e. full f32 arithmetic; so does this kernel.
//
// C[M,N] = A * B for either storage order of A and of B, arbitrary leading dimensions and alignments, with an epilogue
// applied to the finished tile:
//   NONE      C = acc
//   ADD       C = R + acc                 the residual connections of the block (gpt.rs:237-239)
//   RELU_SQ   r = max(acc, 0); C = r*r; AUX = r     relu and y*y of the MLP (gpt.rs:194-196)
//   MUL_AUX2  t = acc * AUX; C = t + t    the backward of y*y and relu in one (ops.rs:210-214, 560-568)
//
// What bounds it: the model's products are small (1024 x 576 x 192 and the like): 150 tiles of 64 x 64, one per SM, so
// a product takes as long as ONE block takes for its walk over K.  The block is built around that walk:
//   * 128 threads own the tile (patches of PM x PN) and KS such groups take a share of every stage's k each: loads,
//     waits and arithmetic of a group are its own, so the groups drift apart and one's shared-memory bursts meet another's
//     multiply-adds;
//   * the loop is bound by issue slots, register banks and shared memory together.  Two products share a slot
//     (fma.rn.f32x2, each an IEEE f32 fma): neighbouring columns where B is in MN order, even and odd k in small patches with both
//     operands in K order (large ones would need twice the accumulators and stay with single products; packing columns there
//     costs two moves per pair and was slower: 11.4 -> 15.4 us at 1024 x 768 x 192).  Lanes lie in the tile so that a 16-byte
//     shared-memory read costs 2.1 cycles instead of 4: it does when each quarter warp asks for at most four addresses and
//     neighbouring lanes share them (lane % 8 along a row does not, (lane / 2) % 4 does; measured);
//   * operands travel by cp.async straight into shared memory in their storage order (no transposition, no
//     registers), up to (STAGES - 1) * 64 k ahead: 192 in tiles of up to 4096 elements, 128 in the wider ones;
//   * k groups, and the blocks of a cluster that split a long K among them (weight gradients), meet in shared
//     memory: group 0..KS-1 of block 0..P-1 are added in that order by the threads that write the tile (distributed
//     shared memory, one cluster barrier), so nothing goes through global memory, no counter, no workspace, and the
//     result does not depend on timing.
// Back to back in a graph, with single products and stages shared by 512 threads and now (us): 1024 x 768 x 192 11.4 -> 10.7,
// 1024 x 192 x 768 13.1 -> 12.5, 231 x 500 x 192 4.0 -> 3.7; both operands in MN order (weight gradients) 192 x 768 x 1024
// 13.6 -> 11.0, 231 x 500 x 192 4.6 -> 4.1; both in K order with large patches as it was (1024 x 576 x 192 8.5 -> 8.6).
#pragma once
#include "common.cuh"
#include "f32_util.cuh"

#include <cooperative_groups.h>

struct GemmArgs {
    const float* a; const float* b; float* c;
    const float* r;          // ADD: residual [M][ldr]
    float* aux;              // RELU_SQ: written; MUL_AUX2: read; [M][ldc]
    long long lda, ldb, ldc, ldr;
    int M, N, K;
    int a_vec, b_vec, c_vec; // 16-byte accesses allowed
    int epi;
    int k_chunk;             // K elements per part (multiple of BK)
    // FUSED kernels only: A is a residual stream, its rows are normalised on the way (C = rmsnorm(A) * B), and the columns
    // [0, rope_cols) of C, heads of rope_d columns, are rotated by the row's position (m % rope_t)
    float eps, inv_n;        // inverse norm of a row: 1 / sqrt(sum(a * a) * inv_n + eps)
    float* inv;              // written [M] (nullptr: not wanted)
    const float* cosv; const float* sinv;
    int rope_cols, rope_d, rope_t;
};

struct GemmPlan {
    int cfg;        // index into kVariants
    int parts, k_chunk;
    int waves;      // blocks an SM runs one after another
    double cost;    // cycles
};

// Products with an operand whose rows lie on no 16-byte boundary (gemm_f32_loose.cu).  A module of their own: the first product of a
// process loads all kernels of its module, and most programs never need these (first training step of a process 8.4 ms, 17 with them).
int launch_gemm_f32_loose(deers_ctx* ctx, const GemmPlan& p, const GemmArgs& g, int a_mn, int b_mn, bool fused);

// Products on the tensor core (gemm_f32_tc.cu, the tile: gemm_f32_tc.cuh).
int launch_gemm_f32_tc(deers_ctx* ctx, int parts, const GemmArgs& g, int a_mn, int b_mn, bool fused);
int launch_gemm_f32_tc_loose(deers_ctx* ctx, int parts, const GemmArgs& g, int a_mn, int b_mn);

namespace {
namespace cg = cooperative_groups;

constexpr int GT = 128;                                 // threads of a k group
constexpr int BK = 64;                                  // depth of one stage, shared evenly by the k groups
constexpr int MAX_PARTS = 8;                            // blocks of a cluster along K (portable cluster size)

__device__ __forceinline__ float4 ld4(const float* p, int valid, bool vec) {
    if (vec && valid >= 4) return *reinterpret_cast<const float4*>(p);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (valid > 0) v.x = p[0];
    if (valid > 1) v.y = p[1];
    if (valid > 2) v.z = p[2];
    if (valid > 3) v.w = p[3];
    return v;
}

// The threads of a k group meet (barrier 0 is __syncthreads).
__device__ __forceinline__ void group_sync(int g) { asm volatile("bar.sync %0, 128;" ::"r"(g + 1) : "memory"); }

// One operand's stage of one k group in shared memory, in its storage order: R rows (m or n) of KG k when k is contiguous,
// KG rows of R when m / n is.  Row strides are 4 mod 16 words (16-byte pieces of neighbouring rows fall into different banks).
// LOOSE: takes rows that lie on no 16-byte boundary as well, float by float with neighbouring lanes side by side: a copy
// instruction of a warp then touches one or two rows of 16 k, where four floats per lane touch eight, four times over.
// 66 x 249 x 689 7.6 -> 5.4 us, 2133 x 769 x 1405 185 -> 147.  Kernels of their own, because the branch costs aligned products
// 2 to 4 % (192 x 768 x 1024 12.85 -> 13.4).  Rows of 96 floats do not fit the lanes and keep the four floats per lane.
// PERM: see row_of(); for small patches (32 x 96 tiles lose more by the registers, 1024 x 192 x 576 11.9 -> 12.9).
template <int R, bool MN, int KG, bool LOOSE, bool PERM>
struct Operand {
    static constexpr int LD = MN ? R + 4 : KG + 4;
    static constexpr int FLOATS = MN ? KG * LD : R * LD;
    static constexpr int LEN = MN ? R : KG, ROWS = MN ? KG : R;     // contiguous floats per row, rows
    static constexpr int PIECES = ROWS * LEN / 4;
    static constexpr int NP = (PIECES + GT - 1) / GT;               // 16-byte pieces per thread and stage
    static constexpr bool HALF = PIECES < GT;                       // 16 rows of 16 k: half of the threads have one
    static_assert(HALF || NP * GT == PIECES, "whole pieces per thread");
    const float* base;
    const float* src[NP];    // this thread's pieces of the next stage
    int dst[NP];             // their places in the stage (floats)
    int along_r[NP];         // floats of a piece inside the matrix along m / n (K order: 4 or 0)
    int along_k[NP];         // k of a piece inside the group's share of the stage
    long long step;          // from one stage to the next
    // A quarter warp stores two rows of 16 floats: rows i and i + 4 lie 16 banks apart, i and i + 1 would meet in four banks
    // (231 x 192 x 500 5.67 -> 5.50 us, 192 x 768 x 1024 12.4 -> 11.4; B in MN order).
    static __device__ __forceinline__ int row_of(int i) { return PERM && LEN == 16 ? (i & ~7) | (i & 1) * 4 | ((i >> 1) & 3) : i; }
    __device__ __forceinline__ void init(const float* b, long long ld, int r0, int rmax, int k0, int t) {
        base = b;
        step = MN ? BK * ld : BK;
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            const int idx = HALF ? t % PIECES : t + i * GT;
            const int row = row_of(idx / (LEN / 4)), col = (idx % (LEN / 4)) * 4;
            const int r = r0 + (MN ? col : row), k = MN ? row : col;
            along_k[i] = k;
            along_r[i] = MN ? min(4, max(0, rmax - r)) : (r < rmax ? 4 : 0);
            dst[i] = row * LD + col;
            src[i] = b + (MN ? (long long)(k0 + k) * ld + r : (long long)r * ld + k0 + k);
        }
    }
    // Enqueues the next stage's pieces; kv is the number of the group's k that exist, rv that of the tile's m / n.
    __device__ __forceinline__ void fetch(float* s, int kv, bool vec, long long ld, int rv, int t) {
        if constexpr (LOOSE && GT % LEN == 0) {
            if (!vec) {
                int row = t / LEN;
                const int col = t % LEN;
                const int piece = HALF ? t % PIECES : t;
                const float* p = src[0] - (row_of(piece / (LEN / 4)) * ld + piece % (LEN / 4) * 4) + (row * ld + col);
                float* d = s + row * LD + col;
#pragma unroll 4
                for (int i = 0; i < ROWS * LEN / GT; ++i) {
                    const bool in = MN ? row < kv && col < rv : row < rv && col < kv;
                    cp4(d, in ? p : base, in ? 4 : 0);
                    row += GT / LEN; p += GT / LEN * ld; d += GT / LEN * LD;
                }
                src[0] += step;
                return;
            }
        }
        if (HALF && t >= PIECES) return;
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            int valid = along_r[i];
            if (kv < KG) valid = MN ? (along_k[i] < kv ? valid : 0) : min(valid, max(0, kv - along_k[i]));
            const float* p = valid > 0 ? src[i] : base;
            if (vec) {
                cp16(s + dst[i], p, 4 * valid);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) cp4(s + dst[i] + e, valid > e ? p + e : base, valid > e ? 4 : 0);
            }
            src[i] += step;
        }
    }
    // Index inside the tile of element i of thread group coordinate t: contiguous groups of four for MN order (one
    // LDS.128 per four; the last two of six are a group of two), interleaved for K order (one LDS.128 per row and four k).
    template <int P>
    static __device__ __forceinline__ int index(int t, int i) {
        constexpr int G = R / P;                                   // thread groups along this side
        if (!MN) return t + G * i;
        const int q = i / 4 * 4, w = P - q >= 4 ? 4 : P - q;       // first element and width of i's group
        return q * G + t * w + (i - q);
    }
    // The P elements of this thread for U (2 or 4) consecutive k.
    template <int P, int U>
    static __device__ __forceinline__ void read(const float* s, int t, int k, float (&v)[U][P]) {
        if constexpr (!MN) {
#pragma unroll
            for (int i = 0; i < P; ++i) {
                const float* q = s + index<P>(t, i) * LD + k;
                if constexpr (U == 4) {
                    const float4 x = *reinterpret_cast<const float4*>(q);
                    v[0][i] = x.x; v[1][i] = x.y; v[2][i] = x.z; v[3][i] = x.w;
                } else {
                    const float2 x = *reinterpret_cast<const float2*>(q);
                    v[0][i] = x.x; v[1][i] = x.y;
                }
            }
        } else {
#pragma unroll
            for (int kk = 0; kk < U; ++kk)
#pragma unroll
                for (int i = 0; i < P; i += 4) {
                    if (P - i >= 4) {
                        const float4 x = *reinterpret_cast<const float4*>(s + (k + kk) * LD + index<P>(t, i));
                        v[kk][i] = x.x; v[kk][i + 1] = x.y; v[kk][i + 2] = x.z; v[kk][i + 3] = x.w;
                    } else {
                        const float2 x = *reinterpret_cast<const float2*>(s + (k + kk) * LD + index<P>(t, i));
                        v[kk][i] = x.x; v[kk][i + 1] = x.y;
                    }
                }
        }
    }
};

template <int PM, int PN, int KS, bool A_MN, bool B_MN, bool LOOSE>
struct GemmShape {
    static constexpr int BM = 8 * PM, BN = 16 * PN, THREADS = GT * KS, KG = BK / KS;
    using OA = Operand<BM, A_MN, KG, LOOSE, (PM * PN <= 16)>;
    using OB = Operand<BN, B_MN, KG, LOOSE, (PM * PN <= 16)>;
    static constexpr int STAGE = KS * (OA::FLOATS + OB::FLOATS);
    static constexpr int RLD = BN + 4;                              // row stride of the patch staging tile
    static constexpr int RED = KS * BM * RLD;
    static constexpr int STAGES = BM * BN > 64 * 64 ? 3 : 4;
    static constexpr int SQ_AT = STAGES * STAGE > RED ? STAGES * STAGE : RED;    // row sums of squares of the FUSED kernels
    static constexpr size_t NEED = (size_t)(SQ_AT + (KS + 1) * BM) * sizeof(float);
    // A large block has an SM to itself: two of them share its issue slots while others idle (chained launches place the
    // next product's blocks before this one's have left).  Only the 32 x 64 tiles fit twice: 512 x 512 x 64 4.0 -> 3.2 us, GPT forward of
    // 4 layers, C 320, 200 tokens 234 -> 204; nothing measured got slower.
    static constexpr size_t ALONE = 116 * 1024;
    static constexpr size_t SMEM = PM * PN >= 16 && NEED < ALONE ? ALONE : NEED;
};

// Sum of a tile element's partial sums: the k groups of this block, or the blocks of the cluster (every load on its way before the
// first addition).
template <int KS, int PATCH>
__device__ __forceinline__ float4 patch_sum(const float* q, int parts) {
    if (parts > 1) {
        float4 u[MAX_PARTS];
#pragma unroll
        for (int z = 0; z < MAX_PARTS; ++z)
            if (z < parts) u[z] = *reinterpret_cast<const float4*>(cg::this_cluster().map_shared_rank(q, z));
        float4 v = u[0];
#pragma unroll
        for (int z = 1; z < MAX_PARTS; ++z)
            if (z < parts) { v.x += u[z].x; v.y += u[z].y; v.z += u[z].z; v.w += u[z].w; }
        return v;
    }
    float4 v = *reinterpret_cast<const float4*>(q);
#pragma unroll
    for (int z = 1; z < KS; ++z) {
        const float4 u = *reinterpret_cast<const float4*>(q + z * PATCH);
        v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
    }
    return v;
}

// What follows a tile's products: KS patches of BM x BN partial sums lie in `red` (rows of BN + 4), with FUSED the rows' sums of squares
// in sq_s [KS][BM] (and room for BM more).  Meets, adds the k groups and the blocks of the cluster, applies norm, rotation and epilogue, and stores.
// What the epilogue reads from global memory is requested before the block's meeting (behind it, it cost 400 to 700 cycles of a product's 5000), and
// behind a cluster's, whose arrival would wait for it, beside the reads of the other blocks' patches.
template <int BM, int BN, int KS, int THREADS, bool FUSED>
__device__ __forceinline__ void finish_tile(const GemmArgs& g, float* const red, float* const sq_s, const int m0, const int n0, const int parts,
                                            const int rank) {
    constexpr int RLD = BN + 4, ITEMS = (BM * BN / 4 + THREADS - 1) / THREADS;     // four columns each
    // Rows of the tile this block finishes: all of them, or its share of the cluster's.
    int r_begin = 0, r_end = BM;
    if (parts > 1) {
        const int share = (BM + parts - 1) / parts;
        r_begin = rank * share;
        r_end = min(BM, r_begin + share);
    }
    const int first = r_begin * (BN / 4) + threadIdx.x, last = r_end * (BN / 4);
    const bool from_r = g.epi == DEERS_EPI_ADD, from_aux = g.epi == DEERS_EPI_MUL_AUX2;
    float4 ext[ITEMS], c4[FUSED ? ITEMS : 1], s4[FUSED ? ITEMS : 1];
    // Where a thread's items lie in one column (all tiles but the 96 wide) it divides once, not per item: with that and the square root
    // and division of the norm in every item a tile of 128 x 64 took 9000 to 11000 cycles here, one of 16 x 32 2500 (1024 x 576 and 768 x 192 in the
    // model 13.7 -> 12.0 us; 22 M parameters, 4 training steps and a forward 5130 -> 5040).
    constexpr bool ONE_COLUMN = THREADS % (BN / 4) == 0;
    constexpr int ROW_STEP = THREADS / (BN / 4);
    bool second[ITEMS];                                             // the column lies in the second half of its head
    auto request = [&]() {
        unsigned pos = 0, hc = 0;
        if constexpr (FUSED) {
            if (g.rope_cols) {
                pos = (unsigned)(m0 + first / (BN / 4)) % (unsigned)g.rope_t;
                hc = (unsigned)(n0 + first % (BN / 4) * 4) % (unsigned)g.rope_d;
            }
        }
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const int idx = first + i * THREADS, m = m0 + idx / (BN / 4), n = n0 + (idx % (BN / 4)) * 4;
            const bool in = idx < last && m < g.M && n < g.N;
            if (in && (from_r || from_aux))
                ext[i] = ld4(from_r ? g.r + (long long)m * g.ldr + n : g.aux + (long long)m * g.ldc + n, g.N - n, g.c_vec);
            second[i] = false;
            if constexpr (FUSED) {
                if (g.rope_cols && i > 0) {
                    if constexpr (ONE_COLUMN) {
                        pos += ROW_STEP;
                        if (pos >= (unsigned)g.rope_t) pos = g.rope_t >= ROW_STEP ? pos - g.rope_t : pos % (unsigned)g.rope_t;
                    } else {
                        pos = (unsigned)m % (unsigned)g.rope_t;
                        hc = (unsigned)n % (unsigned)g.rope_d;
                    }
                }
                if (in && n < g.rope_cols) {
                    const unsigned half = (unsigned)g.rope_d / 2;
                    second[i] = hc >= half;
                    const size_t at = (size_t)(pos * half + (second[i] ? hc - half : hc));
                    c4[i] = *reinterpret_cast<const float4*>(g.cosv + at);
                    s4[i] = *reinterpret_cast<const float4*>(g.sinv + at);
                }
            }
        }
    };
    if (parts == 1) request();
    __syncthreads();
    if (parts > 1) {
        for (int idx = threadIdx.x; idx < BM * BN / 4; idx += THREADS) {
            float* q = red + (idx / (BN / 4)) * RLD + (idx % (BN / 4)) * 4;
            float4 v = *reinterpret_cast<float4*>(q);
#pragma unroll
            for (int z = 1; z < KS; ++z) {
                const float4 u = *reinterpret_cast<const float4*>(q + z * BM * RLD);
                v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
            }
            *reinterpret_cast<float4*>(q) = v;
        }
        if constexpr (FUSED) {
            if (threadIdx.x < BM) {
                float v = sq_s[threadIdx.x];
#pragma unroll
                for (int z = 1; z < KS; ++z) v += sq_s[z * BM + threadIdx.x];
                sq_s[threadIdx.x] = v;
            }
        }
        cg::this_cluster().sync();
        request();
    }
    if constexpr (FUSED) {                                          // inverse norms, once per row, behind the sums [KS][BM]
        if (threadIdx.x < BM) {
            const int row = threadIdx.x;
            float t = 0.f;
            if (parts > 1) {
                for (int z = 0; z < parts; ++z) t += *cg::this_cluster().map_shared_rank(sq_s + row, z);
            } else {
#pragma unroll
                for (int z = 0; z < KS; ++z) t += sq_s[z * BM + row];
            }
            const float inv = 1.0f / sqrtf(t * g.inv_n + g.eps);
            sq_s[KS * BM + row] = inv;
            if (g.inv && n0 == 0 && row >= r_begin && row < r_end && m0 + row < g.M) g.inv[m0 + row] = inv;
        }
        __syncthreads();
    }
    chain_next();                                                   // (at the loop or earlier, successors crowd out the side stream)
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const int idx = first + i * THREADS;
        if (idx >= last) break;
        const int row = idx / (BN / 4), col = (idx % (BN / 4)) * 4;
        const int m = m0 + row, n = n0 + col;
        if (m >= g.M || n >= g.N) continue;
        const float* q = red + row * RLD + col;
        const float4 v = patch_sum<KS, BM * RLD>(q, parts);
        const int valid = g.N - n;
        float o[4] = {v.x, v.y, v.z, v.w}, x[4] = {0.f, 0.f, 0.f, 0.f};
        float* cp = g.c + (long long)m * g.ldc + n;
        if constexpr (FUSED) {
            const float inv = sq_s[KS * BM + row];
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] *= inv;
            if (n < g.rope_cols) {
                // the other half of the head lies in this tile (tiles hold whole heads); rounded as the rotary pack does
                const int half = g.rope_d / 2;
                const float4 u = patch_sum<KS, BM * RLD>(second[i] ? q - half : q + half, parts);
                const float p[4] = {u.x * inv, u.y * inv, u.z * inv, u.w * inv};
                const float cs[4] = {c4[i].x, c4[i].y, c4[i].z, c4[i].w}, sn[4] = {s4[i].x, s4[i].y, s4[i].z, s4[i].w};
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    o[e] = second[i] ? __fadd_rn(__fmul_rn(p[e], -sn[e]), __fmul_rn(o[e], cs[e]))
                                     : __fadd_rn(__fmul_rn(o[e], cs[e]), __fmul_rn(p[e], sn[e]));
            }
        }
        if (from_r) {
            o[0] = ext[i].x + o[0]; o[1] = ext[i].y + o[1]; o[2] = ext[i].z + o[2]; o[3] = ext[i].w + o[3];
        } else if (g.epi == DEERS_EPI_RELU_SQ) {
#pragma unroll
            for (int e = 0; e < 4; ++e) { x[e] = fmaxf(o[e], 0.f); o[e] = x[e] * x[e]; }
        } else if (from_aux) {
            o[0] *= ext[i].x; o[1] *= ext[i].y; o[2] *= ext[i].z; o[3] *= ext[i].w;
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] = o[e] + o[e];
        }
        if (g.c_vec && valid >= 4) {
            *reinterpret_cast<float4*>(cp) = make_float4(o[0], o[1], o[2], o[3]);
            if (g.epi == DEERS_EPI_RELU_SQ && g.aux)
                *reinterpret_cast<float4*>(g.aux + (long long)m * g.ldc + n) = make_float4(x[0], x[1], x[2], x[3]);
        } else {
            for (int e = 0; e < 4 && e < valid; ++e) {
                cp[e] = o[e];
                if (g.epi == DEERS_EPI_RELU_SQ && g.aux) g.aux[(long long)m * g.ldc + n + e] = x[e];
            }
        }
    }
    if (parts > 1) cg::this_cluster().sync();                       // nobody leaves while a peer still reads its patch
}

// One tile (tile_m, tile_n) of a product and one part of its K.  setup() only computes addresses and may run before the
// predecessor has finished; run() does the work.
template <int PM, int PN, int KS, bool A_MN, bool B_MN, bool FUSED, bool LOOSE>
struct TileProduct {
    using S = GemmShape<PM, PN, KS, A_MN, B_MN, LOOSE>;
    static constexpr int BM = S::BM, BN = S::BN, STAGES = S::STAGES, KG = S::KG;
    typename S::OA la;
    typename S::OB lb;
    int m0, n0, kbeg, kend;
    __device__ __forceinline__ void setup(const GemmArgs& g, int tile_m, int tile_n, int part) {
        const int tid = threadIdx.x % GT, kg = threadIdx.x / GT;
        m0 = tile_m * BM; n0 = tile_n * BN;
        kbeg = part * g.k_chunk;
        kend = min(g.K, kbeg + g.k_chunk);
        la.init(g.a, g.lda, m0, g.M, kbeg + kg * KG, tid);
        lb.init(g.b, g.ldb, n0, g.N, kbeg + kg * KG, tid);
    }
    __device__ __forceinline__ void run(const GemmArgs& g, int parts, int rank);
};

template <int PM, int PN, int KS, bool A_MN, bool B_MN, bool FUSED, bool LOOSE>
__device__ __forceinline__ void TileProduct<PM, PN, KS, A_MN, B_MN, FUSED, LOOSE>::run(const GemmArgs& g, const int parts, const int rank) {
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x % GT, kg = threadIdx.x / GT;        // position in the tile, k group
    const int w = tid / 32, lane = tid % 32;
    const int ty = (w & 1) * 4 + (lane & 1) + 2 * ((lane >> 3) & 1), tx = (w >> 1) * 8 + ((lane >> 1) & 3) + 4 * (lane >> 4);
    const int nk = kend > kbeg ? (kend - kbeg + BK - 1) / BK : 0;
    // FUSED: SQ_LANES threads of a group share a row's squares of the group's k, SQ_K each
    constexpr int SQ_LANES = GT / BM, SQ_K = KG / SQ_LANES;
    float sq = 0.f;
    float* const sq_s = smem + S::SQ_AT;                            // [KS][BM]

    int kv = kend - kbeg - kg * KG;                                 // k left to fetch (of the group's share and what follows)
    float* const ring = smem + kg * (S::OA::FLOATS + S::OB::FLOATS);
    int st_in = 0, left = nk;                                       // stage to fill next
    auto fetch = [&]() {
        if (left > 0) {
            la.fetch(ring + st_in, kv, g.a_vec, g.lda, g.M - m0, tid);
            lb.fetch(ring + st_in + S::OA::FLOATS, kv, g.b_vec, g.ldb, g.N - n0, tid);
            kv -= BK;
            --left;
            st_in = st_in == (STAGES - 1) * S::STAGE ? 0 : st_in + S::STAGE;
        }
        cp_commit();
    };
#pragma unroll
    for (int t = 0; t < STAGES - 1; ++t) fetch();

    // Pairs of products: neighbouring columns with B in MN order (a's element twice), even and odd k with both operands in K order
    // (an A in MN order would cost two moves per pair: 192 x 768 x 1024 17.2 us, single products 12.6).
    // Tall patches with both operands in MN order pair rows instead: fewer doubled elements (0.89 of the FMA rate in a bare loop
    // of 8 x 6, 0.81 with columns).
    constexpr bool PAIR_M = A_MN && B_MN && PM >= 8, PAIR_N = B_MN && !PAIR_M, PAIR_K = !A_MN && !B_MN && PM * PN <= 16;
    constexpr bool AHEAD = B_MN || PM * PN <= 16;                   // registers for the next fragments as well
    constexpr int U = !AHEAD || (!(A_MN && B_MN) && PM * PN <= 16) ? 4 : 2;
    constexpr int PR = PAIR_M ? PM / 2 : PM, PC = PAIR_N ? PN / 2 : PAIR_K || PAIR_M ? PN : 1;
    uint64_t acc2[PR][PC];
#pragma unroll
    for (int i = 0; i < PR; ++i)
#pragma unroll
        for (int j = 0; j < PC; ++j) acc2[i][j] = 0;
    float acc[PM][PN];
#pragma unroll
    for (int i = 0; i < PM; ++i)
#pragma unroll
        for (int j = 0; j < PN; ++j) acc[i][j] = 0.f;

    int st_out = 0;
    for (int t = 0; t < nk; ++t) {
        cp_wait<STAGES - 2>();
        group_sync(kg);                                             // stage t has landed, stage t-1 is free
        fetch();
        const float* sa = ring + st_out;
        const float* sb = sa + S::OA::FLOATS;
        if constexpr (FUSED) {
            const float* q = sa + (tid / SQ_LANES) * S::OA::LD + (tid % SQ_LANES) * SQ_K;
            if constexpr (SQ_K == 2) {
                const float2 x = *reinterpret_cast<const float2*>(q);
                sq = fmaf(x.x, x.x, sq); sq = fmaf(x.y, x.y, sq);
            } else {
#pragma unroll
                for (int e = 0; e < SQ_K; e += 4) {
                    const float4 x = *reinterpret_cast<const float4*>(q + e);
                    sq = fmaf(x.x, x.x, sq); sq = fmaf(x.y, x.y, sq); sq = fmaf(x.z, x.z, sq); sq = fmaf(x.w, x.w, sq);
                }
            }
        }
        float a[AHEAD ? 2 : 1][U][PM], b[AHEAD ? 2 : 1][U][PN];     // fragments of U k (and of the next U)
        if constexpr (AHEAD) {
            S::OA::template read<PM, U>(sa, ty, 0, a[0]);
            S::OB::template read<PN, U>(sb, tx, 0, b[0]);
        }
#pragma unroll
        for (int k = 0; k < KG; k += U) {
            const int cur = AHEAD ? (k / U) & 1 : 0;
            if constexpr (!AHEAD) {
                S::OA::template read<PM, U>(sa, ty, k, a[0]);
                S::OB::template read<PN, U>(sb, tx, k, b[0]);
            } else if (k + U < KG) {
                S::OA::template read<PM, U>(sa, ty, k + U, a[cur ^ 1]);
                S::OB::template read<PN, U>(sb, tx, k + U, b[cur ^ 1]);
            }
#pragma unroll
            for (int kk = 0; kk < U; ++kk) {
                if constexpr (PAIR_K) {
                    if (kk % 2 == 0) {
#pragma unroll
                        for (int j = 0; j < PN; ++j)
#pragma unroll
                            for (int i = 0; i < PM; ++i)
                                acc2[i][j] = fma2(pack_f32x2(a[cur][kk][i], a[cur][kk + 1][i]), pack_f32x2(b[cur][kk][j], b[cur][kk + 1][j]), acc2[i][j]);
                    }
                } else if constexpr (PAIR_M) {
                    uint64_t bd[PN];
#pragma unroll
                    for (int j = 0; j < PN; ++j) bd[j] = pack_f32x2(b[cur][kk][j], b[cur][kk][j]);
#pragma unroll
                    for (int i = 0; i < PM / 2; ++i)
#pragma unroll
                        for (int j = 0; j < PN; ++j) acc2[i][j] = fma2(pack_f32x2(a[cur][kk][2 * i], a[cur][kk][2 * i + 1]), bd[j], acc2[i][j]);
                } else if constexpr (PAIR_N) {
                    uint64_t ad[PM];
#pragma unroll
                    for (int i = 0; i < PM; ++i) ad[i] = pack_f32x2(a[cur][kk][i], a[cur][kk][i]);
#pragma unroll
                    for (int j = 0; j < PN / 2; ++j)
#pragma unroll
                        for (int i = 0; i < PM; ++i) acc2[i][j] = fma2(ad[i], pack_f32x2(b[cur][kk][2 * j], b[cur][kk][2 * j + 1]), acc2[i][j]);
                } else {
#pragma unroll
                    for (int i = 0; i < PM; ++i)
#pragma unroll
                        for (int j = 0; j < PN; ++j) acc[i][j] = fmaf(a[cur][kk][i], b[cur][kk][j], acc[i][j]);
                }
            }
        }
        st_out = st_out == (STAGES - 1) * S::STAGE ? 0 : st_out + S::STAGE;
    }
    cp_wait<0>();
    __syncthreads();                                                // operand stages are free: patches meet here
#pragma unroll
    for (int i = 0; i < PR; ++i)
#pragma unroll
        for (int j = 0; j < PC; ++j) {
            if constexpr (PAIR_M) unpack_f32x2(acc2[i][j], acc[2 * i][j], acc[2 * i + 1][j]);
            if constexpr (PAIR_N) unpack_f32x2(acc2[i][j], acc[i][2 * j], acc[i][2 * j + 1]);
            if constexpr (PAIR_K) {
                float even, odd;
                unpack_f32x2(acc2[i][j], even, odd);
                acc[i][j] = even + odd;
            }
        }

    if constexpr (FUSED) {
#pragma unroll
        for (int o = 1; o < SQ_LANES; o *= 2) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if (tid % SQ_LANES == 0) sq_s[kg * BM + tid / SQ_LANES] = sq;
    }
    float* red = smem;
#pragma unroll
    for (int i = 0; i < PM; ++i) {
        float* row = red + (kg * BM + S::OA::template index<PM>(ty, i)) * S::RLD;
        if constexpr (B_MN) {
#pragma unroll
            for (int j = 0; j < PN; j += 4) {
                float* q = row + S::OB::template index<PN>(tx, j);
                if (PN - j >= 4) *reinterpret_cast<float4*>(q) = make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
                else *reinterpret_cast<float2*>(q) = make_float2(acc[i][j], acc[i][j + 1]);
            }
        } else {
#pragma unroll
            for (int j = 0; j < PN; ++j) row[S::OB::template index<PN>(tx, j)] = acc[i][j];
        }
    }
    finish_tile<BM, BN, KS, S::THREADS, FUSED>(g, red, sq_s, m0, n0, parts, rank);
}

template <int PM, int PN, int KS, bool A_MN, bool B_MN, bool FUSED, bool LOOSE>
__global__ void __launch_bounds__(GT * KS, PM * PN < 16 && !LOOSE ? 2 : 1) gemm_f32_kernel(const GemmArgs g) {
    TileProduct<PM, PN, KS, A_MN, B_MN, FUSED, LOOSE> tile;
    tile.setup(g, blockIdx.y, blockIdx.x, blockIdx.z);
    chain_wait();
    tile.run(g, gridDim.z, blockIdx.z);
}

template <int PM, int PN, int KS, bool A_MN, bool B_MN, bool FUSED, bool LOOSE>
int launch_variant(deers_ctx* ctx, const GemmPlan& p, const GemmArgs& g) {
    using S = GemmShape<PM, PN, KS, A_MN, B_MN, LOOSE>;
    const auto kernel = gemm_f32_kernel<PM, PN, KS, A_MN, B_MN, FUSED, LOOSE>;
    DEERS_SMEM_ONCE(ctx, (gemm_f32_kernel<PM, PN, KS, A_MN, B_MN, FUSED, LOOSE>), S::SMEM);
    const dim3 grid((g.N + S::BN - 1) / S::BN, (g.M + S::BM - 1) / S::BM, p.parts);
    DEERS_CUDA_TRY(ctx, launch_chained(ctx, kernel, grid, S::THREADS, S::SMEM, dim3(1, 1, p.parts), g));
    return DEERS_OK;
}

template <int PM, int PN, int KS, bool LOOSE>
int launch_orders(deers_ctx* ctx, const GemmPlan& p, const GemmArgs& g, int a_mn, int b_mn, bool fused) {
    if (fused) return launch_variant<PM, PN, KS, false, true, true, LOOSE>(ctx, p, g);
    if (a_mn) return b_mn ? launch_variant<PM, PN, KS, true, true, false, LOOSE>(ctx, p, g) : launch_variant<PM, PN, KS, true, false, false, LOOSE>(ctx, p, g);
    return b_mn ? launch_variant<PM, PN, KS, false, true, false, LOOSE>(ctx, p, g) : launch_variant<PM, PN, KS, false, false, false, LOOSE>(ctx, p, g);
}

template <bool LOOSE>
int launch_tiles(deers_ctx* ctx, const GemmPlan& p, const GemmArgs& g, int a_mn, int b_mn, bool fused) {
    switch (p.cfg) {
        case 0: return launch_orders<8, 8, 2, LOOSE>(ctx, p, g, a_mn, b_mn, fused);
        case 1: return launch_orders<8, 4, 4, LOOSE>(ctx, p, g, a_mn, b_mn, fused);
        case 2: return launch_orders<4, 4, 4, LOOSE>(ctx, p, g, a_mn, b_mn, fused);
        case 3: return launch_orders<4, 2, 4, LOOSE>(ctx, p, g, a_mn, b_mn, fused);
        case 4: return launch_orders<8, 6, 4, LOOSE>(ctx, p, g, a_mn, b_mn, fused);
        case 5: return launch_orders<4, 6, 4, LOOSE>(ctx, p, g, a_mn, b_mn, fused);
        default: return launch_orders<2, 2, 4, LOOSE>(ctx, p, g, a_mn, b_mn, fused);
    }
}

}  // namespace
