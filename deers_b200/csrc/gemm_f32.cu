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
#include "common.cuh"
#include "f32_util.cuh"

#include <cooperative_groups.h>

namespace {
namespace cg = cooperative_groups;

constexpr int GT = 128;                                 // threads of a k group
constexpr int BK = 64;                                  // depth of one stage, shared evenly by the k groups
constexpr int MAX_PARTS = 8;                            // blocks of a cluster along K (portable cluster size)

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
    static constexpr int NP = ROWS * LEN / 4 / GT;                  // 16-byte pieces per thread and stage
    static_assert(NP * GT * 4 == ROWS * LEN, "whole pieces per thread");
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
            const int idx = t + i * GT;
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
                const float* p = src[0] - (row_of(t / (LEN / 4)) * ld + t % (LEN / 4) * 4) + (row * ld + col);
                float* d = s + row * LD + col;
#pragma unroll 4
                for (int i = 0; i < 4 * NP; ++i) {
                    const bool in = MN ? row < kv && col < rv : row < rv && col < kv;
                    cp4(d, in ? p : base, in ? 4 : 0);
                    row += GT / LEN; p += GT / LEN * ld; d += GT / LEN * LD;
                }
                src[0] += step;
                return;
            }
        }
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
    static constexpr size_t NEED = (size_t)(SQ_AT + KS * BM) * sizeof(float);
    // A large block has an SM to itself: two of them share its issue slots while others idle (chained launches place the
    // next product's blocks before this one's have left).  Only the 32 x 64 tiles fit twice: 512 x 512 x 64 4.0 -> 3.2 us, GPT forward of
    // 4 layers, C 320, 200 tokens 234 -> 204; nothing measured got slower.
    static constexpr size_t ALONE = 116 * 1024;
    static constexpr size_t SMEM = PM * PN >= 16 && NEED < ALONE ? ALONE : NEED;
};

// Sum of a tile element's partial sums: the k groups of this block, or the blocks of the cluster.
template <int KS, int PATCH>
__device__ __forceinline__ float4 patch_sum(const float* q, int parts) {
    if (parts > 1) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int z = 0; z < parts; ++z) {
            const float4 u = *reinterpret_cast<const float4*>(cg::this_cluster().map_shared_rank(q, z));
            v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
        }
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
#pragma unroll
            for (int e = 0; e < SQ_K; e += 4) {
                const float4 x = *reinterpret_cast<const float4*>(q + e);
                sq = fmaf(x.x, x.x, sq); sq = fmaf(x.y, x.y, sq); sq = fmaf(x.z, x.z, sq); sq = fmaf(x.w, x.w, sq);
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
    __syncthreads();

    // Rows of the tile this block finishes: all of them, or its share of the cluster's.
    int r_begin = 0, r_end = BM;
    if (parts > 1) {
        for (int idx = threadIdx.x; idx < BM * BN / 4; idx += S::THREADS) {
            float* q = red + (idx / (BN / 4)) * S::RLD + (idx % (BN / 4)) * 4;
            float4 v = *reinterpret_cast<float4*>(q);
#pragma unroll
            for (int z = 1; z < KS; ++z) {
                const float4 u = *reinterpret_cast<const float4*>(q + z * BM * S::RLD);
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
        const int share = (BM + parts - 1) / parts;
        r_begin = rank * share;
        r_end = min(BM, r_begin + share);
    }
    chain_next();                                                   // (at the loop or earlier, successors crowd out the side stream)
    for (int idx = r_begin * (BN / 4) + threadIdx.x; idx < r_end * (BN / 4); idx += S::THREADS) {
        const int row = idx / (BN / 4), col = (idx % (BN / 4)) * 4;
        const int m = m0 + row, n = n0 + col;
        const float* q = red + row * S::RLD + col;
        const float4 v = patch_sum<KS, BM * S::RLD>(q, parts);
        if (m >= g.M || n >= g.N) continue;
        const int valid = g.N - n;
        float o[4] = {v.x, v.y, v.z, v.w}, x[4] = {0.f, 0.f, 0.f, 0.f};
        float* cp = g.c + (long long)m * g.ldc + n;
        if constexpr (FUSED) {
            float t = 0.f;
            if (parts > 1) {
                for (int z = 0; z < parts; ++z) t += *cg::this_cluster().map_shared_rank(sq_s + row, z);
            } else {
#pragma unroll
                for (int z = 0; z < KS; ++z) t += sq_s[z * BM + row];
            }
            const float inv = 1.0f / sqrtf(t * g.inv_n + g.eps);
            if (g.inv && n == 0) g.inv[m] = inv;
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] *= inv;
            if (n < g.rope_cols) {
                // the other half of the head lies in this tile (tiles hold whole heads); rounded as the rotary pack does
                const int half = g.rope_d / 2, hc = n % g.rope_d;
                const bool second = hc >= half;
                const float4 u = patch_sum<KS, BM * S::RLD>(second ? q - half : q + half, parts);
                const long long at = (long long)(m % g.rope_t) * half + (second ? hc - half : hc);
                const float4 c4 = *reinterpret_cast<const float4*>(g.cosv + at), s4 = *reinterpret_cast<const float4*>(g.sinv + at);
                const float p[4] = {u.x * inv, u.y * inv, u.z * inv, u.w * inv}, cs[4] = {c4.x, c4.y, c4.z, c4.w}, sn[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    o[e] = second ? __fadd_rn(__fmul_rn(p[e], -sn[e]), __fmul_rn(o[e], cs[e])) : __fadd_rn(__fmul_rn(o[e], cs[e]), __fmul_rn(p[e], sn[e]));
            }
        }
        if (g.epi == DEERS_EPI_ADD) {
            const float4 t = ld4(g.r + (long long)m * g.ldr + n, valid, g.c_vec);
            o[0] = t.x + o[0]; o[1] = t.y + o[1]; o[2] = t.z + o[2]; o[3] = t.w + o[3];
        } else if (g.epi == DEERS_EPI_RELU_SQ) {
#pragma unroll
            for (int e = 0; e < 4; ++e) { x[e] = fmaxf(o[e], 0.f); o[e] = x[e] * x[e]; }
        } else if (g.epi == DEERS_EPI_MUL_AUX2) {
            const float4 t = ld4(g.aux + (long long)m * g.ldc + n, valid, g.c_vec);
            o[0] *= t.x; o[1] *= t.y; o[2] *= t.z; o[3] *= t.w;
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

template <int PM, int PN, int KS, bool A_MN, bool B_MN, bool FUSED, bool LOOSE>
__global__ void __launch_bounds__(GT * KS) gemm_f32_kernel(const GemmArgs g) {
    TileProduct<PM, PN, KS, A_MN, B_MN, FUSED, LOOSE> tile;
    tile.setup(g, blockIdx.y, blockIdx.x, blockIdx.z);
    chain_wait();
    tile.run(g, gridDim.z, blockIdx.z);
}

// Several products of one shape of operands (both in MN order) and one K in a launch: the weight gradients of a block, whose
// tiles do not fill the chip one product at a time.  blockIdx.x counts the tiles of all of them.
struct GemmGroup {
    GemmArgs g[GEMM_GROUP_MAX];
    int first[GEMM_GROUP_MAX];       // first tile of a product
    int tiles_n[GEMM_GROUP_MAX];
    int n;
    __device__ __forceinline__ int pick(int tile) const {
        int i = 0;
        while (i + 1 < n && tile >= first[i + 1]) ++i;
        return i;
    }
    __device__ __forceinline__ int tile_m(int i, int tile) const { return (tile - first[i]) / tiles_n[i]; }
    __device__ __forceinline__ int tile_n(int i, int tile) const { return (tile - first[i]) % tiles_n[i]; }
    __device__ __forceinline__ const GemmArgs& args(int i) const { return g[i]; }
};

template <int PM, int PN, int KS>
__global__ void __launch_bounds__(GT * KS) gemm_f32_group_kernel(const __grid_constant__ GemmGroup gg) {
    const int i = gg.pick(blockIdx.x);
    TileProduct<PM, PN, KS, true, true, false, true> tile;
    tile.setup(gg.args(i), gg.tile_m(i, blockIdx.x), gg.tile_n(i, blockIdx.x), blockIdx.z);
    chain_wait();
    tile.run(gg.args(i), gridDim.z, blockIdx.z);
}

struct GemmPlan {
    int cfg;        // index into kVariants
    int parts, k_chunk;
    int waves;      // blocks an SM runs one after another
    double cost;    // cycles
};

// Tile variants: the cycles at 1.965 GHz that the choice reckons with, a block's walk over 64 k and what a launch costs around it.
// They were measured on loops of single products, one figure for every order.  The present ones walk (both in MN order / A in K and B in
// MN / both in K): 64 x 128 5810 / 6210 / 8180, 64 x 64 2920 / 3680 / 3990, 32 x 64 1850 / 1810 / 2200, 32 x 32 1690 / 1910 / 1740,
// 64 x 96 4620 / 4710 / 5250, 32 x 96 2430 / 2900 / 3280, and 3800 to 9200 around it (148 tiles, K 320 and 1600).  The 96-wide tiles are
// there for products whose 64-wide ones just miss one wave (1024 x 768: 192 tiles on 148 SMs, 128 of 64 x 96; 13.3 -> 11.7 us at K =
// 192, and 16.3 -> 13.7 for 1024 x 192 x 768 in clusters of four).
struct Variant { int bm, bn; double walk, around; };
constexpr Variant kVariants[6] = {{64, 128, 7420, 6000}, {64, 64, 3700, 4900}, {32, 64, 2360, 4000}, {32, 32, 1680, 3200}, {64, 96, 5400, 5300}, {32, 96, 3200, 4300}};

// How many clusters of 1..MAX_PARTS blocks (one block per SM) the device holds at a time: a cluster lives inside one
// GPC, so e.g. 48 clusters of three do not fit 148 SMs although their 144 blocks would.
int cluster_capacity(deers_ctx* ctx) {
    if (ctx->cluster_capacity[1] > 0) return DEERS_OK;
    static std::atomic<int> known[64][MAX_PARTS + 1];                    // asked once per device: a tenth of a millisecond each
    std::atomic<int>* dev = known[ctx->device & 63];
    if (dev[1].load(std::memory_order_acquire) > 0) {
        for (int parts = 1; parts <= MAX_PARTS; ++parts) ctx->cluster_capacity[parts] = dev[parts].load(std::memory_order_relaxed);
        return DEERS_OK;
    }
    using S = GemmShape<8, 4, 4, false, true, false>;
    const auto kernel = gemm_f32_kernel<8, 4, 4, false, true, false, false>;
    DEERS_SMEM_ONCE(ctx, (gemm_f32_kernel<8, 4, 4, false, true, false, false>), S::SMEM);
    for (int parts = 2; parts <= MAX_PARTS; ++parts) {
        cudaLaunchConfig_t lc{};
        lc.gridDim = dim3(1, 1, parts);
        lc.blockDim = dim3(S::THREADS);
        lc.dynamicSmemBytes = S::SMEM;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = 1; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = (unsigned)parts;
        lc.attrs = at; lc.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kernel, &lc) != cudaSuccess) { cudaGetLastError(); n = 0; }
        ctx->cluster_capacity[parts] = n;
        dev[parts].store(n, std::memory_order_relaxed);
    }
    ctx->cluster_capacity[1] = ctx->sm_count;
    dev[1].store(ctx->sm_count, std::memory_order_release);
    return DEERS_OK;
}

// Picks the variant and the K split with the least estimated time: the blocks an SM has to run one after another times
// a block's walk over its K, plus what a block spends before and after it (and at the cluster's meeting).
// n products of one K; whole_heads: tiles must hold whole heads of that many columns (0: any).  cfg < 0: no variant does.
GemmPlan plan_gemm(int n, const int* M, const int* N, int K, const int* capacity, int whole_heads) {
    GemmPlan best{};
    best.cfg = -1;
    best.cost = 1e30;
    double best_cost = -1.0;
    const int steps = (K + BK - 1) / BK;
    for (int c = 0; c < 6; ++c) {
        const Variant& v = kVariants[c];
        if (whole_heads && v.bn % whole_heads) continue;
        long long tiles = 0;
        for (int i = 0; i < n; ++i) tiles += (long long)((M[i] + v.bm - 1) / v.bm) * ((N[i] + v.bn - 1) / v.bn);
        for (int parts = 1; parts <= MAX_PARTS; ++parts) {
            const int chunk = (steps + parts - 1) / parts;
            if (parts > 1 && (chunk < 2 || (long long)chunk * (parts - 1) >= steps)) continue;      // no empty part
            if (capacity[parts] < 1) continue;
            const double waves = (double)((tiles + capacity[parts] - 1) / capacity[parts]);
            const double cost = waves * chunk * v.walk + v.around + 1200.0 * (waves - 1.0) + (parts > 1 ? 3300.0 : 0.0);
            if (best_cost < 0.0 || cost < best_cost) {
                best_cost = cost;
                best.cost = cost; best.cfg = c; best.parts = parts; best.k_chunk = chunk * BK; best.waves = (int)waves;
            }
        }
    }
    if (K == 0) { best.parts = 1; best.k_chunk = BK; }
    return best;
}

template <int PM, int PN, int KS, bool A_MN, bool B_MN, bool FUSED = false, bool LOOSE = false>
int launch_variant(deers_ctx* ctx, const GemmPlan& p, const GemmArgs& g) {
    if constexpr (!LOOSE) {
        if (!g.a_vec || !g.b_vec) return launch_variant<PM, PN, KS, A_MN, B_MN, FUSED, true>(ctx, p, g);
    }
    using S = GemmShape<PM, PN, KS, A_MN, B_MN, LOOSE>;
    const auto kernel = gemm_f32_kernel<PM, PN, KS, A_MN, B_MN, FUSED, LOOSE>;
    DEERS_SMEM_ONCE(ctx, (gemm_f32_kernel<PM, PN, KS, A_MN, B_MN, FUSED, LOOSE>), S::SMEM);
    const dim3 grid((g.N + S::BN - 1) / S::BN, (g.M + S::BM - 1) / S::BM, p.parts);
    DEERS_CUDA_TRY(ctx, launch_chained(ctx, kernel, grid, S::THREADS, S::SMEM, dim3(1, 1, p.parts), g));
    return DEERS_OK;
}

template <int PM, int PN, int KS>
int launch_orders(deers_ctx* ctx, const GemmPlan& p, const GemmArgs& g, int a_mn, int b_mn, bool fused) {
    if (fused) return launch_variant<PM, PN, KS, false, true, true>(ctx, p, g);
    if (a_mn) return b_mn ? launch_variant<PM, PN, KS, true, true>(ctx, p, g) : launch_variant<PM, PN, KS, true, false>(ctx, p, g);
    return b_mn ? launch_variant<PM, PN, KS, false, true>(ctx, p, g) : launch_variant<PM, PN, KS, false, false>(ctx, p, g);
}

template <int PM, int PN, int KS>
int launch_group(deers_ctx* ctx, const GemmPlan& p, GemmGroup& gg) {
    using S = GemmShape<PM, PN, KS, true, true, true>;
    const auto kernel = gemm_f32_group_kernel<PM, PN, KS>;
    DEERS_SMEM_ONCE(ctx, (gemm_f32_group_kernel<PM, PN, KS>), S::SMEM);
    int tiles = 0;
    for (int i = 0; i < gg.n; ++i) {
        gg.first[i] = tiles;
        gg.tiles_n[i] = (gg.g[i].N + S::BN - 1) / S::BN;
        tiles += gg.tiles_n[i] * ((gg.g[i].M + S::BM - 1) / S::BM);
        gg.g[i].k_chunk = p.k_chunk;
    }
    DEERS_CUDA_TRY(ctx, launch_chained(ctx, kernel, dim3(tiles, 1, p.parts), S::THREADS, S::SMEM, dim3(1, 1, p.parts), gg));
    return DEERS_OK;
}

GemmArgs gemm_args(int M, int N, int K, const float* a, long long lda, const float* b, long long ldb, float* c, long long ldc, int epi,
                   const float* r, long long ldr, float* aux) {
    GemmArgs g{};
    g.a = a; g.b = b; g.c = c; g.r = r; g.aux = aux;
    g.lda = lda; g.ldb = ldb; g.ldc = ldc; g.ldr = ldr;
    g.M = M; g.N = N; g.K = K; g.epi = epi;
    g.a_vec = ((uintptr_t)a & 15u) == 0 && lda % 4 == 0;
    g.b_vec = ((uintptr_t)b & 15u) == 0 && ldb % 4 == 0;
    g.c_vec = ((uintptr_t)c & 15u) == 0 && ldc % 4 == 0 && (!r || (((uintptr_t)r & 15u) == 0 && ldr % 4 == 0)) &&
              (!aux || ((uintptr_t)aux & 15u) == 0);
    return g;
}

int launch_planned(deers_ctx* ctx, const GemmPlan& p, GemmArgs& g, int a_mn, int b_mn, bool fused) {
    g.k_chunk = p.k_chunk;
    int rc;
    {
        KernelTimerScope ts(ctx, DEERS_K_GEMM);
        if (p.cfg == 0) rc = launch_orders<8, 8, 2>(ctx, p, g, a_mn, b_mn, fused);
        else if (p.cfg == 1) rc = launch_orders<8, 4, 4>(ctx, p, g, a_mn, b_mn, fused);
        else if (p.cfg == 2) rc = launch_orders<4, 4, 4>(ctx, p, g, a_mn, b_mn, fused);
        else if (p.cfg == 3) rc = launch_orders<4, 2, 4>(ctx, p, g, a_mn, b_mn, fused);
        else if (p.cfg == 4) rc = launch_orders<8, 6, 4>(ctx, p, g, a_mn, b_mn, fused);
        else rc = launch_orders<4, 6, 4>(ctx, p, g, a_mn, b_mn, fused);
    }
    ctx->launches += 1;
    return rc;
}

}  // namespace

int launch_gemm_f32(deers_ctx* ctx, int M, int N, int K, const float* a, long long lda, int a_mn, const float* b,
                    long long ldb, int b_mn, float* c, long long ldc, int epi, const float* r, long long ldr, float* aux) {
    if (M == 0 || N == 0) return DEERS_OK;
    // Row tiles lie along gridDim.y, which ends at 65535: taller products (tiles are 32 rows or more) go in several launches.
    constexpr int MOST = 65535 * 32;
    for (; M > MOST; M -= MOST) {
        const int rc = launch_gemm_f32(ctx, MOST, N, K, a, lda, a_mn, b, ldb, b_mn, c, ldc, epi, r, ldr, aux);
        if (rc) return rc;
        a += a_mn ? MOST : MOST * lda;
        c += MOST * ldc;
        if (r) r += MOST * ldr;
        if (aux) aux += MOST * ldc;
    }
    const int rc = cluster_capacity(ctx);
    if (rc) return rc;
    const GemmPlan p = plan_gemm(1, &M, &N, K, ctx->cluster_capacity, 0);
    GemmArgs g = gemm_args(M, N, K, a, lda, b, ldb, c, ldc, epi, r, ldr, aux);
    return launch_planned(ctx, p, g, a_mn, b_mn, false);
}

// C = rmsnorm(A) * B with an optional rotation of the leading columns (see GemmNorm in common.cuh); M <= 65535 rows.
int launch_gemm_f32_norm(deers_ctx* ctx, int M, int N, int K, const float* a, const float* b, float* c, int epi, float* aux, const GemmNorm& f,
                         bool* rotated) {
    *rotated = false;
    if (M == 0 || N == 0) return DEERS_OK;
    const int rc = cluster_capacity(ctx);
    if (rc) return rc;
    GemmPlan p = plan_gemm(1, &M, &N, K, ctx->cluster_capacity, 0);
    GemmArgs g = gemm_args(M, N, K, a, K, b, N, c, N, epi, nullptr, 0, aux);
    if (f.rope_cols && f.rope_d % 8 == 0) {
        // A rotary launch of its own takes about 3000 cycles (1.5 us): rotate here unless tiles that hold whole heads cost more
        // than that (heads of 48 columns leave 32 x 96 and 64 x 96 tiles: 231 x 576 x 192 takes 7.5 us in them, 3.6 in 32 x 32).
        // Several waves of clusters do not count: the estimate takes them to follow one another without a gap (forwards of 4 layers,
        // rotating in them and beside: C 512, 256 tokens 363 and 335 us, C 384, 640 tokens 533 and 501).
        const GemmPlan w = plan_gemm(1, &M, &N, K, ctx->cluster_capacity, f.rope_d);
        if (w.cfg >= 0 && w.cost < p.cost + 3000.0 && (w.cost == p.cost || w.parts == 1 || w.waves == 1)) {
            p = w;
            *rotated = true;
            g.cosv = f.cosv; g.sinv = f.sinv; g.rope_cols = f.rope_cols; g.rope_d = f.rope_d; g.rope_t = f.rope_t;
        }
    }
    g.eps = f.eps; g.inv_n = (float)(1.0 / (double)K); g.inv = f.inv;
    return launch_planned(ctx, p, g, 0, 1, true);
}

// Whether the group of these products is one wave of blocks.  One of several waves keeps the SMs from what runs beside it until
// its last, where products on their own take turns with it (GPT training step of 6 layers, 1024 tokens: C 192, one wave, 980 us
// grouped and 998 apart; C 320 2235 and 2219; C 512 4472 and 4028).
bool gemm_f32_group_fits(deers_ctx* ctx, int n, const GemmTN* t, int K) {
    if (n < 1 || n > GEMM_GROUP_MAX || cluster_capacity(ctx)) return false;
    int M[GEMM_GROUP_MAX], N[GEMM_GROUP_MAX];
    for (int i = 0; i < n; ++i) { M[i] = t[i].M; N[i] = t[i].N; }
    return plan_gemm(n, M, N, K, ctx->cluster_capacity, 0).waves == 1;
}

// C_i = A_i^T B_i, A_i [K, M_i] and B_i [K, N_i] row-major, one K, in one launch.
int launch_gemm_f32_group(deers_ctx* ctx, int n, const GemmTN* t, int K) {
    if (n < 1 || n > GEMM_GROUP_MAX) return DEERS_ERR_SHAPE;
    const int rc = cluster_capacity(ctx);
    if (rc) return rc;
    GemmGroup gg{};
    int M[GEMM_GROUP_MAX], N[GEMM_GROUP_MAX];
    gg.n = n;
    for (int i = 0; i < n; ++i) {
        M[i] = t[i].M; N[i] = t[i].N;
        gg.g[i] = gemm_args(t[i].M, t[i].N, K, t[i].a, t[i].M, t[i].b, t[i].N, t[i].c, t[i].N, DEERS_EPI_NONE, nullptr, 0, nullptr);
    }
    const GemmPlan p = plan_gemm(n, M, N, K, ctx->cluster_capacity, 0);
    int res;
    {
        KernelTimerScope ts(ctx, DEERS_K_GEMM);
        if (p.cfg == 0) res = launch_group<8, 8, 2>(ctx, p, gg);
        else if (p.cfg == 1) res = launch_group<8, 4, 4>(ctx, p, gg);
        else if (p.cfg == 2) res = launch_group<4, 4, 4>(ctx, p, gg);
        else if (p.cfg == 3) res = launch_group<4, 2, 4>(ctx, p, gg);
        else if (p.cfg == 4) res = launch_group<8, 6, 4>(ctx, p, gg);
        else res = launch_group<4, 6, 4>(ctx, p, gg);
    }
    ctx->launches += 1;
    return res;
}

extern "C" size_t deers_b200_gemm_f32_workspace_bytes(deers_ctx* ctx, int32_t M, int32_t N, int32_t K) {
    if (!ctx || M < 0 || N < 0 || K < 0) return 0;
    return 0;                                                       // K splits meet in shared memory
}

extern "C" int deers_b200_gemm_f32(deers_ctx* ctx, int32_t M, int32_t N, int32_t K, const float* a, int64_t lda,
                                   int32_t a_mn_major, const float* b, int64_t ldb, int32_t b_mn_major, float* c,
                                   int64_t ldc, const deers_gemm_epilogue* epilogue, void* workspace,
                                   size_t workspace_bytes) {
    if (!ctx || !a || !b || !c) return DEERS_ERR_NULL;
    if (M < 0 || N < 0 || K < 0) return DEERS_ERR_SHAPE;
    if ((((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 3u) != 0) return DEERS_ERR_LAYOUT;
    if (lda < (a_mn_major ? M : K) || ldb < (b_mn_major ? N : K) || ldc < N) return DEERS_ERR_LAYOUT;
    int epi = DEERS_EPI_NONE;
    const float* r = nullptr;
    long long ldr = 0;
    float* aux = nullptr;
    if (epilogue) {
        epi = epilogue->kind;
        if (epi < DEERS_EPI_NONE || epi > DEERS_EPI_MUL_AUX2) return DEERS_ERR_SHAPE;
        if (epi == DEERS_EPI_ADD) {
            if (!epilogue->residual) return DEERS_ERR_NULL;
            if (epilogue->ld_residual < N || ((uintptr_t)epilogue->residual & 3u)) return DEERS_ERR_LAYOUT;
            r = epilogue->residual; ldr = epilogue->ld_residual;
        } else if (epi != DEERS_EPI_NONE) {
            if (!epilogue->aux) return DEERS_ERR_NULL;
            if ((uintptr_t)epilogue->aux & 3u) return DEERS_ERR_LAYOUT;
            aux = epilogue->aux;
        }
    }
    (void)workspace; (void)workspace_bytes;
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    return launch_gemm_f32(ctx, M, N, K, a, lda, a_mn_major, b, ldb, b_mn_major, c, ldc, epi, r, ldr, aux);
}
