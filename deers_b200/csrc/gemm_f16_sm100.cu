// f16 GEMM with f32 accumulation on tcgen05 / TMEM / TMA, for the projections around the attention op.
//
// The reference runs `Linear::forward` (src/nn.rs:184-190: y = x.matmul(weight), weight stored
// [in_features, out_features]) and its backward (src/ops.rs:1089-1101: dx = dy @ W^T, dW = x^T @ dy)
// through cublasGemmStridedBatchedEx (src/storage/cuda.rs:1147-1177).  One kernel covers the three
// products through the two operand layouts of the tensor core:
//     C[M,N] = A * B,  A stored [M,K] (K contiguous: "K-major") or [K,M] (M contiguous: "MN-major"),
//                      B stored [N,K] (K-major)                or [K,N] (MN-major)
//     forward  y  = x   * W      : A = x  [M,K]  K-major,  B = W  [K,N] MN-major
//     dgrad    dx = dy  * W^T    : A = dy [M,N]  K-major,  B = W  [K,N] read as [N'=K, K'=N]: K-major
//     wgrad    dW = x^T * dy     : A = x  [m,K]  read as [K'=m, M'=K]: MN-major,  B = dy [m,N] MN-major
// Persistent: one CTA per SM walks 128 x 256 (or 192) output tiles (consecutive CTAs share a B column block, which
// L2 then serves), or a pair of CTAs on two SMs walks tiles of 256 x 256.  Warp 0 streams 64-deep K blocks of A (16 KB) and B (32 KB) through a
// 4-stage ring (TMA, 128-byte swizzle, out-of-range rows / columns read as zero), warp 1 issues four 128x256x16 tcgen05.mma per K block into one
// of two TMEM accumulators, warps 2-9 move a finished accumulator to registers 64 columns at a time, convert to f16 and store rows transposed
// within 8-lane groups (contiguous 128-byte segments), then release the accumulator.  Few tiles and a long K (weight gradients) leave most SMs
// idle: there a cluster of CTAs shares a tile and its K (768 x 768 x 8192: 18 tiles, 51 us on 18 SMs; 22 us as 24 narrower tiles of five parts.
// 768 x 2304 x 8192: 52 -> 31 us).  192 columns where 256-wide tiles just miss a wave (8192 x 768 x 2304: 192 tiles on 148 SMs, 29 us; 256 tiles
// 24 us).  Bound: tensor pipe for large products (4096^3: 1.38 PFLOP/s by pairs, 1.25 without), L2 reads of both operands for the split ones.
#include "sm100_ptx.cuh"
#include "tma_host.cuh"

#include <cooperative_groups.h>
#include <type_traits>

namespace {
using namespace sm100;

constexpr int GM = 128, GK = 64;                // output tile rows and K block
constexpr uint32_t G_A_BYTES = GM * GK * 2;     // 16 KB per stage
constexpr int G_EPI_WG = 2;                     // epilogue warpgroups, each with half of a tile's columns
constexpr int G_THREADS = 64 + 128 * G_EPI_WG;
constexpr int G_MAX_PARTS = 6;                  // CTAs of a cluster along K (of eight only 15 clusters fit the device)
// Tiles of GN columns by one CTA, or of 256 rows by a pair of CTAs, each with half of the rows and half of B's columns.
template <int GN, bool PAIR>
struct GemmShape {
    static constexpr int BN = PAIR ? GN / 2 : GN;                            // columns of B in a CTA's stage
    static constexpr uint32_t B_BYTES = BN * GK * 2u;
    static constexpr int STAGES = PAIR ? 6 : 4;
    static constexpr uint32_t RING = STAGES * (G_A_BYTES + B_BYTES);         // a split-K CTA parks its f32 partial tile (rows of GN + 4) over it
    static constexpr uint32_t SMEM = RING + 256;
    static_assert((uint32_t)GM * (GN + 4) * 4 <= RING && SMEM <= 232448, "partial tile fits over the ring, and the ring in shared memory");
    // barriers
    static constexpr int FULL = 0, EMPTY = STAGES, ACC_FULL = 2 * STAGES, ACC_EMPTY = ACC_FULL + 2, COUNT = ACC_EMPTY + 2;
    static_assert(COUNT * 8 + 16 <= 256, "barriers");
};
// Shared-memory layouts of a stage (what the TMA boxes below write, 128-byte swizzle):
//   K-major operand of R rows (R = 128 for A, 256 for B): one block of R rows x 64 K-columns (R * 128 bytes)
//   MN-major operand of C columns (C = 128 / 256): C / 64 blocks of 64 K-rows x 64 columns (8 KB each)
constexpr uint32_t G_MN_BLOCK = GK * 128;       // 8 KB

struct GemmParams {
    __half* c;
    long long ldc;
    int M, N, K;
    int kb_chunk;               // K blocks per part
    unsigned int* err;
};

// The part of the start that needs nothing of global memory (see started()).
template <int GN, bool PAIR>
__device__ __forceinline__ void gemm_f16_prologue(const void* tmap_a, const void* tmap_b) {
    using S = GemmShape<GN, PAIR>;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::RING);
    uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(bars + S::COUNT);
    if (threadIdx.x == 0) {
        tmem_base_s[1] = 0;                                     // the abort flag
        tmem_base_s[3] = 0;                                     // epilogue threads whose rows are parked
        for (int s = 0; s < S::STAGES; ++s) { mbar_init(&bars[S::FULL + s], 1); mbar_init(&bars[S::EMPTY + s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&bars[S::ACC_FULL + s], 1); mbar_init(&bars[S::ACC_EMPTY + s], (PAIR ? 8 : 4) * G_EPI_WG); }
        fence_barrier_init();
        tma_prefetch_desc(tmap_a); tma_prefetch_desc(tmap_b);
    }
    if (uniform((int)threadIdx.x / 32) == 1) {
        if (PAIR) { tmem_alloc_pair(tmem_base_s, 512); tmem_relinquish_pair(); }
        else { tmem_alloc(tmem_base_s, 512); tmem_relinquish(); }
    }
}

// SPLIT: one tile per cluster, whose CTAs take a share of K each; the partial tiles meet in distributed shared memory and are
// added in the order of their K ranges (reproducible, no workspace).
// PAIR: a cluster of two, the first of which issues the products of both; either brings its rows of A and half of B's columns and
// finishes its own 128 rows.  A CTA alone is held up by its shared memory: a stage's operands arrive there and are read from it at
// 187 bytes a cycle against the 128 it has; of a pair's, B is read from both memories, 128.
template <int A_MN, int B_MN, int GN, bool SPLIT, bool PAIR>
__global__ void __launch_bounds__(G_THREADS, 1)
gemm_f16_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const GemmParams p) {
    gemm_f16_prologue<GN, PAIR>(&tmap_a, &tmap_b);
    chain_wait();
    namespace cg = cooperative_groups;
    using S = GemmShape<GN, PAIR>;
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int G_STAGES = S::STAGES, TM = PAIR ? 2 * GM : GM;
    constexpr uint32_t G_B_BYTES = S::B_BYTES;
    uint8_t* sA = smem;
    uint8_t* sB = smem + G_STAGES * G_A_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::RING);
    uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(bars + S::COUNT);
    volatile uint32_t* abort_s = tmem_base_s + 1;
    uint32_t* skip_s = tmem_base_s + 2;

    const int warp = uniform((int)threadIdx.x / 32), lane = threadIdx.x % 32;
    const int tiles_m = (p.M + TM - 1) / TM, tiles_n = (p.N + GN - 1) / GN;
    const int n_tiles = tiles_m * tiles_n;
    static_assert(!(SPLIT && PAIR), "pairs do not share K");
    const int kb_all = (p.K + GK - 1) / GK;
    const int rank = SPLIT || PAIR ? (int)cg::this_cluster().block_rank() : 0, half = PAIR ? rank & 1 : 0;
    const int group = SPLIT ? (int)cg::this_cluster().num_blocks() : PAIR ? 2 : 1;             // CTAs per tile
    const int parts = SPLIT ? group : 1, part = SPLIT ? rank : 0;
    const int kb0 = part * p.kb_chunk, kb1 = SPLIT ? min(kb_all, kb0 + p.kb_chunk) : kb_all;   // this CTA's K blocks: never none
    const int t0 = (int)blockIdx.x / group, t_step = SPLIT ? n_tiles : (int)gridDim.x / group;

    // (a CTA of a cluster stays: its peers read its shared memory)
    bool skip = !started(smem, skip_s, p.err, DEERS_KERR_GEMM | 0x20);
    if constexpr (PAIR) {
        cg::this_cluster().sync();                          // both have their barriers, and both go on or neither
        skip = skip || *cg::this_cluster().map_shared_rank(skip_s, rank ^ 1) != 0;
    }
    if (!SPLIT && !PAIR && skip) {
        if (warp == 1) tmem_dealloc(*tmem_base_s, 512);
        return;
    }
    const uint32_t tmem = (uint32_t)uniform((int)*tmem_base_s);
    WaitState ws{abort_s, p.err};

    bool done = !skip;                                      // (epilogue warps) the tile has arrived
    if (skip) {
    } else if (warp == 0) {
        // ------------------------------ TMA producer ------------------------------
        if (lane == 0) {
            uint32_t g = 0;                                     // K blocks loaded so far (ring position)
            bool ok = true;
            for (int t = t0; ok && t < n_tiles; t += t_step) {
                const int tm = t % tiles_m, tn = t / tiles_m;
                for (int kb = kb0; kb < kb1; ++kb, ++g) {
                    const uint32_t s = g % G_STAGES;
                    if (!mbar_wait(ws, &bars[S::EMPTY + s], ((g / G_STAGES) & 1u) ^ 1u, DEERS_KERR_GEMM | 1)) { ok = false; break; }
                    // (a pair's stage is announced at its first CTA, for the bytes of both)
                    constexpr uint32_t BYTES = G_A_BYTES + G_B_BYTES;
                    if (half == 0) mbar_arrive_expect_tx(&bars[S::FULL + s], PAIR ? 2 * BYTES : BYTES);
                    uint8_t* a_dst = sA + s * G_A_BYTES;
                    uint8_t* b_dst = sB + s * G_B_BYTES;
                    const int m0 = tm * TM + half * GM, n0 = tn * GN + half * S::BN;
                    const auto load = [&](uint8_t* dst, const CUtensorMap* map, int x, int y) {
                        if constexpr (PAIR) tma_load_4d_pair(dst, map, cluster_addr(&bars[S::FULL + s], 0), x, y, 0, 0);
                        else tma_load_4d(dst, map, &bars[S::FULL + s], x, y, 0, 0);
                    };
                    // K-major: box {64 of K, rows}; MN-major: boxes {64 of M / N, 64 rows of K}
                    if (A_MN) {
#pragma unroll
                        for (int blk = 0; blk < GM / 64; ++blk) load(a_dst + blk * G_MN_BLOCK, &tmap_a, m0 + blk * 64, kb * GK);
                    } else {
                        load(a_dst, &tmap_a, kb * GK, m0);
                    }
                    if (B_MN) {
#pragma unroll
                        for (int blk = 0; blk < S::BN / 64; ++blk) load(b_dst + blk * G_MN_BLOCK, &tmap_b, n0 + blk * 64, kb * GK);
                    } else {
                        load(b_dst, &tmap_b, kb * GK, n0);
                    }
                }
            }
        }
        __syncwarp();
        chain_next();                                           // all loads are under way: the end is near
    } else if (warp == 1) {
        // ------------------------------ MMA issuer ------------------------------
        // The whole warp runs this; one elected lane issues (see elect_one).
        if (half == 0) {
            constexpr uint32_t IDESC = idesc_f16(TM, GN, A_MN, B_MN);
            const auto commit = [&](uint64_t* bar) {
                if constexpr (PAIR) umma_commit_pair(bar, 3u);
                else umma_commit(bar);
            };
            constexpr uint64_t A_STEP = G_A_BYTES >> 4, B_STEP = G_B_BYTES >> 4;
            const uint32_t sa0 = (uint32_t)uniform((int)smem_u32(sA)), sb0 = (uint32_t)uniform((int)smem_u32(sB));
            const uint64_t a0 = A_MN ? desc_mnmajor(sa0, 0, G_MN_BLOCK) : desc_kmajor(sa0, 0, 0);
            const uint64_t b0 = B_MN ? desc_mnmajor(sb0, 0, G_MN_BLOCK) : desc_kmajor(sb0, 0, 0);
            uint32_t g = 0;
            int n = 0;
            bool ok = true;
            for (int t = t0; ok && t < n_tiles; t += t_step, ++n) {
                const uint32_t buf = (uint32_t)n & 1u;
                if (!mbar_wait_warp(ws, &bars[S::ACC_EMPTY + buf], (((uint32_t)n >> 1) & 1u) ^ 1u, DEERS_KERR_GEMM | 2)) break;
                tc_fence_after_sync();
                for (int kb = kb0; kb < kb1; ++kb, ++g) {
                    const uint32_t s = g % G_STAGES;
                    if (!mbar_wait_warp(ws, &bars[S::FULL + s], (g / G_STAGES) & 1u, DEERS_KERR_GEMM | 3)) { ok = false; break; }
                    tc_fence_after_sync();
                    const uint64_t a = a0 + (uint64_t)s * A_STEP, b = b0 + (uint64_t)s * B_STEP;
                    if (elect_one()) {
#pragma unroll
                        for (int ks = 0; ks < GK / 16; ++ks) {             // ks < 4: a K-major step stays inside its block
                            const uint64_t ad = a + (A_MN ? mnmajor_step(ks) : kmajor_step(ks, 0));
                            const uint64_t bd = b + (B_MN ? mnmajor_step(ks) : kmajor_step(ks, 0));
                            if constexpr (PAIR) umma_ss_pair(tmem + buf * 256u, ad, bd, IDESC, (kb > kb0 || ks > 0));
                            else umma_ss(tmem + buf * 256u, ad, bd, IDESC, (kb > kb0 || ks > 0));
                        }
                        commit(&bars[S::EMPTY + s]);
                        if (kb == kb1 - 1) commit(&bars[S::ACC_FULL + buf]);
                    }
                    __syncwarp();
                }
            }
        }
    } else {
        // ------------------------------ epilogue ------------------------------
        const int lane_base = (warp & 3) * 32;
        const uint32_t t_lane = (uint32_t)lane_base << 16;
        constexpr int SHARE = GN / G_EPI_WG, CH = SHARE % 64 ? 32 : 64;      // a warpgroup's columns, and those it takes at a time
        const int share0 = ((warp - 2) >> 2) * SHARE;
        int n = 0;
        for (int t = t0; t < n_tiles; t += t_step, ++n) {
            const int tm = t % tiles_m, tn = t / tiles_m;
            const uint32_t buf = (uint32_t)n & 1u;
            if (!__all_sync(0xffffffffu, mbar_wait(ws, &bars[S::ACC_FULL + buf], ((uint32_t)n >> 1) & 1u, DEERS_KERR_GEMM | 4))) { done = false; break; }
            tc_fence_after_sync();
            if constexpr (SPLIT) {
                // every product of this CTA has finished: the ring is free for its partial tile
                float* row = reinterpret_cast<float*>(smem) + (lane_base + lane) * (GN + 4);
#pragma unroll 1
                for (int c0 = share0; c0 < share0 + SHARE; c0 += 32) {
                    uint32_t r[32];
                    tmem_ld_x32(tmem + t_lane + c0, r);
                    tmem_wait_ld();
#pragma unroll
                    for (int c = 0; c < 32; c += 4) *reinterpret_cast<uint4*>(row + c0 + c) = make_uint4(r[c], r[c + 1], r[c + 2], r[c + 3]);
                }
                break;
            }
            constexpr int NP = CH / 8;                          // 16-byte pieces of a row
            const int row0 = tm * TM + half * GM + lane_base + (lane & ~(NP - 1));
#pragma unroll 1
            for (int c0 = share0; c0 < share0 + SHARE; c0 += CH) {
                uint32_t r[CH];
                uint4 pc[NP];
#pragma unroll
                for (int c = 0; c < CH; c += 32) tmem_ld_x32(tmem + buf * 256u + t_lane + c0 + c, *reinterpret_cast<uint32_t(*)[32]>(&r[c]));
                tmem_wait_ld();
                if (c0 == share0 + SHARE - CH) {                // this warp's share of the accumulator is in registers
                    tc_fence_before_sync();
                    if constexpr (PAIR) mbar_arrive_cluster_warp(cluster_addr(&bars[S::ACC_EMPTY + buf], 0));
                    else mbar_arrive_warp(&bars[S::ACC_EMPTY + buf]);
                }
#pragma unroll
                for (int q8 = 0; q8 < NP; ++q8) pc[q8] = pack8_f16(r + q8 * 8, 1.0f);
                transpose_pieces<NP>(pc, (uint32_t)lane);
                const int col = tn * GN + c0 + (lane & (NP - 1)) * 8;
#pragma unroll
                for (int c = 0; c < NP; ++c) {
                    const int row = row0 + c;
                    if (row < p.M && col < p.N) *reinterpret_cast<uint4*>(p.c + (long long)row * p.ldc + col) = pc[c];
                }
            }
        }
    }
    if constexpr (SPLIT) {
        cg::cluster_group cluster = cg::this_cluster();
        uint32_t* have_s = skip_s + 1;                          // (zeroed at the start) epilogue threads whose rows are parked
        if (warp >= 2 && done) atomicAdd(have_s, 1u);
        __syncwarp();
        cluster.sync();
        bool all = true;
        for (int z = 0; z < parts; ++z) all = all && *cluster.map_shared_rank(have_s, z) == 128u * G_EPI_WG;
        const int tm = t0 % tiles_m, tn = t0 / tiles_m;
        const int share = (GM + parts - 1) / parts, r_end = min(GM, (part + 1) * share);
        if (all) {
            float* mine = reinterpret_cast<float*>(smem);
            const auto add = [&](auto parts_c) {
                constexpr int P = decltype(parts_c)::value, U = P <= 2 ? 4 : P <= 4 ? 2 : 1;    // U pieces of 8 columns in flight
                const float* from[P];
#pragma unroll
                for (int z = 0; z < P; ++z) from[z] = cluster.map_shared_rank(mine, z);
                const int end = r_end * (GN / 8);
#pragma unroll 1
                for (int i0 = part * share * (GN / 8) + (int)threadIdx.x; i0 < end; i0 += U * G_THREADS) {
                    float4 x[U][P][2];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int idx = min(i0 + u * G_THREADS, end - 1), at = idx / (GN / 8) * (GN + 4) + idx % (GN / 8) * 8;
#pragma unroll
                        for (int z = 0; z < P; ++z) {
                            x[u][z][0] = *reinterpret_cast<const float4*>(from[z] + at);
                            x[u][z][1] = *reinterpret_cast<const float4*>(from[z] + at + 4);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int idx = i0 + u * G_THREADS;
                        const int row = tm * GM + idx / (GN / 8), col = tn * GN + idx % (GN / 8) * 8;
                        if (idx >= end || row >= p.M || col >= p.N) continue;
                        float4 lo = x[u][0][0], hi = x[u][0][1];
#pragma unroll
                        for (int z = 1; z < P; ++z) {
                            lo.x += x[u][z][0].x; lo.y += x[u][z][0].y; lo.z += x[u][z][0].z; lo.w += x[u][z][0].w;
                            hi.x += x[u][z][1].x; hi.y += x[u][z][1].y; hi.z += x[u][z][1].z; hi.w += x[u][z][1].w;
                        }
                        const uint32_t o[8] = {__float_as_uint(lo.x), __float_as_uint(lo.y), __float_as_uint(lo.z), __float_as_uint(lo.w),
                                               __float_as_uint(hi.x), __float_as_uint(hi.y), __float_as_uint(hi.z), __float_as_uint(hi.w)};
                        *reinterpret_cast<uint4*>(p.c + (long long)row * p.ldc + col) = pack8_f16(o, 1.0f);
                    }
                }
            };
            switch (parts) {
                case 2: add(std::integral_constant<int, 2>()); break;
                case 3: add(std::integral_constant<int, 3>()); break;
                case 4: add(std::integral_constant<int, 4>()); break;
                case 5: add(std::integral_constant<int, 5>()); break;
                default: add(std::integral_constant<int, 6>()); break;
            }
        }
    }
    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if constexpr (SPLIT || PAIR) cg::this_cluster().sync();     // nobody leaves while a peer still reads its memory or arrives at its barriers
    if (warp == 1) {
        if constexpr (PAIR) tmem_dealloc_pair(tmem, 512);
        else tmem_dealloc(tmem, 512);
    }
}

// 2-D tensor map over a row-major f16 matrix [rows][inner] with leading dimension ld (elements).
int make_tmap_matrix(deers_ctx* ctx, CUtensorMap* out, const void* base, long long rows, long long inner, long long ld,
                     int box_rows) {
    const int64_t strides[4] = {rows * ld, rows * ld, ld, 1};
    return make_tmap_bhtd_f16(ctx, out, base, 1, 1, (int)rows, (int)inner, strides, box_rows);
}

struct GemmPlan { int gn, parts, kb_chunk; bool pair; };

// Clusters of n CTAs (one per SM) the device holds at a time.
int cluster_room(deers_ctx* ctx) {
    if (ctx->cluster_room_f16[1] > 0) return DEERS_OK;
    constexpr int MOST = G_MAX_PARTS;
    static std::atomic<int> known[64][MOST + 1];                           // asked once per device: a tenth of a millisecond each
    std::atomic<int>* dev = known[ctx->device & 63];
    if (dev[1].load(std::memory_order_acquire) > 0) {
        for (int n = 1; n <= MOST; ++n) ctx->cluster_room_f16[n] = dev[n].load(std::memory_order_relaxed);
        return DEERS_OK;
    }
    using S = GemmShape<256, false>;
    const auto kernel = gemm_f16_kernel<0, 1, 256, true, false>;
    DEERS_SMEM_ONCE(ctx, (gemm_f16_kernel<0, 1, 256, true, false>), S::SMEM);
    for (int n = 2; n <= MOST; ++n) {
        cudaLaunchConfig_t lc{};
        lc.gridDim = dim3(n);
        lc.blockDim = dim3(G_THREADS);
        lc.dynamicSmemBytes = S::SMEM;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)n; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        lc.attrs = at; lc.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &lc) != cudaSuccess) { cudaGetLastError(); clusters = 0; }
        ctx->cluster_room_f16[n] = clusters;
        dev[n].store(clusters, std::memory_order_relaxed);
    }
    ctx->cluster_room_f16[1] = ctx->sm_count;
    dev[1].store(ctx->sm_count, std::memory_order_release);
    return DEERS_OK;
}

// Tile width, K split, and pair or single CTA, with the least estimated time, in microseconds as measured: a K block takes 0.40 with
// 256 columns and 0.335 with 192 (A passes through shared memory as often), 0.35 with a pair's 256 x 256, whose launch costs 1.5 more; the
// tiles an SM has to take follow one another, and a meeting of the parts costs 4.0 + 0.9 for each (launch of the cluster, partial tiles
// through shared memory, two cluster barriers).  Pairs and the best of the others: 8192 x 2304 x 768 24.4 and 26.2 us, 4096^3 100 and 110,
// 16384 x 6144 x 2048 298 and 340, 2048 x 6144 x 16384 335 and 462; 8192 x 768 x 2304 28.7 and 24.0, 1024 x 1536 x 512 8.1 and 6.2.  Pairs on
// 192 columns and pairs that share K were never the quickest (768 x 2304 x 8192 31.0 and 29.1, 8192 x 768 x 768 13.5 and 12.4).
GemmPlan plan_gemm_f16(deers_ctx* ctx, int M, int N, int K) {
    const int kb = (K + GK - 1) / GK;
    GemmPlan best{256, 1, kb, false};
    double best_cost = -1.0;
    for (int gn = 256; gn >= 192; gn -= 64) {
        const long long tiles = (long long)((M + GM - 1) / GM) * ((N + gn - 1) / gn);
        for (int parts = 1; parts <= G_MAX_PARTS; ++parts) {
            const int chunk = (kb + parts - 1) / parts;
            const int room = ctx->cluster_room_f16[parts];
            if (room < 1 || (parts > 1 && (chunk < 4 || chunk * (parts - 1) >= kb))) continue;      // no empty part
            const double waves = (double)((tiles + room - 1) / room);
            const double cost = waves * (chunk * (gn == 256 ? 0.40 : 0.335) + (parts > 1 ? 4.0 + 0.9 * parts : 0.4));
            if (best_cost < 0.0 || cost < best_cost) { best_cost = cost; best = GemmPlan{gn, parts, chunk, false}; }
        }
    }
    const int pairs = ctx->cluster_room_f16[2];
    if (pairs > 0) {
        const long long tiles = (long long)((M + 2 * GM - 1) / (2 * GM)) * ((N + 255) / 256);
        const double cost = (double)((tiles + pairs - 1) / pairs) * (kb * 0.35 + 0.4) + 1.5;
        if (cost < best_cost) best = GemmPlan{256, 1, kb, true};
    }
    return best;
}

template <int A_MN, int B_MN, int GN, bool PAIR>
int gemm_launch(deers_ctx* ctx, const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, int parts) {
    using S = GemmShape<GN, PAIR>;
    constexpr int TM = PAIR ? 2 * GM : GM, CTAS = PAIR ? 2 : 1;
    const long long tiles = (long long)((p.M + TM - 1) / TM) * ((p.N + GN - 1) / GN);
    {
        KernelTimerScope ts(ctx, DEERS_K_GEMM);
        if (PAIR || parts == 1) {
            DEERS_SMEM_ONCE(ctx, (gemm_f16_kernel<A_MN, B_MN, GN, false, PAIR>), S::SMEM);
            const int room = ctx->cluster_room_f16[CTAS];
            const unsigned grid = (unsigned)(tiles < room ? tiles : room);
            const ChainScope chain(ctx, tiles * p.kb_chunk / grid);
            DEERS_CUDA_TRY(ctx, launch_chained(ctx, gemm_f16_kernel<A_MN, B_MN, GN, false, PAIR>, grid * CTAS, G_THREADS, S::SMEM, CTAS, ta, tb, p));
        } else if constexpr (!PAIR) {
            const auto kernel = gemm_f16_kernel<A_MN, B_MN, GN, true, false>;
            DEERS_SMEM_ONCE(ctx, (gemm_f16_kernel<A_MN, B_MN, GN, true, false>), S::SMEM);
            DEERS_CUDA_TRY(ctx, launch_chained(ctx, kernel, (unsigned)(tiles * parts), G_THREADS, S::SMEM, parts, ta, tb, p));
        }
    }
    ctx->launches += 1;
    DEERS_CUDA_TRY(ctx, cudaGetLastError());
    return DEERS_OK;
}

template <int GN, bool PAIR>
int gemm_orders(deers_ctx* ctx, const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, int parts, int a_mn, int b_mn) {
    if (a_mn) return b_mn ? gemm_launch<1, 1, GN, PAIR>(ctx, ta, tb, p, parts) : gemm_launch<1, 0, GN, PAIR>(ctx, ta, tb, p, parts);
    return b_mn ? gemm_launch<0, 1, GN, PAIR>(ctx, ta, tb, p, parts) : gemm_launch<0, 0, GN, PAIR>(ctx, ta, tb, p, parts);
}

}  // namespace

// How many pairs of CTAs (one CTA per SM) the device holds at a time.
int gemm_f16_pairs(deers_ctx* ctx, int* pairs) {
    const int rc = cluster_room(ctx);
    *pairs = rc ? 0 : ctx->cluster_room_f16[2];
    return rc;
}

int route_gemm_f16(deers_ctx* ctx, int M, int N, int K, deers_product_route* r) {
    const int rc = cluster_room(ctx);
    if (rc) return rc;
    const GemmPlan p = plan_gemm_f16(ctx, M, N, K);
    r->tile_m = p.pair ? 2 * GM : GM; r->tile_n = p.gn; r->parts = p.parts; r->tensor_core = 1; r->pair = p.pair;
    return DEERS_OK;
}

extern "C" int deers_b200_gemm_f16(deers_ctx* ctx, int32_t M, int32_t N, int32_t K, const void* a, int64_t lda, int32_t a_mn_major,
                                   const void* b, int64_t ldb, int32_t b_mn_major, void* c, int64_t ldc) {
    if (!ctx || !a || !b || !c) return DEERS_ERR_NULL;
    if (M < 1 || N < 1 || K < 1) return DEERS_ERR_SHAPE;
    // 16-byte rows for TMA and for the epilogue's 16-byte stores
    if ((N % 8) || (lda % 8) || (ldb % 8) || (ldc % 8) || lda < (a_mn_major ? M : K) || ldb < (b_mn_major ? N : K) || ldc < N)
        return DEERS_ERR_LAYOUT;
    if (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 15u) return DEERS_ERR_LAYOUT;
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    CUtensorMap ta, tb;
    int rc = cluster_room(ctx);
    if (rc) return rc;
    const GemmPlan plan = plan_gemm_f16(ctx, M, N, K);
    // K-major A: [M rows][K inner], box {64, 128}; MN-major A: [K rows][M inner], box {64, 64}.  Same for B with
    // N (K-major box {64, tile columns}).
    if ((rc = a_mn_major ? make_tmap_matrix(ctx, &ta, a, K, M, lda, GK) : make_tmap_matrix(ctx, &ta, a, M, K, lda, GM))) return rc;
    const int b_rows = plan.pair ? plan.gn / 2 : plan.gn;
    if ((rc = b_mn_major ? make_tmap_matrix(ctx, &tb, b, K, N, ldb, GK) : make_tmap_matrix(ctx, &tb, b, N, K, ldb, b_rows))) return rc;
    GemmParams p;
    p.c = (__half*)c; p.ldc = ldc; p.M = M; p.N = N; p.K = K; p.kb_chunk = plan.kb_chunk; p.err = ctx->dev_err;
    const auto orders = plan.pair ? gemm_orders<256, true> : plan.gn == 256 ? gemm_orders<256, false> : gemm_orders<192, false>;
    return orders(ctx, ta, tb, p, plan.parts, a_mn_major, b_mn_major);
}
