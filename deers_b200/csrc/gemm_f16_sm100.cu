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
// L2 then serves).  Warp 0 streams 64-deep K blocks of A (16 KB) and B (32 KB) through a 4-stage ring (TMA,
// 128-byte swizzle, out-of-range rows / columns read as zero), warp 1 issues four 128x256x16 tcgen05.mma
// per K block into one of two TMEM accumulators, warps 2-5 move a finished accumulator to
// registers 64 columns at a time, convert to f16 and store rows transposed within 8-lane groups
// (contiguous 128-byte segments), then release the accumulator.
// Few tiles and a long K (weight gradients) leave most SMs idle: there a cluster of CTAs shares a tile and its K
// (768 x 768 x 8192: 18 tiles, 51 us on 18 SMs; 22 us as 24 narrower tiles of five parts.  768 x 2304 x 8192: 52 -> 31 us).
// 192 columns where 256-wide tiles just miss a wave (8192 x 768 x 2304: 192 tiles on 148 SMs, 29 us; 256 tiles 24 us).
// Bound: tensor pipe for large products (4096^3: 1.3 PFLOP/s), L2 reads of both operands for the split ones.
#include "sm100_ptx.cuh"
#include "tma_host.cuh"

#include <cooperative_groups.h>
#include <type_traits>

namespace {
using namespace sm100;

constexpr int GM = 128, GK = 64;                // output tile rows and K block
constexpr uint32_t G_A_BYTES = GM * GK * 2;     // 16 KB per stage
constexpr int G_STAGES = 4;
constexpr int G_THREADS = 192;
constexpr int G_MAX_PARTS = 6;                  // CTAs of a cluster along K (of eight only 15 clusters fit the device)
// Shared memory for tiles of gn columns: the ring; a split-K CTA then parks its f32 partial tile (rows of gn + 4) over it.
constexpr uint32_t g_ring(int gn) { return G_STAGES * (G_A_BYTES + (uint32_t)gn * GK * 2u); }
constexpr uint32_t g_smem(int gn) { return g_ring(gn) + 256; }
static_assert((uint32_t)GM * (256 + 4) * 4 <= g_ring(256) && (uint32_t)GM * (192 + 4) * 4 <= g_ring(192), "partial tile fits over the ring");
// Shared-memory layouts of a stage (what the TMA boxes below write, 128-byte swizzle):
//   K-major operand of R rows (R = 128 for A, 256 for B): one block of R rows x 64 K-columns (R * 128 bytes)
//   MN-major operand of C columns (C = 128 / 256): C / 64 blocks of 64 K-rows x 64 columns (8 KB each)
constexpr uint32_t G_MN_BLOCK = GK * 128;       // 8 KB

enum GBar { G_FULL = 0, G_EMPTY = 4, G_ACC_FULL = 8, G_ACC_EMPTY = 10, G_COUNT = 12 };

struct GemmParams {
    __half* c;
    long long ldc;
    int M, N, K;
    int kb_chunk;               // K blocks per part
    unsigned int* err;
};

// The part of the start that needs nothing of global memory (see started()).
template <int GN>
__device__ __forceinline__ void gemm_f16_prologue(const void* tmap_a, const void* tmap_b) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + G_STAGES * (G_A_BYTES + GN * GK * 2));
    uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(bars + G_COUNT);
    if (threadIdx.x == 0) {
        tmem_base_s[1] = 0;                                     // the abort flag
        tmem_base_s[3] = 0;                                     // epilogue threads whose rows are parked
        for (int s = 0; s < G_STAGES; ++s) { mbar_init(&bars[G_FULL + s], 1); mbar_init(&bars[G_EMPTY + s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&bars[G_ACC_FULL + s], 1); mbar_init(&bars[G_ACC_EMPTY + s], 128); }
        fence_barrier_init();
        tma_prefetch_desc(tmap_a); tma_prefetch_desc(tmap_b);
    }
    if (uniform((int)threadIdx.x / 32) == 1) {
        tmem_alloc(tmem_base_s, 512);
        tmem_relinquish();
    }
}

// SPLIT: one tile per cluster, whose CTAs take a share of K each; the partial tiles meet in distributed shared memory and are
// added in the order of their K ranges (reproducible, no workspace).
template <int A_MN, int B_MN, int GN, bool SPLIT>
__global__ void __launch_bounds__(G_THREADS, 1)
gemm_f16_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const GemmParams p) {
    gemm_f16_prologue<GN>(&tmap_a, &tmap_b);
    chain_wait();
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr uint32_t G_B_BYTES = GN * GK * 2;
    uint8_t* sA = smem;
    uint8_t* sB = smem + G_STAGES * G_A_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + G_STAGES * (G_A_BYTES + G_B_BYTES));
    uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(bars + G_COUNT);
    volatile uint32_t* abort_s = tmem_base_s + 1;
    uint32_t* skip_s = tmem_base_s + 2;

    const int warp = uniform((int)threadIdx.x / 32), lane = threadIdx.x % 32;
    const int tiles_m = (p.M + GM - 1) / GM, tiles_n = (p.N + GN - 1) / GN;
    const int n_tiles = tiles_m * tiles_n;
    const int kb_all = (p.K + GK - 1) / GK;
    const int parts = SPLIT ? (int)cooperative_groups::this_cluster().num_blocks() : 1;
    const int part = SPLIT ? (int)cooperative_groups::this_cluster().block_rank() : 0;
    const int kb0 = part * p.kb_chunk, kb1 = SPLIT ? min(kb_all, kb0 + p.kb_chunk) : kb_all;   // this CTA's K blocks: never none
    const int t0 = SPLIT ? (int)blockIdx.x / parts : (int)blockIdx.x, t_step = SPLIT ? n_tiles : (int)gridDim.x;

    // (a split-K CTA stays: its peers read its shared memory)
    const bool skip = !started(smem, skip_s, p.err, DEERS_KERR_GEMM | 0x20);
    if (!SPLIT && skip) {
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
                    if (!mbar_wait(ws, &bars[G_EMPTY + s], ((g / G_STAGES) & 1u) ^ 1u, DEERS_KERR_GEMM | 1)) { ok = false; break; }
                    mbar_arrive_expect_tx(&bars[G_FULL + s], G_A_BYTES + G_B_BYTES);
                    uint8_t* a_dst = sA + s * G_A_BYTES;
                    uint8_t* b_dst = sB + s * G_B_BYTES;
                    // K-major: box {64 of K, rows}; MN-major: boxes {64 of M / N, 64 rows of K}
                    if (A_MN) {
#pragma unroll
                        for (int blk = 0; blk < GM / 64; ++blk)
                            tma_load_4d(a_dst + blk * G_MN_BLOCK, &tmap_a, &bars[G_FULL + s], tm * GM + blk * 64, kb * GK, 0, 0);
                    } else {
                        tma_load_4d(a_dst, &tmap_a, &bars[G_FULL + s], kb * GK, tm * GM, 0, 0);
                    }
                    if (B_MN) {
#pragma unroll
                        for (int blk = 0; blk < GN / 64; ++blk)
                            tma_load_4d(b_dst + blk * G_MN_BLOCK, &tmap_b, &bars[G_FULL + s], tn * GN + blk * 64, kb * GK, 0, 0);
                    } else {
                        tma_load_4d(b_dst, &tmap_b, &bars[G_FULL + s], kb * GK, tn * GN, 0, 0);
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
            constexpr uint32_t IDESC = idesc_f16(GM, GN, A_MN, B_MN);
            constexpr uint64_t A_STEP = G_A_BYTES >> 4, B_STEP = G_B_BYTES >> 4;
            const uint32_t sa0 = (uint32_t)uniform((int)smem_u32(sA)), sb0 = (uint32_t)uniform((int)smem_u32(sB));
            const uint64_t a0 = A_MN ? desc_mnmajor(sa0, 0, G_MN_BLOCK) : desc_kmajor(sa0, 0, 0);
            const uint64_t b0 = B_MN ? desc_mnmajor(sb0, 0, G_MN_BLOCK) : desc_kmajor(sb0, 0, 0);
            uint32_t g = 0;
            int n = 0;
            bool ok = true;
            for (int t = t0; ok && t < n_tiles; t += t_step, ++n) {
                const uint32_t buf = (uint32_t)n & 1u;
                if (!mbar_wait_warp(ws, &bars[G_ACC_EMPTY + buf], (((uint32_t)n >> 1) & 1u) ^ 1u, DEERS_KERR_GEMM | 2)) break;
                for (int kb = kb0; kb < kb1; ++kb, ++g) {
                    const uint32_t s = g % G_STAGES;
                    if (!mbar_wait_warp(ws, &bars[G_FULL + s], (g / G_STAGES) & 1u, DEERS_KERR_GEMM | 3)) { ok = false; break; }
                    tc_fence_after_sync();
                    const uint64_t a = a0 + (uint64_t)s * A_STEP, b = b0 + (uint64_t)s * B_STEP;
                    if (elect_one()) {
#pragma unroll
                        for (int ks = 0; ks < GK / 16; ++ks)               // ks < 4: a K-major step stays inside its block
                            umma_ss(tmem + buf * 256u, a + (A_MN ? mnmajor_step(ks) : kmajor_step(ks, 0)),
                                    b + (B_MN ? mnmajor_step(ks) : kmajor_step(ks, 0)), IDESC, (kb > kb0 || ks > 0));
                        umma_commit(&bars[G_EMPTY + s]);
                        if (kb == kb1 - 1) umma_commit(&bars[G_ACC_FULL + buf]);
                    }
                    __syncwarp();
                }
            }
        }
    } else {
        // ------------------------------ epilogue ------------------------------
        const int lane_base = (warp & 3) * 32;
        const uint32_t t_lane = (uint32_t)lane_base << 16;
        int n = 0;
        for (int t = t0; t < n_tiles; t += t_step, ++n) {
            const int tm = t % tiles_m, tn = t / tiles_m;
            const uint32_t buf = (uint32_t)n & 1u;
            if (!__all_sync(0xffffffffu, mbar_wait(ws, &bars[G_ACC_FULL + buf], ((uint32_t)n >> 1) & 1u, DEERS_KERR_GEMM | 4))) { done = false; break; }
            tc_fence_after_sync();
            if constexpr (SPLIT) {
                // every product of this CTA has finished: the ring is free for its partial tile
                float* row = reinterpret_cast<float*>(smem) + (lane_base + lane) * (GN + 4);
#pragma unroll 1
                for (int c0 = 0; c0 < GN; c0 += 32) {
                    uint32_t r[32];
                    tmem_ld_x32(tmem + t_lane + c0, r);
                    tmem_wait_ld();
#pragma unroll
                    for (int c = 0; c < 32; c += 4) *reinterpret_cast<uint4*>(row + c0 + c) = make_uint4(r[c], r[c + 1], r[c + 2], r[c + 3]);
                }
                break;
            }
            const int row0 = tm * GM + lane_base + (lane & ~7);
#pragma unroll 1
            for (int part = 0; part < GN / 64; ++part) {        // 64 columns at a time
                uint32_t r[64];
                uint4 pc[8];
                tmem_ld_x32(tmem + buf * 256u + t_lane + part * 64, *reinterpret_cast<uint32_t(*)[32]>(&r[0]));
                tmem_ld_x32(tmem + buf * 256u + t_lane + part * 64 + 32, *reinterpret_cast<uint32_t(*)[32]>(&r[32]));
                tmem_wait_ld();
                if (part == GN / 64 - 1) {                      // accumulator is in registers: the next tile may use it
                    tc_fence_before_sync();
                    mbar_arrive(&bars[G_ACC_EMPTY + buf]);
                }
#pragma unroll
                for (int q8 = 0; q8 < 8; ++q8) pc[q8] = pack8_f16(r + q8 * 8, 1.0f);
                transpose_pieces<8>(pc, (uint32_t)lane);
                const int col = tn * GN + part * 64 + (lane & 7) * 8;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const int row = row0 + c;
                    if (row < p.M && col < p.N) *reinterpret_cast<uint4*>(p.c + (long long)row * p.ldc + col) = pc[c];
                }
            }
        }
    }
    if constexpr (SPLIT) {
        namespace cg = cooperative_groups;
        cg::cluster_group cluster = cg::this_cluster();
        uint32_t* have_s = skip_s + 1;                          // (zeroed at the start) epilogue threads whose rows are parked
        if (warp >= 2 && done) atomicAdd(have_s, 1u);
        __syncwarp();
        cluster.sync();
        bool all = true;
        for (int z = 0; z < parts; ++z) all = all && *cluster.map_shared_rank(have_s, z) == 128u;
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
        cluster.sync();                                         // nobody leaves while a peer still reads its partial tile
    }
    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

// 2-D tensor map over a row-major f16 matrix [rows][inner] with leading dimension ld (elements).
int make_tmap_matrix(deers_ctx* ctx, CUtensorMap* out, const void* base, long long rows, long long inner, long long ld,
                     int box_rows) {
    const int64_t strides[4] = {rows * ld, rows * ld, ld, 1};
    return make_tmap_bhtd_f16(ctx, out, base, 1, 1, (int)rows, (int)inner, strides, box_rows);
}

struct GemmPlan { int gn, parts, kb_chunk; };

// Clusters of n CTAs (one per SM) the device holds at a time.
int cluster_room(deers_ctx* ctx) {
    if (ctx->cluster_room_f16[1] > 0) return DEERS_OK;
    static std::atomic<int> known[64][G_MAX_PARTS + 1];                    // asked once per device: a tenth of a millisecond each
    std::atomic<int>* dev = known[ctx->device & 63];
    if (dev[1].load(std::memory_order_acquire) > 0) {
        for (int parts = 1; parts <= G_MAX_PARTS; ++parts) ctx->cluster_room_f16[parts] = dev[parts].load(std::memory_order_relaxed);
        return DEERS_OK;
    }
    const auto kernel = gemm_f16_kernel<0, 1, 256, true>;
    DEERS_SMEM_ONCE(ctx, (gemm_f16_kernel<0, 1, 256, true>), g_smem(256));
    for (int parts = 2; parts <= G_MAX_PARTS; ++parts) {
        cudaLaunchConfig_t lc{};
        lc.gridDim = dim3(parts);
        lc.blockDim = dim3(G_THREADS);
        lc.dynamicSmemBytes = g_smem(256);
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)parts; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        lc.attrs = at; lc.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kernel, &lc) != cudaSuccess) { cudaGetLastError(); n = 0; }
        ctx->cluster_room_f16[parts] = n;
        dev[parts].store(n, std::memory_order_relaxed);
    }
    ctx->cluster_room_f16[1] = ctx->sm_count;
    dev[1].store(ctx->sm_count, std::memory_order_release);
    return DEERS_OK;
}

// Tile width and K split with the least estimated time, in microseconds as measured: a K block takes 0.40 with 256 columns and
// 0.335 with 192 (A passes through shared memory as often), the tiles an SM has to take follow one another, and a meeting of
// the parts costs 4.0 + 0.9 for each (launch of the cluster, partial tiles through shared memory, two cluster barriers).
GemmPlan plan_gemm_f16(deers_ctx* ctx, int M, int N, int K) {
    GemmPlan best{256, 1, (K + GK - 1) / GK};
    double best_cost = -1.0;
    const int kb = (K + GK - 1) / GK;
    for (int gn = 256; gn >= 192; gn -= 64) {
        const long long tiles = (long long)((M + GM - 1) / GM) * ((N + gn - 1) / gn);
        for (int parts = 1; parts <= G_MAX_PARTS; ++parts) {
            const int chunk = (kb + parts - 1) / parts;
            const int room = ctx->cluster_room_f16[parts];
            if (room < 1 || (parts > 1 && (chunk < 4 || chunk * (parts - 1) >= kb))) continue;      // no empty part
            const double waves = (double)((tiles + room - 1) / room);
            const double cost = waves * (chunk * (gn == 256 ? 0.40 : 0.335) + (parts > 1 ? 4.0 + 0.9 * parts : 0.4));
            if (best_cost < 0.0 || cost < best_cost) { best_cost = cost; best = GemmPlan{gn, parts, chunk}; }
        }
    }
    return best;
}

template <int A_MN, int B_MN, int GN>
int gemm_launch(deers_ctx* ctx, const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, int parts) {
    const long long tiles = (long long)((p.M + GM - 1) / GM) * ((p.N + GN - 1) / GN);
    {
        KernelTimerScope ts(ctx, DEERS_K_GEMM);
        if (parts == 1) {
            DEERS_SMEM_ONCE(ctx, (gemm_f16_kernel<A_MN, B_MN, GN, false>), g_smem(GN));
            const unsigned grid = (unsigned)(tiles < ctx->sm_count ? tiles : ctx->sm_count);
            const ChainScope chain(ctx, tiles * p.kb_chunk / grid);
            DEERS_CUDA_TRY(ctx, launch_chained(ctx, gemm_f16_kernel<A_MN, B_MN, GN, false>, grid, G_THREADS, g_smem(GN), 1, ta, tb, p));
        } else {
            const auto kernel = gemm_f16_kernel<A_MN, B_MN, GN, true>;
            DEERS_SMEM_ONCE(ctx, (gemm_f16_kernel<A_MN, B_MN, GN, true>), g_smem(GN));
            DEERS_CUDA_TRY(ctx, launch_chained(ctx, kernel, (unsigned)(tiles * parts), G_THREADS, g_smem(GN), parts, ta, tb, p));
        }
    }
    ctx->launches += 1;
    DEERS_CUDA_TRY(ctx, cudaGetLastError());
    return DEERS_OK;
}

template <int GN>
int gemm_orders(deers_ctx* ctx, const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, int parts, int a_mn, int b_mn) {
    if (a_mn) return b_mn ? gemm_launch<1, 1, GN>(ctx, ta, tb, p, parts) : gemm_launch<1, 0, GN>(ctx, ta, tb, p, parts);
    return b_mn ? gemm_launch<0, 1, GN>(ctx, ta, tb, p, parts) : gemm_launch<0, 0, GN>(ctx, ta, tb, p, parts);
}

}  // namespace

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
    if ((rc = b_mn_major ? make_tmap_matrix(ctx, &tb, b, K, N, ldb, GK) : make_tmap_matrix(ctx, &tb, b, N, K, ldb, plan.gn))) return rc;
    GemmParams p;
    p.c = (__half*)c; p.ldc = ldc; p.M = M; p.N = N; p.K = K; p.kb_chunk = plan.kb_chunk; p.err = ctx->dev_err;
    return plan.gn == 256 ? gemm_orders<256>(ctx, ta, tb, p, plan.parts, a_mn_major, b_mn_major)
                          : gemm_orders<192>(ctx, ta, tb, p, plan.parts, a_mn_major, b_mn_major);
}
