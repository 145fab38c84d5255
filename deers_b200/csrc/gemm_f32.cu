// f32 GEMM: the choice of tile and split, the launches and the C ABI (the kernels: gemm_f32_kernel.cuh).
#include "gemm_f32_tc.cuh"

namespace {

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
__global__ void __launch_bounds__(GT * KS, PM * PN < 16 ? 2 : 1) gemm_f32_group_kernel(const __grid_constant__ GemmGroup gg) {
    const int i = gg.pick(blockIdx.x);
    TileProduct<PM, PN, KS, true, true, false, false> tile;
    tile.setup(gg.args(i), gg.tile_m(i, blockIdx.x), gg.tile_n(i, blockIdx.x), blockIdx.z);
    chain_wait();
    tile.run(gg.args(i), gridDim.z, blockIdx.z);
}

__global__ void __launch_bounds__(TC_T, 1) gemm_f32_tc_group_kernel(const __grid_constant__ GemmGroup gg, unsigned int* err) {
    gemm_f32_tc_prologue();
    chain_wait();
    const int i = gg.pick(blockIdx.x);
    gemm_f32_tc_tile<true, true, false, false>(gg.args(i), gg.tile_m(i, blockIdx.x), gg.tile_n(i, blockIdx.x), blockIdx.z, gridDim.z, err);
}

// Tile variants: the cycles at 1.965 GHz that the choice reckons with, a block's walk over 64 k and what a launch costs around it.
// They were measured on loops of single products, one figure for every order.  The present ones walk (both in MN order / A in K and B in
// MN / both in K): 64 x 128 5810 / 6210 / 8180, 64 x 64 2920 / 3680 / 3990, 32 x 64 1850 / 1810 / 2200, 32 x 32 1690 / 1910 / 1740,
// 64 x 96 4620 / 4710 / 5250, 32 x 96 2430 / 2900 / 3280, and 3800 to 9200 around it (148 tiles, K 320 and 1600).  The 96-wide tiles are
// there for products whose 64-wide ones just miss one wave (1024 x 768: 192 tiles on 148 SMs, 128 of 64 x 96; 13.3 -> 11.7 us at K =
// 192, and 16.3 -> 13.7 for 1024 x 192 x 768 in clusters of four).
// 16 x 32 is for products that leave half of the SMs idle in 32 x 32: 100 x 576 x 192 3.7 -> 3.1 us, 231 x 192 x 192 3.7 -> 3.1, 64 x 64 x 400
// in clusters of four 3.9 -> 3.5, 100 x 192 x 768 in clusters of three, where 32 x 32 takes six, 5.5 -> 4.7 (five and more blocks meet for
// longer); two blocks on an SM gain nothing (231 x 576 x 192 3.8 and 4.7).  The last is the tensor core's: a block starts only where one has
// left, and so do clusters, so all of it counts per wave.  Measured in a graph: K = 64 4.6 us, 192 7.7, 384 12.0, 768 19.8, 1024 24.5; 1024 x
// 192 x 768 in clusters of four 9.5; three waves of K = 192 22.2.  Rows on no 16-byte boundary take a tenth to a fifth more (TC_LOOSE).  Short
// products stay with the FFMA tiles (1024 x 192 x 192 5.1 us, here 6.3; 231 x 576 x 192 3.8 and 6.1).
struct Variant { int bm, bn; double walk, around; };
constexpr int TC_CFG = 7;
constexpr double TC_LOOSE = 1.1;
constexpr Variant kVariants[8] = {{64, 128, 7420, 6000}, {64, 64, 3700, 4900}, {32, 64, 2360, 4000}, {32, 32, 1680, 3200},
                                  {64, 96, 5400, 5300},  {32, 96, 3200, 4300}, {16, 32, 970, 3800},  {TC_M, TC_N, 2640, 7300}};

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
// n products of one K; tc: what a tensor core's tile costs of its figure (0: not for these products); whole_heads: tiles must hold whole heads
// of that many columns (0: any).  cfg < 0: no variant does.
GemmPlan plan_gemm(int n, const int* M, const int* N, int K, double tc, const int* capacity, int whole_heads) {
    GemmPlan best{};
    best.cfg = -1;
    best.cost = 1e30;
    double best_cost = -1.0;
    const int steps = (K + BK - 1) / BK;
    for (int c = 0; c < 8; ++c) {
        const Variant& v = kVariants[c];
        if (whole_heads && v.bn % whole_heads) continue;
        if (c == TC_CFG && (tc == 0.0 || K == 0)) continue;
        long long tiles = 0;
        for (int i = 0; i < n; ++i) tiles += (long long)((M[i] + v.bm - 1) / v.bm) * ((N[i] + v.bn - 1) / v.bn);
        for (int parts = 1; parts <= MAX_PARTS; ++parts) {
            const int chunk = (steps + parts - 1) / parts;
            if (parts > 1 && ((chunk < 2 && c != TC_CFG) || (long long)chunk * (parts - 1) >= steps)) continue;      // no empty part
            if (capacity[parts] < 1) continue;
            const double waves = (double)((tiles + capacity[parts] - 1) / capacity[parts]);
            const double meet = parts > 1 ? 3300.0 + (c != TC_CFG && parts > 4 ? 600.0 * (parts - 4) : 0.0) : 0.0;
            const double cost = c == TC_CFG ? waves * (tc * (chunk * v.walk + v.around) + meet)
                                            : waves * chunk * v.walk + v.around + 1200.0 * (waves - 1.0) + meet;
            if (best_cost < 0.0 || cost < best_cost) {
                best_cost = cost;
                best.cost = cost; best.cfg = c; best.parts = parts; best.k_chunk = chunk * BK; best.waves = (int)waves;
            }
        }
    }
    if (K == 0) { best.parts = 1; best.k_chunk = BK; }
    return best;
}

// Lays the group's tiles out one product after another; their number.
int lay_out_group(GemmGroup& gg, const GemmPlan& p) {
    const Variant& v = kVariants[p.cfg];
    int tiles = 0;
    for (int i = 0; i < gg.n; ++i) {
        gg.first[i] = tiles;
        gg.tiles_n[i] = (gg.g[i].N + v.bn - 1) / v.bn;
        tiles += gg.tiles_n[i] * ((gg.g[i].M + v.bm - 1) / v.bm);
        gg.g[i].k_chunk = p.k_chunk;
    }
    return tiles;
}

template <int PM, int PN, int KS>
int launch_group(deers_ctx* ctx, const GemmPlan& p, const GemmGroup& gg, int tiles) {
    using S = GemmShape<PM, PN, KS, true, true, false>;
    const auto kernel = gemm_f32_group_kernel<PM, PN, KS>;
    DEERS_SMEM_ONCE(ctx, (gemm_f32_group_kernel<PM, PN, KS>), S::SMEM);
    DEERS_CUDA_TRY(ctx, launch_chained(ctx, kernel, dim3(tiles, 1, p.parts), S::THREADS, S::SMEM, dim3(1, 1, p.parts), gg));
    return DEERS_OK;
}

int launch_group_tc(deers_ctx* ctx, const GemmPlan& p, const GemmGroup& gg, int tiles) {
    DEERS_SMEM_ONCE(ctx, gemm_f32_tc_group_kernel, TC_SMEM);
    DEERS_CUDA_TRY(ctx, launch_chained(ctx, gemm_f32_tc_group_kernel, dim3(tiles, 1, p.parts), TC_T, TC_SMEM, dim3(1, 1, p.parts), gg, ctx->dev_err));
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
        const bool aligned = g.a_vec && g.b_vec;
        if (p.cfg == TC_CFG) rc = aligned ? launch_gemm_f32_tc(ctx, p.parts, g, a_mn, b_mn, fused) : launch_gemm_f32_tc_loose(ctx, p.parts, g, a_mn, b_mn);
        else rc = aligned ? launch_tiles<false>(ctx, p, g, a_mn, b_mn, fused) : launch_gemm_f32_loose(ctx, p, g, a_mn, b_mn, fused);
    }
    ctx->launches += 1;
    return rc;
}

GemmPlan plan_single(deers_ctx* ctx, int M, int N, int K, bool aligned) {
    return plan_gemm(1, &M, &N, K, aligned ? 1.0 : TC_LOOSE, ctx->cluster_capacity, 0);
}

// The plan of a product of normalised rows, and whether its tiles rotate heads of `heads` columns (0: there are none).
GemmPlan plan_norm(deers_ctx* ctx, int M, int N, int K, bool aligned, int heads, bool* rotated) {
    const bool rotates = heads && heads % 8 == 0;
    // Products that may rotate heads take the tensor core up to 384 columns: so far was the choice between rotating in a tile and beside it
    // measured on its tiles (further on it would gain too, C 512 626 -> 552 us, with that choice drawn anew).  What rotates nothing has no
    // such line: forwards with the up projection on FFMA and on the tensor core, C 512, 4 layers, 1024 tokens 825 and 626 us, 256 tokens
    // 292 and 271, 128 tokens 201 and 204; C 1024, 2 layers, 1024 tokens 1196 and 1010.
    const double tc = aligned && (!rotates || K <= 384) ? 1.0 : 0.0;
    const GemmPlan p = plan_gemm(1, &M, &N, K, tc, ctx->cluster_capacity, 0);
    *rotated = false;
    if (!rotates) return p;
    // A rotary launch of its own takes up to 4400 of these cycles (1.4 to 2 us): rotate here unless tiles that hold whole heads cost more
    // than that (heads of 48 columns leave 32 x 96 and 64 x 96 tiles: 231 x 576 x 192 takes 7.5 us in them, 3.6 in 32 x 32).
    // Several waves of clusters do not count: the estimate takes them to follow one another without a gap (forwards of 4 layers,
    // rotating in them and beside: C 512, 256 tokens 363 and 335 us, C 384, 640 tokens 533 and 501).
    const GemmPlan w = plan_gemm(1, &M, &N, K, tc, ctx->cluster_capacity, heads);
    *rotated = w.cfg >= 0 && w.cost < p.cost + 4400.0 && (w.cost == p.cost || w.parts == 1 || w.waves == 1);
    return *rotated ? w : p;
}
}  // namespace

int launch_gemm_f32(deers_ctx* ctx, int M, int N, int K, const float* a, long long lda, int a_mn, const float* b,
                    long long ldb, int b_mn, float* c, long long ldc, int epi, const float* r, long long ldr, float* aux) {
    if (M == 0 || N == 0) return DEERS_OK;
    // Row tiles lie along gridDim.y, which ends at 65535: taller products go in several launches.  (Tiles of
    // 16 rows are for products of few tiles: one so tall never takes them.)
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
    GemmArgs g = gemm_args(M, N, K, a, lda, b, ldb, c, ldc, epi, r, ldr, aux);
    const GemmPlan p = plan_single(ctx, M, N, K, g.a_vec && g.b_vec);
    return launch_planned(ctx, p, g, a_mn, b_mn, false);
}

// C = rmsnorm(A) * B with an optional rotation of the leading columns (see GemmNorm in common.cuh); M <= 65535 rows.
int launch_gemm_f32_norm(deers_ctx* ctx, int M, int N, int K, const float* a, const float* b, float* c, int epi, float* aux, const GemmNorm& f,
                         bool* rotated) {
    *rotated = false;
    if (M == 0 || N == 0) return DEERS_OK;
    const int rc = cluster_capacity(ctx);
    if (rc) return rc;
    GemmArgs g = gemm_args(M, N, K, a, K, b, N, c, N, epi, nullptr, 0, aux);
    const GemmPlan p = plan_norm(ctx, M, N, K, g.a_vec && g.b_vec, f.rope_cols ? f.rope_d : 0, rotated);
    if (*rotated) { g.cosv = f.cosv; g.sinv = f.sinv; g.rope_cols = f.rope_cols; g.rope_d = f.rope_d; g.rope_t = f.rope_t; }
    g.eps = f.eps; g.inv_n = (float)(1.0 / (double)K); g.inv = f.inv;
    return launch_planned(ctx, p, g, 0, 1, true);
}

namespace {
GemmPlan plan_group(deers_ctx* ctx, int n, const int* M, const int* N, int K, bool aligned) {
    return plan_gemm(n, M, N, K, aligned ? 1.0 : 0.0, ctx->cluster_capacity, 0);
}
// The same of products with dense operands (rows of M_i and N_i).
GemmPlan plan_group(deers_ctx* ctx, int n, const GemmTN* t, int K) {
    int M[GEMM_GROUP_MAX], N[GEMM_GROUP_MAX];
    bool aligned = true;
    for (int i = 0; i < n; ++i) {
        M[i] = t[i].M; N[i] = t[i].N;
        aligned = aligned && M[i] % 4 == 0 && N[i] % 4 == 0 && (((uintptr_t)t[i].a | (uintptr_t)t[i].b) & 15u) == 0;
    }
    return plan_group(ctx, n, M, N, K, aligned);
}
}  // namespace

// Whether the group of these products is one wave of blocks.  One of several waves keeps the SMs from what runs beside it until
// its last, where products on their own take turns with it (GPT training step of 6 layers, 1024 tokens: C 192, one wave, 980 us
// grouped and 998 apart; C 320 2235 and 2219; C 512 4472 and 4028).
bool gemm_f32_group_fits(deers_ctx* ctx, int n, const GemmTN* t, int K) {
    if (n < 1 || n > GEMM_GROUP_MAX || cluster_capacity(ctx)) return false;
    return plan_group(ctx, n, t, K).waves == 1;
}

// C_i = A_i^T B_i, A_i [K, M_i] and B_i [K, N_i] row-major, one K, in one launch.
int launch_gemm_f32_group(deers_ctx* ctx, int n, const GemmTN* t, int K) {
    if (n < 1 || n > GEMM_GROUP_MAX) return DEERS_ERR_SHAPE;
    const int rc = cluster_capacity(ctx);
    if (rc) return rc;
    GemmGroup gg{};
    gg.n = n;
    for (int i = 0; i < n; ++i)
        gg.g[i] = gemm_args(t[i].M, t[i].N, K, t[i].a, t[i].M, t[i].b, t[i].N, t[i].c, t[i].N, DEERS_EPI_NONE, nullptr, 0, nullptr);
    const GemmPlan p = plan_group(ctx, n, t, K);
    const int tiles = lay_out_group(gg, p);
    int res;
    {
        KernelTimerScope ts(ctx, DEERS_K_GEMM);
        if (p.cfg == 0) res = launch_group<8, 8, 2>(ctx, p, gg, tiles);
        else if (p.cfg == 1) res = launch_group<8, 4, 4>(ctx, p, gg, tiles);
        else if (p.cfg == 2) res = launch_group<4, 4, 4>(ctx, p, gg, tiles);
        else if (p.cfg == 3) res = launch_group<4, 2, 4>(ctx, p, gg, tiles);
        else if (p.cfg == 4) res = launch_group<8, 6, 4>(ctx, p, gg, tiles);
        else if (p.cfg == 5) res = launch_group<4, 6, 4>(ctx, p, gg, tiles);
        else if (p.cfg == 6) res = launch_group<2, 2, 4>(ctx, p, gg, tiles);
        else res = launch_group_tc(ctx, p, gg, tiles);
    }
    ctx->launches += 1;
    return res;
}

extern "C" int deers_b200_product_route(deers_ctx* ctx, int32_t which, int32_t n, const int32_t* M, const int32_t* N, int32_t K, int32_t a_mn_major,
                                        int32_t b_mn_major, int32_t aligned, int32_t heads, deers_product_route* route) {
    if (!ctx || !M || !N || !route) return DEERS_ERR_NULL;
    if (n < 1 || n > (which == DEERS_PRODUCT_F32 && a_mn_major && b_mn_major ? GEMM_GROUP_MAX : 1) || K < 1 || heads < 0) return DEERS_ERR_SHAPE;
    for (int i = 0; i < n; ++i)
        if (M[i] < 1 || N[i] < 1) return DEERS_ERR_SHAPE;
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    deers_product_route r{};
    int rc = DEERS_OK;
    if (which == DEERS_PRODUCT_F16) rc = route_gemm_f16(ctx, M[0], N[0], K, &r);
    else if (which == DEERS_PRODUCT_F16X3) rc = route_gemm_f16x3(ctx, M[0], N[0], K, a_mn_major != 0, b_mn_major != 0, aligned, &r);
    else if (which != DEERS_PRODUCT_F32 && which != DEERS_PRODUCT_F32_NORM) return DEERS_ERR_UNSUPPORTED;
    else if (!(rc = cluster_capacity(ctx))) {
        bool rotated = false;
        const GemmPlan p = which == DEERS_PRODUCT_F32_NORM ? plan_norm(ctx, M[0], N[0], K, aligned != 0, heads, &rotated)
                         : n > 1 ? plan_group(ctx, n, M, N, K, aligned != 0) : plan_single(ctx, M[0], N[0], K, aligned != 0);
        r.tile_m = kVariants[p.cfg].bm; r.tile_n = kVariants[p.cfg].bn; r.parts = p.parts; r.tensor_core = p.cfg == TC_CFG; r.rotated = rotated;
    }
    if (!rc) *route = r;
    return rc;
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
