// f16 causal attention forward for sm_100a.
//
// Persistent kernel: one CTA per SM walks a strided, heaviest-first list of work items, an item
// being 128 query rows of one (batch, head) slice together with the key/value tiles (128 rows
// each) at or left of its diagonal.  The whole list is treated as ONE stream of (item, KV tile)
// steps, so loads and the S product run ahead across item boundaries.
//   warp 0      TMA producer: Q per item (2 buffers), K tiles through a 2-stage ring
//   warp 3      the same for V, which waits for other products than K does
//   warp 2      issues the S = Q K^T products into three TMEM tiles in turn
//   warp 1      issues the O += P V products, with P read from TMEM and the accumulator resident in TMEM; a product starts
//               on the first half of P's columns.  The two streams are ordered by barriers only (S of step g+3 overwrites
//               P of step g once the product that read it has completed).
//   softmax     four warpgroups in two groups: group g takes the steps of parity g (score tile g), its two warpgroups
//               split the 128 key columns (64 each); thread r of a warpgroup owns query row r (= TMEM lane r).  The groups
//               run half a step apart, so that one's exponentials fill the special-function unit (1024 cycles a
//               step, as many as the tensor core needs) while the other loads scores, finds maxima and synchronises.  Per
//               step a thread reads its 64 scores, exchanges its partial row max with its twin, takes the row's reference
//               maximum from the group of the step before and publishes the new one, stores P (f16 pairs) back into
//               TMEM over the scores, and rescales its half of O only when the row max grew by more than 2^8.  At the
//               end of an item the partial sums are combined, O is normalised and O and the row lse are stored.
//   What bounds it at D = 128, per 128 x 128 step: 1024 cycles each of tensor pipe and special-function unit, 1280 of
//   shared memory.  With all sixteen softmax warps in step (one step at a time, 32 columns each) a step took 2170 cycles; two
//   groups with two S tiles 2250 (a group then waits for P V of its last step and for S), with three 1770.  The loops are
//   rolled to 32 columns: unrolled further, warps in different phases evict one another's code.
//   B2 H16 T4096 D128: 247 k -> 202 k cycles per CTA; B16 H12 T1024 D64: 118 k -> 98 k.
// Scale, causal mask, softmax and both products happen in this one pass; the T x T scores
// never reach global memory.
#include "sm100_ptx.cuh"
#include "tma_host.cuh"

#include <type_traits>

namespace {
using namespace sm100;

constexpr int BM = 128;
constexpr int BN = 128;
constexpr uint32_t BLOCK_BYTES = 128 * 128;   // one 64-column block of a 128-row tile
constexpr float LOG2E = 1.4426950408889634f;
constexpr float LN2 = 0.6931471805599453f;
constexpr float RESCALE_THRESHOLD = 8.0f;     // log2 units: P stays below 2^8, safe in f16
constexpr int NWG = 4;                        // softmax warpgroups: two groups of two
constexpr int CW = 64;                        // key columns of a step per warpgroup
constexpr int SM_WARP0 = 4;                   // first softmax warp; warps 0-3 are the Q / K producer, P V issuer, S issuer, V producer
constexpr int FWD_THREADS = 32 * (SM_WARP0 + 4 * NWG);

struct FwdParams {
    __half* o;
    float* lse;
    long long so_b, so_h, so_t;
    int B, H, T;
    int d;                      // head_dim: D or less (columns [d, D) read as zero and are not stored)
    int causal;
    float scale;
    unsigned int* err;
    const int4* sched;          // balanced schedule table[n * grid + cta] = {slot, slice, batch, head} (or nullptr: strided)
    int sched_rows;
};

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
    float y;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
}

// Dynamic shared memory only; the base must be 1024-byte aligned for the 128-byte swizzle (checked).
template <int D>
struct FwdSmem {
    static constexpr uint32_t TILE = 128u * D * 2u;
    static constexpr uint32_t Q = 0;                         // two buffers (alternate between items)
    static constexpr uint32_t K = Q + 2 * TILE;              // two stages
    static constexpr uint32_t V = K + 2 * TILE;              // two stages
    static constexpr uint32_t XCH = V + 2 * TILE;            // [2 groups][2 parities][2 warpgroups][128] partial row max
    static constexpr uint32_t MREF = XCH + 8 * BM * 4;       // [2 groups][128] reference maximum after the group's last step
    static constexpr uint32_t LX = MREF + 2 * BM * 4;        // [4 items][NWG warpgroups][2][128] partial row sum, its reference maximum
    static constexpr uint32_t BARS = LX + 8 * NWG * BM * 4;
    static constexpr uint32_t TOTAL = BARS + 256;
};

// P_FULL (first half of P's columns) and P2_FULL (second half), S_FULL and PV_DONE are one barrier per S tile, so that each
// stays at most one phase ahead of its waiter.
// S_FULL (all S products of a step have finished) also tells the producer that the step's K stage is
// free; PV_DONE (all P V products of a step have finished) also frees the V stage, tells the S
// issuer that the step's P has been consumed and orders a rescale of O behind the product.
enum FwdBar { F_Q_FULL = 0, F_Q_EMPTY = 2, F_K_FULL = 4, F_V_FULL = 6, F_PV_DONE = 8, F_S_FULL = 11,
              F_P_FULL = 14, F_XCH = 17, F_MREF = 19, F_LX = 21, F_O_DONE = 22, F_O_FREE = 24, F_P2_FULL = 26, F_COUNT = 29 };

// Work order: groups of 16 slices; inside a group the heaviest (latest) query tiles of all its
// slices come first (balance) and the group's K and V (a few MB) stay in L2.
struct WorkCursor {
    int n;          // index of the item inside this CTA's list
    int w;          // >= 0 while the cursor points at an item
    int4 e_next;    // table entry of the item after this one (prefetched)
    int j;          // KV tile inside the item
    int ntiles, qt, bh, b, h;
    // {slot, slice, batch, head} of this CTA's idx-th item; slot < 0 past the end.  With a host-built table
    // this is one load; the strided fallback pays the integer divisions.
    __device__ __forceinline__ int4 table(const FwdParams& p, int idx, int nq, int n_items) const {
        if (p.sched) return idx < p.sched_rows ? p.sched[idx * (int)gridDim.x + (int)blockIdx.x] : make_int4(-1, 0, 0, 0);
        const int v = (int)blockIdx.x + idx * (int)gridDim.x;
        if (v >= n_items) return make_int4(-1, 0, 0, 0);
        const int BH = p.B * p.H;
        const int group = v / (16 * nq);
        const int gsize = min(16, BH - group * 16);
        const int within = v - group * 16 * nq;
        const int s = group * 16 + within % gsize;
        return make_int4(within / gsize, s, s / p.H, s % p.H);
    }
    // Item n becomes current; the table entry of item n+1 is requested now and not looked at before the
    // next call, so its L2 round trip is off the item boundary.
    __device__ __forceinline__ void fetch(const FwdParams& p, int nq, int n_items) {
        const int4 e = uniform(e_next);                     // every user runs as a whole warp
        e_next = table(p, n + 1, nq, n_items);
        w = e.x;
        if (e.x >= 0) {
            qt = nq - 1 - e.x;                              // heaviest (latest) query tiles first
            bh = e.y; b = e.z; h = e.w;
            ntiles = p.causal ? qt + 1 : nq;
        }
    }
    __device__ __forceinline__ void init(const FwdParams& p, int nq, int n_items) {
        n = 0; j = 0;
        e_next = table(p, 0, nq, n_items);
        fetch(p, nq, n_items);
    }
    __device__ __forceinline__ bool valid(int) const { return w >= 0; }
    __device__ __forceinline__ void advance(const FwdParams& p, int nq, int n_items) {
        if (++j == ntiles) {
            j = 0; ++n;
            fetch(p, nq, n_items);
        }
    }
};

// The part of the start that needs nothing of global memory (see started()).
template <int D>
__device__ __forceinline__ void attn_fwd_f16_prologue(const void* tmap_q, const void* tmap_k, const void* tmap_v) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + FwdSmem<D>::BARS);
    uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(bars + F_COUNT);
    if (threadIdx.x == 0) {
        tmem_base_s[1] = 0;                                     // the abort flag
        for (int s = 0; s < 2; ++s) {
            mbar_init(&bars[F_Q_FULL + s], 1); mbar_init(&bars[F_Q_EMPTY + s], 1);
            mbar_init(&bars[F_K_FULL + s], 1);
            mbar_init(&bars[F_V_FULL + s], 1);
            mbar_init(&bars[F_O_DONE + s], 1); mbar_init(&bars[F_O_FREE + s], 4 * NWG);
            mbar_init(&bars[F_XCH + s], 8); mbar_init(&bars[F_MREF + s], 4);
        }
        for (int s = 0; s < 3; ++s) {
            mbar_init(&bars[F_S_FULL + s], 1); mbar_init(&bars[F_PV_DONE + s], 1);
            mbar_init(&bars[F_P_FULL + s], 8); mbar_init(&bars[F_P2_FULL + s], 8); // one arrival per warp of the step's group
        }
        mbar_init(&bars[F_LX], 4 * NWG);
        fence_barrier_init();
        tma_prefetch_desc(tmap_q); tma_prefetch_desc(tmap_k); tma_prefetch_desc(tmap_v);
    }
    if (uniform((int)threadIdx.x / 32) == 1) {
        tmem_alloc(tmem_base_s, 512);
        tmem_relinquish();
    }
}

template <int D>
__global__ void __launch_bounds__(FWD_THREADS, 1)
attn_fwd_f16_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                    const __grid_constant__ CUtensorMap tmap_v, const FwdParams p) {
    attn_fwd_f16_prologue<D>(&tmap_q, &tmap_k, &tmap_v);
    chain_wait();
    using L = FwdSmem<D>;
    constexpr uint32_t TILE_BYTES = L::TILE;
    constexpr int DBLK = D / 64;
    constexpr int DH = D / NWG;                              // O columns per softmax warpgroup
    constexpr uint32_t TMEM_COLS = 512;
    // three S tiles in turn (P in place) | O, two at D = 64 (even and odd items).  A third S tile is worth more than a second O:
    // with two, a group waits for P V of its last step and then for S before it can start the next.
    constexpr uint32_t TM_S = 0, TM_O = 384;
    constexpr int NOB = D == 64 ? 2 : 1;

    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sQ = smem + L::Q;
    uint8_t* sK = smem + L::K;
    uint8_t* sV = smem + L::V;
    float* xch = reinterpret_cast<float*>(smem + L::XCH);
    float* mref = reinterpret_cast<float*>(smem + L::MREF);
    float* lx = reinterpret_cast<float*>(smem + L::LX);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BARS);
    uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(bars + F_COUNT);
    volatile uint32_t* abort_s = tmem_base_s + 1;
    uint32_t* skip_s = tmem_base_s + 2;

    const int warp = uniform((int)threadIdx.x / 32), lane = threadIdx.x % 32;
    const int nq = (p.T + BM - 1) / BM;
    const int n_items = p.B * p.H * nq;

    if (!started(smem, skip_s, p.err, DEERS_KERR_FWD_F16 | 0x20)) {
        if (warp == 1) tmem_dealloc(*tmem_base_s, 512);
        return;
    }
    const uint32_t tmem = (uint32_t)uniform((int)*tmem_base_s);
    WaitState ws{abort_s, p.err};

    if (warp == 0) {
        // ------------------------------ TMA producer ------------------------------
        {
            WorkCursor c;
            c.init(p, nq, n_items);
            for (uint32_t g = 0; c.valid(n_items); ++g) {      // g: global step = K / V stage use
                const int b = c.b, h = c.h;
                if (c.j == 0) {
                    const int qb = c.n & 1;
                    if (!mbar_wait_warp(ws, &bars[F_Q_EMPTY + qb], (((uint32_t)c.n >> 1) & 1u) ^ 1u, DEERS_KERR_FWD_F16 | 1)) break;
                    if (elect_one()) {
                        mbar_arrive_expect_tx(&bars[F_Q_FULL + qb], TILE_BYTES);
#pragma unroll
                        for (int blk = 0; blk < DBLK; ++blk)
                            tma_load_4d(sQ + qb * TILE_BYTES + blk * BLOCK_BYTES, &tmap_q, &bars[F_Q_FULL + qb], blk * 64, c.qt * BM, h, b);
                    }
                    __syncwarp();
                }
                const uint32_t st = g & 1u;
                if (g >= 2 && !mbar_wait_warp(ws, &bars[F_S_FULL + (g - 2u) % 3u], ((g - 2u) / 3u) & 1u, DEERS_KERR_FWD_F16 | 2)) break;      // S of step g-2 done
                if (elect_one()) {
                    mbar_arrive_expect_tx(&bars[F_K_FULL + st], TILE_BYTES);
#pragma unroll
                    for (int blk = 0; blk < DBLK; ++blk)
                        tma_load_4d(sK + st * TILE_BYTES + blk * BLOCK_BYTES, &tmap_k, &bars[F_K_FULL + st], blk * 64, c.j * BN, h, b);
                }
                __syncwarp();
                c.advance(p, nq, n_items);
            }
        }
        __syncwarp();
        chain_next();                                           // all loads are under way: the end is near
    } else if (warp == 1) {
        // ------------------------------ P V issuer ------------------------------
        {
            constexpr uint32_t IDESC_O = idesc_f16(BM, D, 0, 1);       // O: A = P from TMEM, B = V MN-major
            constexpr uint64_t STAGE_STEP = TILE_BYTES >> 4;
            const uint64_t v_mn0 = desc_mnmajor((uint32_t)uniform((int)smem_u32(sV)), 0, BLOCK_BYTES);
            WorkCursor pc;
            pc.init(p, nq, n_items);
            for (uint32_t gp = 0; pc.valid(n_items); ++gp) {
                const uint32_t st = gp & 1u, sb = gp % 3u;
                if (!mbar_wait_warp(ws, &bars[F_P_FULL + sb], (gp / 3u) & 1u, DEERS_KERR_FWD_F16 | 6)) break;
                if (!mbar_wait_warp(ws, &bars[F_V_FULL + st], (gp >> 1) & 1u, DEERS_KERR_FWD_F16 | 7)) break;
                // The epilogue of the item that last used the accumulator must be over.
                if (pc.j == 0 && !mbar_wait_warp(ws, &bars[F_O_FREE + pc.n % NOB], ((uint32_t)(pc.n / NOB) & 1u) ^ 1u, DEERS_KERR_FWD_F16 | 8)) break;
                tc_fence_after_sync();
                const uint64_t v_mn = v_mn0 + (uint64_t)st * STAGE_STEP;
                const uint32_t o_tmem = tmem + TM_O + (uint32_t)(pc.n % NOB) * D;
                const uint32_t p_tmem = tmem + TM_S + sb * 128u;       // P sits where this step's S was
                // A warpgroup hands over the first 32 of its 64 columns, then the other 32: the product starts on the first.
                if (elect_one()) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int ks = (i >> 1) * 4 + (i & 1);
                        umma_ts(o_tmem, p_tmem + (uint32_t)(ks >> 2) * CW + (uint32_t)(ks & 3) * 8u, v_mn + mnmajor_step(ks), IDESC_O, (pc.j > 0 || i > 0));
                    }
                }
                __syncwarp();
                if (!mbar_wait_warp(ws, &bars[F_P2_FULL + sb], (gp / 3u) & 1u, DEERS_KERR_FWD_F16 | 6)) break;
                tc_fence_after_sync();
                if (elect_one()) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int ks = (i >> 1) * 4 + 2 + (i & 1);
                        umma_ts(o_tmem, p_tmem + (uint32_t)(ks >> 2) * CW + (uint32_t)(ks & 3) * 8u, v_mn + mnmajor_step(ks), IDESC_O, 1u);
                    }
                    umma_commit(&bars[F_PV_DONE + sb]);
                    if (pc.j == pc.ntiles - 1) umma_commit(&bars[F_O_DONE + pc.n % NOB]);
                }
                __syncwarp();
                pc.advance(p, nq, n_items);
            }
        }
    } else if (warp == 2) {
        // ------------------------------ S issuer ------------------------------
        {
            constexpr uint32_t IDESC_S = idesc_f16(BM, BN, 0, 0);      // S: K-major A (Q) and B (K)
            constexpr uint64_t STAGE_STEP = TILE_BYTES >> 4;
            const uint64_t q_km0 = desc_kmajor((uint32_t)uniform((int)smem_u32(sQ)), 0, BLOCK_BYTES);
            const uint64_t k_km0 = desc_kmajor((uint32_t)uniform((int)smem_u32(sK)), 0, BLOCK_BYTES);
            WorkCursor sc;
            sc.init(p, nq, n_items);
            for (uint32_t gs = 0; sc.valid(n_items); ++gs) {
                const uint32_t st = gs & 1u, sb = gs % 3u;
                const int qb = sc.n & 1;
                if (sc.j == 0 && !mbar_wait_warp(ws, &bars[F_Q_FULL + qb], ((uint32_t)sc.n >> 1) & 1u, DEERS_KERR_FWD_F16 | 4)) break;
                if (!mbar_wait_warp(ws, &bars[F_K_FULL + st], (gs >> 1) & 1u, DEERS_KERR_FWD_F16 | 5)) break;
                // This S tile still holds P of step gs-3 until the product reading it has finished.
                if (!mbar_wait_warp(ws, &bars[F_PV_DONE + sb], ((gs / 3u) & 1u) ^ 1u, DEERS_KERR_FWD_F16 | 0x15)) break;
                tc_fence_after_sync();
                const uint64_t q_km = q_km0 + (uint64_t)qb * STAGE_STEP, k_km = k_km0 + (uint64_t)st * STAGE_STEP;
                const uint32_t d_tmem = tmem + TM_S + sb * 128u;
                if (elect_one()) {
#pragma unroll
                    for (int ks = 0; ks < D / 16; ++ks)
                        umma_ss(d_tmem, q_km + kmajor_step(ks, BLOCK_BYTES), k_km + kmajor_step(ks, BLOCK_BYTES), IDESC_S, ks > 0);
                    umma_commit(&bars[F_S_FULL + sb]);
                    if (sc.j == sc.ntiles - 1) umma_commit(&bars[F_Q_EMPTY + qb]); // last product reading this Q
                }
                __syncwarp();
                sc.advance(p, nq, n_items);
            }
        }
    } else if (warp == 3) {
        // ------------------------------ V producer ------------------------------
        // A warp of its own: V of a step waits for P V two steps back, and K of the next step must not wait behind it.
        WorkCursor c;
        c.init(p, nq, n_items);
        for (uint32_t g = 0; c.valid(n_items); ++g) {
            const uint32_t st = g & 1u;
            if (g >= 2 && !mbar_wait_warp(ws, &bars[F_PV_DONE + (g - 2u) % 3u], ((g - 2u) / 3u) & 1u, DEERS_KERR_FWD_F16 | 3)) break;
            if (elect_one()) {
                mbar_arrive_expect_tx(&bars[F_V_FULL + st], TILE_BYTES);
#pragma unroll
                for (int blk = 0; blk < DBLK; ++blk)
                    tma_load_4d(sV + st * TILE_BYTES + blk * BLOCK_BYTES, &tmap_v, &bars[F_V_FULL + st], blk * 64, c.j * BN, c.h, c.b);
            }
            __syncwarp();
            c.advance(p, nq, n_items);
        }
    } else if (warp >= SM_WARP0) {
        // ------------------------------ softmax + epilogue ------------------------------
        const int wg = (warp - SM_WARP0) >> 2;                  // 0..3
        const int grp = wg >> 1, half = wg & 1;                 // steps of parity grp, key columns [64 half, 64 half + 64)
        const int lane_base = (warp & 3) * 32;
        const int row = lane_base + lane;                       // row inside the query tile == TMEM lane
        const uint32_t t_lane = (uint32_t)lane_base << 16;
        const float sl2 = p.scale * LOG2E;
        uint32_t gstep0 = 0;                                    // global step of the item's first KV tile
        bool alive = true;

        // Deferred epilogue of the previous item (runs after this item's first P has been handed over).
        int pend_n = -1, pend_grow = 0, pend_bh = 0, pend_b = 0, pend_h = 0;
        auto epilogue = [&]() -> bool {
            if (pend_n < 0) return true;
            const int n = pend_n;
            pend_n = -1;
            // Combine the partial row sums of the warpgroups, each relative to the reference maximum its group saw last; the
            // largest of these is the one O is scaled by.
            const float* lxp = lx + (n & 3) * 2 * NWG * BM + row;
            if (!__all_sync(0xffffffffu, mbar_wait(ws, &bars[F_LX], (uint32_t)n & 1u, DEERS_KERR_FWD_F16 | 9))) return false;
            float m = -INFINITY, l = 0.f;
#pragma unroll
            for (int w = 0; w < NWG; ++w) m = fmaxf(m, lxp[(2 * w + 1) * BM]);
            const float m_safe = (m == -INFINITY) ? 0.f : m;
#pragma unroll
            for (int w = 0; w < NWG; ++w) l = fmaf(lxp[2 * w * BM], ex2(lxp[(2 * w + 1) * BM] - m_safe), l);   // same order everywhere
            if (!__all_sync(0xffffffffu, mbar_wait(ws, &bars[F_O_DONE + n % NOB], (uint32_t)(n / NOB) & 1u, DEERS_KERR_FWD_F16 | 10))) return false;
            tc_fence_after_sync();
            const float inv = 1.f / l;
            // The thread's quarter row of O, as 16-byte pieces, is transposed within lane groups so that
            // every store instruction writes whole contiguous row segments.
            constexpr int NP = DH / 8;
            uint4 oc[NP];
            {
                uint32_t r[DH];
                const uint32_t to = tmem + TM_O + (uint32_t)(n % NOB) * D + t_lane + wg * DH;
                if constexpr (DH == 32) tmem_ld_x32(to, *reinterpret_cast<uint32_t(*)[32]>(&r[0]));
                else tmem_ld_x16(to, *reinterpret_cast<uint32_t(*)[16]>(&r[0]));
                tmem_wait_ld();
                tc_fence_before_sync();
                mbar_arrive_warp(&bars[F_O_FREE + n % NOB]);    // accumulator is in registers: release it
#pragma unroll
                for (int q8 = 0; q8 < NP; ++q8) oc[q8] = pack8_f16(r + q8 * 8, inv);
            }
            transpose_pieces<NP>(oc, (uint32_t)lane);
            const int grow0 = pend_grow - lane + (lane & ~(NP - 1));
            const int col = wg * DH + (lane & (NP - 1)) * 8;
            __half* ob = p.o + pend_b * p.so_b + pend_h * p.so_h + col;
#pragma unroll
            for (int c = 0; c < NP; ++c) {
                const int grow = grow0 + c;
                if (grow < p.T && col < p.d) *reinterpret_cast<uint4*>(ob + (long long)grow * p.so_t) = oc[c];
            }
            if (wg == 0 && pend_grow < p.T) p.lse[(long long)pend_bh * p.T + pend_grow] = (m + log2f(l)) * LN2;
            return true;
        };

        WorkCursor c;
        c.init(p, nq, n_items);
        // One more round than items, without steps, for the last epilogue: it has a single call site (and one in
        // the rare rescale: its code four times over no longer fits the instruction cache).
        for (;;) {
            const bool valid = c.valid(n_items);
            const int n = c.n, qt = c.qt, ntiles = valid ? c.ntiles : 0;
            const int q0 = qt * BM;
            float m_seen = -INFINITY, l = 0.f;                  // l: partial sum over this warpgroup's columns, relative to 2^m_seen
            for (int j = (int)((gstep0 ^ (uint32_t)grp) & 1u); alive; j += 2) {
                if (j < ntiles) {
                    const uint32_t gstep = gstep0 + (uint32_t)j;    // gstep & 1 == grp
                    const uint32_t ph = (gstep >> 1) & 1u, sb = gstep % 3u;
                    if (!__all_sync(0xffffffffu, mbar_wait(ws, &bars[F_S_FULL + sb], (gstep / 3u) & 1u, DEERS_KERR_FWD_F16 | 11))) { alive = false; break; }
                    tc_fence_after_sync();
                    const uint32_t ts = tmem + TM_S + sb * 128u + t_lane + CW * half;
                    // Column CW*half + i of this tile is valid iff i <= lim: on the diagonal tile (where k0 == q0) the key may not
                    // lie right of the query, and keys end at T.
                    const int k0 = j * BN;
                    const bool edge = (p.causal && j == qt) || (k0 + BN > p.T);
                    int lim = edge ? p.T - 1 - k0 - CW * half : CW;
                    if (p.causal && j == qt) lim = min(lim, row - CW * half);
                    // Two sweeps over the scores, 32 at a time: a row's 64 scores and their exponentials do not fit in 96 registers,
                    // and reading TMEM again is cheaper than spilling.
                    // Two copies of each loop: only the diagonal / tail tile pays for masking.
                    float mx = -INFINITY;
                    auto row_max = [&](auto edge_c) {
                        constexpr bool EDGE = decltype(edge_c)::value;
#pragma unroll 1
                        for (int q = 0; q < CW / 32; ++q) {
                            float s[32];
                            tmem_ld_x32(ts + q * 32, *reinterpret_cast<uint32_t(*)[32]>(&s[0]));
                            tmem_wait_ld();
                            if (EDGE) {
#pragma unroll
                                for (int i = 0; i < 32; ++i) s[i] = (i > lim - q * 32) ? -INFINITY : s[i] * sl2;
                            }
                            float m4[4] = {mx, s[0], s[1], s[2]};                // four chains: a single one is latency-bound
#pragma unroll
                            for (int i = 3; i < 31; i += 2) m4[(i >> 1) & 3] = max3(m4[(i >> 1) & 3], s[i], s[i + 1]);
                            mx = max3(max3(m4[0], m4[1], m4[2]), m4[3], s[31]);
                        }
                    };
                    if (edge || sl2 < 0.f) row_max(std::true_type{});
                    else { row_max(std::false_type{}); mx *= sl2; }
                    // The reference maximum after the previous step, which the other group took.  Read before this warp's arrival
                    // below: this group publishes its own after that exchange, and the other group may write again only then.
                    float m_prev = -INFINITY;
                    if (gstep > 0) {
                        const uint32_t g1 = gstep - 1u;
                        if (!__all_sync(0xffffffffu, mbar_wait(ws, &bars[F_MREF + (g1 & 1u)], (g1 >> 1) & 1u, DEERS_KERR_FWD_F16 | 14))) { alive = false; break; }
                        if (j > 0) m_prev = mref[(g1 & 1u) * BM + row];
                    }
                    // Exchange the partial row max with the twin thread of the other warpgroup.
                    float* xp = xch + (grp * 2 + ph) * 2 * BM + row;
                    xp[half * BM] = mx;
                    mbar_arrive_warp(&bars[F_XCH + grp]);
                    if (!__all_sync(0xffffffffu, mbar_wait(ws, &bars[F_XCH + grp], ph, DEERS_KERR_FWD_F16 | 12))) { alive = false; break; }
                    mx = fmaxf(mx, xp[(half ^ 1) * BM]);

                    const float m_new = fmaxf(m_prev, mx);
                    // Lazy rescale: keep the old reference max unless this row grew by more than 2^8.
                    const bool grow = (j > 0) && (m_new - m_prev > RESCALE_THRESHOLD);
                    const float m_cur = (j == 0 || grow) ? m_new : m_prev;
                    if (half == 0) {
                        mref[grp * BM + row] = m_cur;
                        mbar_arrive_warp(&bars[F_MREF + grp]);
                    }
                    const float m_safe = (m_cur == -INFINITY) ? 0.f : m_cur;
                    const bool warp_grow = __any_sync(0xffffffffu, grow);
                    l *= ex2(m_seen - m_safe);                      // 0 * 0 the first time
                    m_seen = m_cur;

                    if (j > 0 && warp_grow) {
                        // O += P V of the previous step must have landed before O is rescaled.  That product may be the item's
                        // first and wait for the previous item's O tile to leave, which is then due here.
                        if (!epilogue()) { alive = false; break; }
                        const float alpha = ex2(m_prev - m_safe);
                        const uint32_t g1 = gstep - 1u;
                        if (!__all_sync(0xffffffffu, mbar_wait(ws, &bars[F_PV_DONE + g1 % 3u], (g1 / 3u) & 1u, DEERS_KERR_FWD_F16 | 13))) { alive = false; break; }
                        tc_fence_after_sync();
                        const uint32_t to = tmem + TM_O + (uint32_t)(n % NOB) * D + t_lane + half * (D / 2);
#pragma unroll 1
                        for (int cc = 0; cc < D / 2; cc += 32) {
                            uint32_t r[32];
                            tmem_ld_x32(to + cc, r);
                            tmem_wait_ld();
#pragma unroll
                            for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
                            tmem_st_x32(to + cc, r);
                        }
                    }

                    const uint64_t c1_2 = pack_f32x2(sl2, sl2), nm_2 = pack_f32x2(-m_safe, -m_safe);
                    uint64_t rs = 0;
                    auto make_p = [&](auto edge_c) {
                        constexpr bool EDGE = decltype(edge_c)::value;
#pragma unroll 1
                        for (int q = 0; q < CW / 32; ++q) {
                            uint32_t sr[32], pk[16];
                            tmem_ld_x32(ts + q * 32, sr);
                            tmem_wait_ld();
#pragma unroll
                            for (int i = 0; i < 16; ++i) {
                                float e0, e1;
                                unpack_f32x2(fma2(pack_f32x2(sr[2 * i], sr[2 * i + 1]), c1_2, nm_2), e0, e1);
                                e0 = ex2(e0); e1 = ex2(e1);
                                if (EDGE) {
                                    if (2 * i > lim - q * 32) e0 = 0.f;
                                    if (2 * i + 1 > lim - q * 32) e1 = 0.f;
                                }
                                rs = add2(rs, pack_f32x2(e0, e1));
                                pk[i] = pack_half2(e0, e1);
                            }
                            // P replaces scores that have been read (32 packed columns, 16 at a time).
                            tmem_st_x16(ts + q * 16, pk);
                            tmem_wait_st();
                            tc_fence_before_sync();
                            mbar_arrive_warp(&bars[F_P_FULL + sb + q * (F_P2_FULL - F_P_FULL)]);
                        }
                    };
                    if (edge) make_p(std::true_type{});
                    else make_p(std::false_type{});
                    float r0, r1;
                    unpack_f32x2(rs, r0, r1);
                    l += r0 + r1;
                }
                // the previous item's O tile, after this item's first P (or right away: an item without a step of this group)
                if (!epilogue()) { alive = false; break; }
                if (j + 2 >= ntiles) break;
            }
            if (!alive || !valid) break;
            pend_n = n; pend_grow = q0 + row; pend_bh = c.bh; pend_b = c.b; pend_h = c.h;
            float* lxp = lx + (n & 3) * 2 * NWG * BM + 2 * wg * BM + row;     // partial row sum for the epilogue
            lxp[0] = l; lxp[BM] = m_seen;
            mbar_arrive_warp(&bars[F_LX]);
            gstep0 += (uint32_t)ntiles;
            // advance the cursor by a whole item
            c.j = ntiles - 1;
            c.advance(p, nq, n_items);
        }
    }

    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, TMEM_COLS);
}

template <int D>
int fwd_launch(deers_ctx* ctx, const deers_attn_desc* d, const void* q, const void* k, const void* v, void* o,
               float* lse) {
    CUtensorMap tq, tk, tv;
    int rc;
    if ((rc = make_tmap_bhtd_f16(ctx, &tq, q, d->B, d->H, d->T, d->D, d->q_strides, BM))) return rc;
    if ((rc = make_tmap_bhtd_f16(ctx, &tk, k, d->B, d->H, d->T, d->D, d->k_strides, BN))) return rc;
    if ((rc = make_tmap_bhtd_f16(ctx, &tv, v, d->B, d->H, d->T, d->D, d->v_strides, BN))) return rc;
    FwdParams p;
    p.o = (__half*)o; p.lse = lse;
    p.so_b = d->o_strides[0]; p.so_h = d->o_strides[1]; p.so_t = d->o_strides[2];
    p.B = d->B; p.H = d->H; p.T = d->T; p.d = d->D; p.causal = d->causal; p.scale = d->scale; p.err = ctx->dev_err;
    const size_t smem = FwdSmem<D>::TOTAL;
    DEERS_SMEM_ONCE(ctx, (attn_fwd_f16_kernel<D>), smem);
    const long long nq = (d->T + BM - 1) / BM;
    const long long items = nq * d->B * d->H;
    if (items > 0x7fffffffLL) return DEERS_ERR_SHAPE;
    const unsigned grid = (unsigned)(items < ctx->sm_count ? items : ctx->sm_count);
    p.sched = deers_get_schedule(ctx, d->B, d->H, (int)nq, d->causal, (int)grid, &p.sched_rows);
    {
        const ChainScope chain(ctx, items * (d->causal ? (nq + 1) / 2 : nq) / grid);
        KernelTimerScope ts(ctx, DEERS_K_FWD);
        DEERS_CUDA_TRY(ctx, launch_chained(ctx, attn_fwd_f16_kernel<D>, grid, FWD_THREADS, smem, 1, tq, tk, tv, p));
    }
    ctx->launches += 1;
    DEERS_CUDA_TRY(ctx, cudaGetLastError());
    return DEERS_OK;
}

}  // namespace

int launch_attn_fwd_f16(deers_ctx* ctx, const deers_attn_desc* d, const void* q, const void* k, const void* v,
                        void* o, float* lse) {
    // Any multiple of 8: TMA fills the columns between head_dim and the tile width with zeros (they change neither
    // Q K^T nor P V), and the epilogue does not store them.
    if (d->D <= 64) return fwd_launch<64>(ctx, d, q, k, v, o, lse);
    return fwd_launch<128>(ctx, d, q, k, v, o, lse);
}
