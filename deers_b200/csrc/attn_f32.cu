// f32 causal attention: the choice of kernel and the launches (the kernels: attn_f32_kernel.cuh).
#include "attn_f32_kernel.cuh"

namespace {

// Blocks of 32 rows of `kinds` kinds.
long long blocks_of(const F32Params& p, int kinds) { return (long long)kinds * p.B * p.H * ((p.T + 31) / 32); }

// Calls of at most per_sm blocks per SM: then a block's walk is what the call takes.
bool few_blocks(const deers_ctx* ctx, const F32Params& p, int kinds, int per_sm) { return blocks_of(p, kinds) <= (long long)per_sm * ctx->sm_count; }

// Stationary rows per thread (an eighth of a block's).  Forward: 8 rows a block while those are one per SM, 16 up to two (us, 32 / 16 / 8 rows:
// B1 H6 T128 D64 7.4 / 5.0 / 4.2, B1 H6 T256 D32 7.2 / 4.8 / 5.4, B1 H12 T333 D32 10.0 / 8.9 / 12.7, B8 H4 T100 D32 4.8 / 4.3 / 5.4, B4 H6 T256
// D32 8.7 / 10.4 / 16.5).
int fwd_rows(const deers_ctx* ctx, const F32Params& p) {
    const long long blocks = blocks_of(p, 1);
    return 4 * blocks <= ctx->sm_count ? 1 : 2 * blocks <= 2 * ctx->sm_count ? 2 : 4;
}
// Backward, `resident` blocks of a kind's size per SM: a wave and a fifth of short walks, two of longer ones, whose causal halves differ (B3 H4 T77
// D48 13.6 / 8.2 / 9.3, B8 H4 T100 D32 10.1 / 12.0 / 16.4; B1 H8 T512 D32 33.0 / 29.3 / 45.6, B2 H6 T256 D96 36 / 48 / 69, B1 H3 T200 D48 20.5 /
// 12.4 / 10.1).
int bwd_rows(const deers_ctx* ctx, const F32Params& p, int resident) {
    const long long blocks = blocks_of(p, 2), slots = (long long)resident * ctx->sm_count;
    if (4 * blocks * 5 <= 6 * ctx->sm_count) return 1;
    return p.T > 128 ? (2 * blocks <= 2 * slots ? 2 : 4) : (2 * blocks * 5 <= 6 * slots ? 2 : 4);
}

// Blocks of 8 or 16 rows (rm 1 or 2), from the module of the tile width.
template <int DP>
int fwd_few_blocks(deers_ctx* ctx, const F32Params& p, int groups, int stream, int rm) {
    return DP == 32 ? launch_attn_fwd_f32_few32(ctx, p, groups, stream, rm) : DP == 64 ? launch_attn_fwd_f32_few64(ctx, p, groups, stream, rm)
         : DP == 96 ? launch_attn_fwd_f32_few96(ctx, p, groups, stream, rm) : launch_attn_fwd_f32_few128(ctx, p, groups, stream, rm);
}
template <int DP>
int bwd_few_blocks(deers_ctx* ctx, const F32Params& p, int groups, int rm) {
    return DP == 32 ? launch_attn_bwd_f32_few32(ctx, p, groups, rm) : DP == 64 ? launch_attn_bwd_f32_few64(ctx, p, groups, rm)
         : DP == 96 ? launch_attn_bwd_f32_few96(ctx, p, groups, rm) : launch_attn_bwd_f32_few128(ctx, p, groups, rm);
}

template <int DP, int NG, int FBN>
int fwd_any_rows(deers_ctx* ctx, const F32Params& p) {
    const int rm = fwd_rows(ctx, p);
    return rm == 4 ? fwd_launch_f32<DP, NG, FBN, 4>(ctx, p) : fwd_few_blocks<DP>(ctx, p, NG, FBN, rm);
}

// Narrow heads stream 64 keys at a time (half the reads of Q per score), unless the sequence has so few tiles that groups
// would go without: up to 128 keys, tiles of 32 (B1 H6 T100 D32 5.8 -> 4.8 us, B3 H4 T77 D48 8.8 -> 6.8).  Heads up to 32 wide
// take eight groups of 32 keys each where the blocks are few: up to 256 keys that is one tile per group (B4 H6 T256 D32 10.8 ->
// 8.7), beyond, with an SM per block, half the walk (B1 H2 T1024 23.2 -> 21.5).  Heads of 64 do not gain (T 256 11.1 against 11.9,
// T 512 19.9 against 20.6).
// With more blocks heads up to 32 wide keep tiles of 32 keys to 512 of them, in blocks of 16 rows up to two of 32 per SM (tiles of 64 / these:
// B8 H6 T256 D32 14.4 / 12.4, B32 H12 T160 48.9 / 39.9, B4 H8 T400 19.4 / 18.2, B8 H8 T512 46.2 / 45.4; B2 H8 T300 13.2 / 8.8; error of O 1.9e-7
// / 1.8e-7).
template <int DP>
int fwd_impl(deers_ctx* ctx, const F32Params& p) {
    if constexpr (DP <= 32) {
        if (p.T > 128 && few_blocks(ctx, p, 1, p.T <= 256 ? 2 : 1)) return fwd_any_rows<DP, 8, 32>(ctx, p);
        if (p.T > 128 && p.T <= 512) return few_blocks(ctx, p, 1, 2) ? fwd_few_blocks<DP>(ctx, p, 4, 32, 2) : fwd_launch_f32<DP, 4, 32, 4>(ctx, p);
        if (p.T > 128) return fwd_launch_f32<DP, 4, 64, 4>(ctx, p);         // (more blocks than SMs: of 32 rows)
    }
    if constexpr (DP == 64) {
        if (p.T > 128) return fwd_any_rows<DP, 4, 64>(ctx, p);
    }
    return fwd_any_rows<DP, 4, 32>(ctx, p);
}

// Eight groups where every block has an SM to itself and more tiles than four groups take at once (B1 H6 T256 D32 14.5 -> 13.0 us,
// B1 H4 T256 D64 27.7 -> 23.3); with more blocks than SMs two of four groups each share one (B4 H6 T256 D32: 20.2 against 23.3).
template <int DP>
int bwd_impl(deers_ctx* ctx, const F32Params& p) {
    if constexpr (DP <= 64) {
        // (one block per SM at most: never 32 rows)
        if (p.T > 128 && few_blocks(ctx, p, 2, 1)) return bwd_few_blocks<DP>(ctx, p, 8, bwd_rows(ctx, p, 1));
    }
    const int rm = bwd_rows(ctx, p, DP <= 64 ? 2 : 1);
    return rm == 4 ? bwd_launch_f32<DP, 4, 4>(ctx, p) : bwd_few_blocks<DP>(ctx, p, 4, rm);
}

F32Params base_params(const deers_attn_desc* d) {
    F32Params p;
    memset(&p, 0, sizeof(p));
    p.B = d->B; p.H = d->H; p.T = d->T; p.D = d->D;
    p.causal = d->causal; p.scale = d->scale;
    p.sq = s3(d->q_strides); p.sk = s3(d->k_strides); p.sv = s3(d->v_strides);
    p.so = s3(d->o_strides); p.sdo = s3(d->do_strides);
    p.sdq = s3(d->dq_strides); p.sdk = s3(d->dk_strides); p.sdv = s3(d->dv_strides);
    return p;
}

}  // namespace

int launch_attn_fwd_f32(deers_ctx* ctx, const deers_attn_desc* d, const float* q, const float* k,
                        const float* v, float* o, float* lse) {
    F32Params p = base_params(d);
    p.q = q; p.k = k; p.v = v; p.out_o = o; p.lse_out = lse;
    p.vec = (d->D % 4 == 0) && rows_vec_ok(q, d->q_strides) && rows_vec_ok(k, d->k_strides) &&
            rows_vec_ok(v, d->v_strides);
    p.vec_out = (d->D % 4 == 0) && rows_vec_ok(o, d->o_strides);
    if (d->D <= 32) return fwd_impl<32>(ctx, p);
    if (d->D <= 64) return fwd_impl<64>(ctx, p);
    if (d->D <= 96) return fwd_impl<96>(ctx, p);
    return fwd_impl<128>(ctx, p);
}

int launch_attn_bwd_f32(deers_ctx* ctx, const deers_attn_desc* d, const float* q, const float* k,
                        const float* v, const float* o, const float* lse, const float* d_o, float* dq,
                        float* dk, float* dv, const float* cosv, const float* sinv) {
    F32Params p = base_params(d);
    p.cosv = cosv; p.sinv = sinv;
    p.q = q; p.k = k; p.v = v; p.o = o; p.lse = lse; p.d_o = d_o;
    p.dq = dq; p.dk = dk; p.dv = dv;
    p.vec = (d->D % 4 == 0) && rows_vec_ok(q, d->q_strides) && rows_vec_ok(k, d->k_strides) &&
            rows_vec_ok(v, d->v_strides) && rows_vec_ok(d_o, d->do_strides) && rows_vec_ok(o, d->o_strides);
    p.vec_out = (d->D % 4 == 0) && rows_vec_ok(dq, d->dq_strides) && rows_vec_ok(dk, d->dk_strides) && rows_vec_ok(dv, d->dv_strides);
    if (d->D <= 32) return bwd_impl<32>(ctx, p);
    if (d->D <= 64) return bwd_impl<64>(ctx, p);
    if (d->D <= 96) return bwd_impl<96>(ctx, p);
    return bwd_impl<128>(ctx, p);
}
