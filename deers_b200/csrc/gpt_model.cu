// The f32 GPT of src/models/gpt.rs as a device-resident object and its training step.
//
// Forward (GPT::forward, gpt.rs:329-355), per block (Block::forward, gpt.rs:236-240), five launches:
//   qkv = rmsnorm(x) * [Wq|Wk|Wv] (one GEMM; the norm's scale and the rotation of q and k in its epilogue); fused attention
//   reading q, k, v in place as strided views and writing O token-major; x1 = x + O * Wout (residual in the GEMM epilogue);
//   r = relu(rmsnorm(x1) * Wup), h = r*r (norm and relu in the GEMM); x2 = x1 + h * Wdown (epilogue).
//   Separate norm and rotary kernels, eight launches per block before, cost 1.4 to 2 us each at these sizes.
// Head: xf = rmsnorm(x) as an f16 pair; logits = xf * Wlm with each row's maximum and sum of exponentials per tile, from which a small kernel
// makes lse and the picked log-probabilities; the backward reads the logits once, in one pass, and feeds the two head GEMMs.
// Backward: the exact transposes of the above, with the relu^2 backward in a GEMM epilogue, the residual
// gradient added inside the RMSNorm backward (which also writes the normalised rows again, for the weight gradients), dQ / dK
// rotated back by the attention backward straight into the fused [N, 3C] gradient buffer next to dV, and one GEMM for the sum of
// the three input gradients.  Every launch is one of this library's kernels; there is no host round trip in a step.
// The weight gradients are off the critical path (nothing in the backward reads them): the four of a block are one
// launch on a second stream (four where one would be several waves of blocks, three and one for the block the backward ends with), forked from
// the main one where their operands are complete and joined before the gradient norm; captured, the two streams become two branches of the
// step's graph.  What they read is double-buffered by block.
#include "common.cuh"

#include <math.h>
#include <new>
#include <string>
#include <vector>

namespace {

struct LayerW {              // offsets (in floats) into the parameter-shaped arenas
    size_t qkv, out, up, down;
};

struct LayerAct {
    float *inv1, *qkv, *o, *lse, *x1, *inv2, *r, *h, *x2;
};

// Gradients inside a block (and its normalised rows): read by the weight gradients while the next block's are made.
struct LayerGrad {
    float *dx, *dh, *dx1, *dqkv, *n1, *n2;      // of the block's output, MLP hidden, x1, q|k|v; rmsnorm(x), rmsnorm(x1)
};

size_t align64(size_t n) { return (n + 63) / 64 * 64; }     // floats: 256-byte boundaries

}  // namespace

struct deers_gpt {
    deers_ctx* ctx;
    deers_gpt_config cfg;
    int max_batch;
    long long max_tokens;
    int D, Vld;
    // parameter-shaped arenas: weights, gradients, first and second moments
    size_t arena_floats;
    float* arena[4];
    size_t off_wte, off_lm;
    std::vector<LayerW> lw;
    std::vector<deers_optim_tensor> opt;           // one entry per physical buffer
    // activations
    float* act_base;
    float *x0, *invf, *xf, *logits, *ce_lse, *picked, *cosv, *sinv;
    std::vector<LayerAct> la;
    LayerGrad lg[2];
    float* dtmp;
    // second stream for the weight gradients; events are markers only (no timing)
    cudaStream_t side;
    cudaEvent_t ev_fork, ev_join, ev_done[2];
    bool done_valid[2];          // ev_done[i] was recorded in the current backward pass
    bool on_side;                // launches currently go to the side stream
    void* optim_scratch;
    float *loss_dev, *norm_dev;
    long long *ids_dev, *tgt_dev;
    // The head on the tensor core (gemm_f16x3_sm100.cu): f16 pairs of xf, of the head weight and of dlogits
    bool tc_head;
    void *xf_hi, *xf_lo, *w_hi, *w_lo, *dl_hi, *dl_lo;
    void* x3_ws;
    void* x3_ws_side;
    float2* ce_stats;            // what a training step's head product leaves of its rows, ce_parts (0: nothing) per row
    int ce_parts;
    size_t x3_ws_bytes;
    // pinned staging for train_step_host
    long long* ids_pin;
    float* out_pin;
    // CUDA graph of forward + loss + backward + gradient norm, for the last (B, T) seen
    bool graph_enabled;
    cudaGraphExec_t graph_exec;
    int graph_B, graph_T;
    int eager_steps_BT;          // eager steps run at (graph_B, graph_T) before capturing
    bool head_pair_current;      // w_hi / w_lo hold the present head weight (of calls that ran, not of calls that were captured)
    bool captured_updates;       // the caller holds a captured training step: its replays change the weights unseen
};

namespace {

#define GPT_TRY(expr)              \
    do {                           \
        int _rc = (expr);          \
        if (_rc) return _rc;       \
    } while (0)

int gemm(deers_gpt* m, int M, int N, int K, const float* a, long long lda, int a_mn, const float* b, long long ldb, int b_mn,
         float* c, long long ldc, int epi = DEERS_EPI_NONE, const float* r = nullptr, long long ldr = 0,
         float* aux = nullptr) {
    return launch_gemm_f32(m->ctx, M, N, K, a, lda, a_mn, b, ldb, b_mn, c, ldc, epi, r, ldr, aux);
}

// Launches made while a SideScope lives go to the weight-gradient stream, ordered after everything the main
// stream holds at construction.  done(i) marks the side stream's progress for a later wait_done(i) on the
// main stream (before it overwrites a buffer the side work reads).  With kernel timing on, or without a
// second stream, everything stays on the main stream.
struct SideScope {
    deers_gpt* m;
    cudaStream_t main;
    bool active;
    int rc;
    explicit SideScope(deers_gpt* m_) : m(m_), main(m_->ctx->stream), active(m_->side && !m_->ctx->timing), rc(DEERS_OK) {
        if (!active) return;
        if (cudaEventRecord(m->ev_fork, main) != cudaSuccess || cudaStreamWaitEvent(m->side, m->ev_fork, 0) != cudaSuccess) {
            rc = DEERS_ERR_CUDA;
            active = false;
            return;
        }
        m->ctx->stream = m->side;
        m->ctx->no_chain = true;
        m->on_side = true;
    }
    int done(int i) {
        if (!active) return rc;
        if (cudaEventRecord(m->ev_done[i], m->side) != cudaSuccess) return DEERS_ERR_CUDA;
        m->done_valid[i] = true;
        return DEERS_OK;
    }
    ~SideScope() {
        if (active) { m->ctx->stream = main; m->ctx->no_chain = false; m->on_side = false; }
    }
};

int wait_done(deers_gpt* m, int i) {
    if (!m->done_valid[i]) return DEERS_OK;
    return cudaStreamWaitEvent(m->ctx->stream, m->ev_done[i], 0) == cudaSuccess ? DEERS_OK : DEERS_ERR_CUDA;
}

// The main stream waits for all side work enqueued so far.
int join_side(deers_gpt* m) {
    if (!m->side || m->ctx->timing) return DEERS_OK;
    if (cudaEventRecord(m->ev_join, m->side) != cudaSuccess || cudaStreamWaitEvent(m->ctx->stream, m->ev_join, 0) != cudaSuccess)
        return DEERS_ERR_CUDA;
    return DEERS_OK;
}

void attn_desc(const deers_gpt* m, int B, int T, deers_attn_desc* d) {
    const int H = m->cfg.n_head, D = m->D, C = m->cfg.n_embd;
    memset(d, 0, sizeof(*d));
    d->B = B; d->H = H; d->T = T; d->D = D;
    d->dtype = DEERS_F32; d->causal = 1;
    d->scale = (float)(1.0 / sqrt((double)D));                       // gpt.rs:139, storage.rs:115-117
    const int64_t qkv[4] = {(int64_t)T * 3 * C, D, (int64_t)3 * C, 1};           // column slices of [N, 3C]
    const int64_t o[4] = {(int64_t)T * C, D, C, 1};                              // token-major [B, T, H, D]
    for (int i = 0; i < 4; ++i) {
        d->q_strides[i] = d->k_strides[i] = d->v_strides[i] = qkv[i];
        d->dq_strides[i] = d->dk_strides[i] = d->dv_strides[i] = qkv[i];
        d->o_strides[i] = o[i]; d->do_strides[i] = o[i];
    }
}

// Rotation of q | k inside [N, 3C], in place: heads that the GEMM's tiles do not hold whole.
int rotate_in_place(deers_gpt* m, int B, int T, int inverse, float* qkv) {
    deers_rope_desc desc, *d = &desc;
    const int H = m->cfg.n_head, D = m->D, C = m->cfg.n_embd;
    memset(d, 0, sizeof(*d));
    d->B = B; d->T = T; d->H = 2 * H; d->D = D;                      // q and k heads side by side
    d->dtype = DEERS_F32; d->inverse = inverse;
    const int64_t tok[4] = {(int64_t)T * 3 * C, (int64_t)3 * C, D, 1};           // (b, t, h, d) in [N, 3C]
    for (int i = 0; i < 4; ++i) d->src_strides[i] = d->dst_strides[i] = tok[i];
    return deers_b200_rope_pack(m->ctx, d, qkv, m->cosv, m->sinv, qkv);
}

GemmNorm norm_in(const deers_gpt* m, float* inv) {
    GemmNorm f{};
    f.eps = (float)m->cfg.rms_norm_eps;
    f.inv = inv;
    return f;
}

// with_head_pair: the head weight's f16 pair is made here (a training step changes the weight every time); otherwise the
// caller has it current.  keep: a backward follows (inverse norms and relu are wanted).  The logits go to `logits`, rows of ldl.
int forward(deers_gpt* m, const long long* ids, int B, int T, bool with_head_pair, bool keep, float* logits, long long ldl) {
    deers_ctx* ctx = m->ctx;
    const deers_gpt_config& c = m->cfg;
    const int C = c.n_embd, Hm = c.mlp_hidden_dim, V = c.vocab_size;
    const long long N = (long long)B * T;
    float* W = m->arena[0];
    for (bool& v : m->done_valid) v = false;
    GPT_TRY(launch_embedding_fwd(ctx, W + m->off_wte, ids, N, C, V, m->x0));                 // gpt.rs:343
    // Beside the blocks, which leave most of the memory bandwidth idle: the head weight's f16 pair (it changes every step) and the
    // cleared gradient of the embedding (its backward adds rows).  Behind the first product: SMs set up for kernels without
    // shared memory have to empty before a product can start on them (10 us at the head of a step).
    auto beside = [&]() -> int {
        const bool make_pair = m->tc_head && with_head_pair;
        if (!make_pair && !keep) return DEERS_OK;
        SideScope side(m);
        GPT_TRY(side.rc);
        if (make_pair) GPT_TRY(launch_split_f16x3(ctx, C, V, W + m->off_lm, m->Vld, 1.0f, m->w_hi, m->w_lo, m->Vld));
        if (keep) DEERS_CUDA_TRY(ctx, cudaMemsetAsync(m->arena[1] + m->off_wte, 0, (size_t)V * C * sizeof(float), ctx->stream));
        return side.done(0);
    };
    deers_attn_desc ad;
    attn_desc(m, B, T, &ad);
    if (c.n_layer == 0) GPT_TRY(beside());
    const float* x = m->x0;
    for (int l = 0; l < c.n_layer; ++l) {
        const LayerW& w = m->lw[l];
        LayerAct& a = m->la[l];
        GemmNorm f = norm_in(m, keep ? a.inv1 : nullptr);
        f.cosv = m->cosv; f.sinv = m->sinv; f.rope_cols = 2 * C; f.rope_d = m->D; f.rope_t = T;             // gpt.rs:135-136
        bool rotated;
        GPT_TRY(launch_gemm_f32_norm(ctx, (int)N, 3 * C, C, x, W + w.qkv, a.qkv, DEERS_EPI_NONE, nullptr, f, &rotated));   // norm1, q | k | v projections
        if (l == 0) GPT_TRY(beside());
        if (!rotated) GPT_TRY(rotate_in_place(m, B, T, 0, a.qkv));
        GPT_TRY(deers_b200_attn_fwd(ctx, &ad, a.qkv, a.qkv + C, a.qkv + 2 * C, a.o, a.lse, nullptr, 0));
        GPT_TRY(gemm(m, (int)N, C, C, a.o, C, 0, W + w.out, C, 1, a.x1, C, DEERS_EPI_ADD, x, C));       // x + out_proj
        GPT_TRY(launch_gemm_f32_norm(ctx, (int)N, Hm, C, a.x1, W + w.up, a.h, DEERS_EPI_RELU_SQ, keep ? a.r : nullptr,
                                     norm_in(m, keep ? a.inv2 : nullptr), &rotated));        // norm2, up_proj, relu^2
        GPT_TRY(gemm(m, (int)N, C, Hm, a.h, Hm, 0, W + w.down, C, 1, a.x2, C, DEERS_EPI_ADD, a.x1, C)); // x1 + down_proj
        x = a.x2;
    }
    GPT_TRY(wait_done(m, 0));
    if (m->tc_head) {
        // lm_head on the tensor core at f32 accuracy: both operands as f16 pairs (the weight changes every step); gpt.rs:347
        int rc = launch_rmsnorm_split(ctx, N, C, c.rms_norm_eps, x, m->invf, m->xf_hi, m->xf_lo);
        if (rc == DEERS_ERR_UNSUPPORTED) {
            GPT_TRY(launch_rmsnorm_fwd(ctx, N, C, c.rms_norm_eps, x, m->xf, m->invf));
            rc = launch_split_f16x3(ctx, N, C, m->xf, C, 1.0f, m->xf_hi, m->xf_lo, C);
        }
        GPT_TRY(rc);
        GPT_TRY(launch_gemm_f16x3(ctx, (int)N, V, C, m->xf_hi, m->xf_lo, C, 0, m->w_hi, m->w_lo, m->Vld, 1, logits, ldl,
                                  1.0f, m->x3_ws, m->x3_ws_bytes, keep ? m->ce_stats : nullptr, &m->ce_parts));
    } else {
        GPT_TRY(launch_rmsnorm_fwd(ctx, N, C, c.rms_norm_eps, x, m->xf, m->invf));
        GPT_TRY(gemm(m, (int)N, V, C, m->xf, C, 0, W + m->off_lm, m->Vld, 1, logits, ldl));  // lm_head
    }
    return DEERS_OK;
}

int loss_and_backward(deers_gpt* m, const long long* ids, const long long* targets, int B, int T) {
    deers_ctx* ctx = m->ctx;
    const deers_gpt_config& c = m->cfg;
    const int C = c.n_embd, Hm = c.mlp_hidden_dim, V = c.vocab_size;
    const long long N = (long long)B * T;
    const int Vld = m->Vld;
    float* W = m->arena[0];
    float* G = m->arena[1];
    for (bool& v : m->done_valid) v = false;
    // (the loss itself is added up beside the backward)
    if (m->tc_head && m->ce_parts)
        GPT_TRY(launch_cross_entropy_merge(ctx, m->ce_stats, m->ce_parts, m->logits, Vld, targets, N, V, m->ce_lse, m->picked));
    else GPT_TRY(launch_cross_entropy_rows(ctx, m->logits, Vld, targets, N, V, m->ce_lse, m->picked));
    const float* x_last = c.n_layer ? m->la[c.n_layer - 1].x2 : m->x0;
    if (m->tc_head) {
        // dlogits leave the cross-entropy backward as f16 pairs scaled by rows * 4096 (|dlogit| <= 1 / rows)
        const float dscale = (float)N * 4096.0f;
        GPT_TRY(launch_cross_entropy_bwd_split(ctx, m->logits, Vld, targets, m->ce_lse, N, V, 1.0f, dscale, m->dl_hi, m->dl_lo, Vld));
        GPT_TRY(launch_gemm_f16x3(ctx, (int)N, C, V, m->dl_hi, m->dl_lo, Vld, 0, m->w_hi, m->w_lo, Vld, 0, m->dtmp, C,
                                  1.0f / dscale, m->x3_ws, m->x3_ws_bytes));                  // d xf = dlogits Wlm^T
        {
            SideScope side(m);
            GPT_TRY(side.rc);
            GPT_TRY(launch_gemm_f16x3(ctx, C, V, (int)N, m->xf_hi, m->xf_lo, C, 1, m->dl_hi, m->dl_lo, Vld, 1, G + m->off_lm, Vld,
                                      1.0f / dscale, m->x3_ws_side, m->x3_ws_bytes));         // d lm_head = xf^T dlogits
            GPT_TRY(launch_cross_entropy_loss(ctx, m->picked, N, m->loss_dev));               // (in front of it, it would start 2 us later)
        }
    } else {
        GPT_TRY(launch_cross_entropy_bwd(ctx, m->logits, Vld, targets, m->ce_lse, N, V, 1.0f, m->logits, Vld));
        GPT_TRY(gemm(m, (int)N, C, V, m->logits, Vld, 0, W + m->off_lm, Vld, 0, m->dtmp, C));    // d xf = dlogits Wlm^T
        {
            SideScope side(m);
            GPT_TRY(side.rc);
            GPT_TRY(gemm(m, C, V, (int)N, m->xf, C, 1, m->logits, Vld, 1, G + m->off_lm, Vld));  // d lm_head = xf^T dlogits
            GPT_TRY(launch_cross_entropy_loss(ctx, m->picked, N, m->loss_dev));
        }
    }
    const int last = c.n_layer ? (c.n_layer - 1) & 1 : 0;
    GPT_TRY(launch_rmsnorm_bwd(ctx, N, C, x_last, m->invf, m->dtmp, nullptr, m->lg[last].dx));
    const float* dx0 = m->lg[last].dx;
    deers_attn_desc ad;
    attn_desc(m, B, T, &ad);
    bool together = false;
    for (int l = c.n_layer - 1; l >= 0; --l) {
        const LayerW& w = m->lw[l];
        LayerAct& a = m->la[l];
        LayerGrad &d = m->lg[l & 1], &below = m->lg[(l & 1) ^ 1];
        const float* x_in = l ? m->la[l - 1].x2 : m->x0;
        // On the second stream: all four at the block's end in one launch, or each as soon as its operands are there.  Of block 0
        // the first three go ahead in one launch: nothing follows that all four could run beside (22 M parameters, 1024 tokens: 25 us of the four
        // behind the last norm, then 16 of the one).
        const GemmTN grads[4] = {{Hm, C, a.h, d.dx, G + w.down}, {C, Hm, d.n2, d.dh, G + w.up},              // d Wdown = h^T dx, d Wup = n2^T du
                                 {C, C, a.o, d.dx1, G + w.out}, {C, 3 * C, d.n1, d.dqkv, G + w.qkv}};        // d Wout = o^T dx1, d [Wq|Wk|Wv]
        if (l == c.n_layer - 1) together = gemm_f32_group_fits(ctx, 4, grads, (int)N);
        auto weight_grads = [&](int first, int n) -> int {
            SideScope side(m);
            GPT_TRY(side.rc);
            if (together && n > 1) GPT_TRY(launch_gemm_f32_group(ctx, n, grads + first, (int)N));
            else
                for (const GemmTN* t = grads + first; t < grads + first + n; ++t)
                    GPT_TRY(gemm(m, t->M, t->N, (int)N, t->a, t->M, 1, t->b, t->N, 1, t->c, t->N));
            return first + n == 4 ? side.done(l & 1) : DEERS_OK;
        };
        if (!together) GPT_TRY(weight_grads(0, 1));
        // MLP branch: x2 = x1 + relu(rmsnorm(x1) Wup)^2 Wdown
        GPT_TRY(gemm(m, (int)N, Hm, C, d.dx, C, 0, W + w.down, C, 0, d.dh, Hm, DEERS_EPI_MUL_AUX2, nullptr, 0, a.r));
        GPT_TRY(gemm(m, (int)N, C, Hm, d.dh, Hm, 0, W + w.up, Hm, 0, m->dtmp, C));           // d n2 = du Wup^T
        GPT_TRY(launch_rmsnorm_bwd(ctx, N, C, a.x1, a.inv2, m->dtmp, d.dx, d.dx1, d.n2));    // d x1
        const bool ahead = together && l == 0;
        if (!together) GPT_TRY(weight_grads(1, 2));
        if (ahead) GPT_TRY(weight_grads(0, 3));
        // attention branch: x1 = x + attn(rmsnorm(x)) Wout
        GPT_TRY(gemm(m, (int)N, C, C, d.dx1, C, 0, W + w.out, C, 0, m->dtmp, C));            // d o (token-major)
        GPT_TRY(launch_attn_bwd_f32(ctx, &ad, a.qkv, a.qkv + C, a.qkv + 2 * C, a.o, a.lse, m->dtmp, d.dqkv, d.dqkv + C, d.dqkv + 2 * C,
                                    m->D % 8 ? nullptr : m->cosv, m->D % 8 ? nullptr : m->sinv));
        if (m->D % 8) GPT_TRY(rotate_in_place(m, B, T, 1, d.dqkv));
        GPT_TRY(gemm(m, (int)N, C, 3 * C, d.dqkv, 3 * C, 0, W + w.qkv, 3 * C, 0, m->dtmp, C)); // d n1 (three terms in one)
        GPT_TRY(wait_done(m, (l & 1) ^ 1));                                                  // the block above has read what this block's input gradient replaces
        GPT_TRY(launch_rmsnorm_bwd(ctx, N, C, x_in, a.inv1, m->dtmp, d.dx1, below.dx, d.n1)); // d x
        dx0 = below.dx;
        GPT_TRY(together && !ahead ? weight_grads(0, 4) : weight_grads(3, 1));
    }
    GPT_TRY(launch_embedding_bwd(ctx, dx0, ids, N, C, V, G + m->off_wte, true));           // (cleared in the forward)
    return join_side(m);
}

int grad_norm(deers_gpt* m) {
    return deers_b200_grad_norm(m->ctx, (int)m->opt.size(), m->opt.data(), m->norm_dev, m->optim_scratch,
                                deers_b200_optim_scratch_bytes());
}

int check_bt(const deers_gpt* m, int B, int T) {
    if (B < 1 || T < 1 || B > m->max_batch || T > m->cfg.sequence_len) return DEERS_ERR_SHAPE;   // gpt.rs:335
    return DEERS_OK;
}

// n ids and n targets in one launch.
__global__ void __launch_bounds__(256) stage_ids_kernel(const long long* ids, const long long* targets, long long n, long long* __restrict__ ids_out,
                                                        long long* __restrict__ targets_out) {
    chain_begin();
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
        const long long a = ids[i], b = targets[i];
        ids_out[i] = a; targets_out[i] = b;
    }
}

// Whether a kernel may touch the caller's memory at p: of this device and on a boundary of `size` bytes.  What is not (pinned or
// managed memory, another device's, a host pointer) is left to the copies, which take or refuse it.
bool plain_device(const deers_ctx* ctx, const void* p, size_t size) {
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) { cudaGetLastError(); return false; }
    return at.type == cudaMemoryTypeDevice && at.device == ctx->device && (uintptr_t)p % size == 0;
}

// Brings the caller's ids / targets into the model's own buffers, so that a captured graph reads fixed addresses.
int stage_ids(deers_gpt* m, const int64_t* ids, const int64_t* targets, long long N, cudaMemcpyKind kind) {
    deers_ctx* ctx = m->ctx;
    if (kind == cudaMemcpyDeviceToDevice && targets && (const long long*)ids != m->ids_dev && (const long long*)targets != m->tgt_dev &&
        plain_device(ctx, ids, sizeof(long long)) && plain_device(ctx, targets, sizeof(long long))) {
        const unsigned grid = (unsigned)((N + 255) / 256);
        DEERS_CUDA_TRY(ctx, launch_chained(ctx, stage_ids_kernel, grid, 256, 0, 1, (const long long*)ids, (const long long*)targets, N, m->ids_dev, m->tgt_dev));
        ctx->launches += 1;
        return DEERS_OK;
    }
    if ((const long long*)ids != m->ids_dev)
        DEERS_CUDA_TRY(ctx, cudaMemcpyAsync(m->ids_dev, ids, (size_t)N * sizeof(long long), kind, ctx->stream));
    if (targets && (const long long*)targets != m->tgt_dev)
        DEERS_CUDA_TRY(ctx, cudaMemcpyAsync(m->tgt_dev, targets, (size_t)N * sizeof(long long), kind, ctx->stream));
    return DEERS_OK;
}

// True while the caller records this stream: what is enqueued now runs later, any number of times or never, so nothing
// about the present may be concluded from it.
bool recording(const deers_gpt* m) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(m->ctx->stream, &st) != cudaSuccess) { cudaGetLastError(); return false; }
    return st != cudaStreamCaptureStatusNone;
}

void drop_graph(deers_gpt* m) {
    if (m->graph_exec) cudaGraphExecDestroy(m->graph_exec);
    m->graph_exec = nullptr;
}

// forward + loss + backward + gradient norm on the staged ids, replayed from a graph once a (B, T) repeats
int run_fwd_bwd(deers_gpt* m, int B, int T, bool with_norm) {
    deers_ctx* ctx = m->ctx;
    const bool can_graph = m->graph_enabled && with_norm && !ctx->timing;
    if (can_graph && m->graph_exec && m->graph_B == B && m->graph_T == T) {
        DEERS_CUDA_TRY(ctx, cudaGraphLaunch(m->graph_exec, ctx->stream));
        ctx->launches += 1;
        return DEERS_OK;
    }
    if (can_graph && (m->graph_B != B || m->graph_T != T)) {
        drop_graph(m);
        m->graph_B = B; m->graph_T = T; m->eager_steps_BT = 0;
    }
    if (can_graph && m->eager_steps_BT >= 1) {
        // the shape has run eagerly once (every kernel's attributes are set): capture it
        cudaGraph_t graph = nullptr;
        if (cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
            int rc = forward(m, m->ids_dev, B, T, true, true, m->logits, m->Vld);
            if (!rc) rc = loss_and_backward(m, m->ids_dev, m->tgt_dev, B, T);
            if (!rc) rc = grad_norm(m);
            const cudaError_t ce = cudaStreamEndCapture(ctx->stream, &graph);
            if (!rc && ce == cudaSuccess && graph &&
                cudaGraphInstantiate(&m->graph_exec, graph, 0) == cudaSuccess) {
                cudaGraphDestroy(graph);
                DEERS_CUDA_TRY(ctx, cudaGraphLaunch(m->graph_exec, ctx->stream));
                ctx->launches += 1;
                return DEERS_OK;
            }
            if (graph) cudaGraphDestroy(graph);
            m->graph_exec = nullptr;
            cudaGetLastError();
            m->graph_enabled = false;                                 // stay eager from here on
            if (rc) return rc;
        } else {
            cudaGetLastError();
            m->graph_enabled = false;
        }
    }
    GPT_TRY(forward(m, m->ids_dev, B, T, true, true, m->logits, m->Vld));
    GPT_TRY(loss_and_backward(m, m->ids_dev, m->tgt_dev, B, T));
    if (with_norm) GPT_TRY(grad_norm(m));
    if (can_graph) m->eager_steps_BT += 1;
    return DEERS_OK;
}

// logits [rows, ld] -> out [rows, V]; blockIdx.y is a row.  Rows of an odd V start on any 4-byte boundary.
__global__ void __launch_bounds__(256) copy_logits_kernel(const float* src, long long ld, float* __restrict__ dst, int V) {
    chain_begin();
    const float* s = src + blockIdx.y * ld;
    float* d = dst + (long long)blockIdx.y * V;
    for (int c = blockIdx.x * 1024 + threadIdx.x; c < V; c += gridDim.x * 1024) {
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = c + 256 * e < V ? ld_stream(s + c + 256 * e) : 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (c + 256 * e < V) __stcs(d + c + 256 * e, v[e]);
    }
}

const char* kBlockNames[6] = {"attn.q_proj", "attn.k_proj", "attn.v_proj", "attn.out_proj", "mlp.up_proj", "mlp.down_proj"};

// Logical parameter `index` -> device pointer inside arena `what`, shape and row stride.
int locate(const deers_gpt* m, int index, int what, float** ptr, long long* rows, long long* cols, long long* ld) {
    const deers_gpt_config& c = m->cfg;
    const int n = 2 + 6 * c.n_layer;
    if (index < 0 || index >= n || what < 0 || what > 3) return DEERS_ERR_SHAPE;
    float* base = m->arena[what];
    const int C = c.n_embd, Hm = c.mlp_hidden_dim;
    if (index == 0) { *ptr = base + m->off_wte; *rows = c.vocab_size; *cols = C; *ld = C; return DEERS_OK; }
    if (index == n - 1) { *ptr = base + m->off_lm; *rows = C; *cols = c.vocab_size; *ld = m->Vld; return DEERS_OK; }
    const int l = (index - 1) / 6, k = (index - 1) % 6;
    const LayerW& w = m->lw[l];
    switch (k) {
        case 0: case 1: case 2: *ptr = base + w.qkv + (size_t)k * C; *rows = C; *cols = C; *ld = 3 * C; break;
        case 3: *ptr = base + w.out; *rows = C; *cols = C; *ld = C; break;
        case 4: *ptr = base + w.up; *rows = C; *cols = Hm; *ld = Hm; break;
        default: *ptr = base + w.down; *rows = Hm; *cols = C; *ld = C; break;
    }
    return DEERS_OK;
}

}  // namespace

extern "C" int deers_b200_gpt_create(deers_ctx* ctx, const deers_gpt_config* cfg, int32_t max_batch, deers_gpt** out) {
    if (!ctx || !cfg || !out) return DEERS_ERR_NULL;
    *out = nullptr;
    if (cfg->vocab_size < 1 || cfg->sequence_len < 1 || cfg->n_layer < 0 || cfg->n_head < 1 || cfg->n_embd < 1 ||
        cfg->mlp_hidden_dim < 1 || max_batch < 1)
        return DEERS_ERR_SHAPE;
    if (cfg->n_embd % cfg->n_head) return DEERS_ERR_SHAPE;            // "n_embd must be divisible by n_head", gpt.rs:301
    const int D = cfg->n_embd / cfg->n_head;
    if (D % 2 || D > 128) return DEERS_ERR_SHAPE;                     // RoPE needs an even head_dim; f32 attention D <= 128
    if (2 + 4 * cfg->n_layer > 256) return DEERS_ERR_SHAPE;           // optimizer tensors per call
    const long long max_tokens = (long long)max_batch * cfg->sequence_len;
    if (max_tokens > 65535) return DEERS_ERR_SHAPE;                   // rows of the cross-entropy backward grid
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    deers_gpt* m = new (std::nothrow) deers_gpt();
    if (!m) return DEERS_ERR_CUDA;
    m->ctx = ctx; m->cfg = *cfg; m->max_batch = max_batch; m->max_tokens = max_tokens; m->D = D;
    m->Vld = (cfg->vocab_size + 7) / 8 * 8;                           // rows of the head, of the logits and of their f16 pairs start 16-byte aligned
    // Heads that fill the tensor core take the split-f16 products; small ones are products like those of the blocks.
    m->tc_head = cfg->vocab_size >= 1024 && cfg->n_embd % 8 == 0 && cfg->n_embd >= 64;
    m->graph_enabled = true; m->graph_exec = nullptr; m->graph_B = m->graph_T = -1; m->eager_steps_BT = 0;
    m->on_side = false;
    m->head_pair_current = m->captured_updates = false;
    {
        // the weight-gradient stream and its markers; without them the step simply runs on one stream
        bool ok = cudaStreamCreateWithFlags(&m->side, cudaStreamNonBlocking) == cudaSuccess;
        if (!ok) m->side = nullptr;
        cudaEvent_t* evs[4] = {&m->ev_fork, &m->ev_join, &m->ev_done[0], &m->ev_done[1]};
        for (cudaEvent_t* e : evs)
            if (cudaEventCreateWithFlags(e, cudaEventDisableTiming) != cudaSuccess) { *e = nullptr; ok = false; }
        if (!ok && m->side) { cudaStreamDestroy(m->side); m->side = nullptr; }
        cudaGetLastError();
    }
    const size_t C = cfg->n_embd, Hm = cfg->mlp_hidden_dim, V = cfg->vocab_size, N = (size_t)max_tokens;

    // ---- parameter-shaped arenas
    size_t off = 0;
    auto take = [&off](size_t n) { const size_t o = off; off += align64(n); return o; };
    m->off_wte = take(V * C);
    m->lw.resize(cfg->n_layer);
    for (auto& w : m->lw) { w.qkv = take(C * 3 * C); w.out = take(C * C); w.up = take(C * Hm); w.down = take(Hm * C); }
    m->off_lm = take(C * (size_t)m->Vld);
    m->arena_floats = off;
    int rc = DEERS_OK;
    for (int a = 0; a < 4 && !rc; ++a) {
        if (cudaMalloc((void**)&m->arena[a], off * sizeof(float)) != cudaSuccess ||
            cudaMemsetAsync(m->arena[a], 0, off * sizeof(float), ctx->stream) != cudaSuccess)
            rc = DEERS_ERR_CUDA;
    }
    auto add_opt = [m](size_t o, size_t n) {
        deers_optim_tensor t;
        t.w = m->arena[0] + o; t.g = m->arena[1] + o; t.m = m->arena[2] + o; t.v = m->arena[3] + o; t.n = (int64_t)n;
        m->opt.push_back(t);
    };
    if (!rc) {
        add_opt(m->off_wte, V * C);
        for (auto& w : m->lw) { add_opt(w.qkv, C * 3 * C); add_opt(w.out, C * C); add_opt(w.up, C * Hm); add_opt(w.down, Hm * C); }
        add_opt(m->off_lm, C * (size_t)m->Vld);
    }

    // ---- activations, scratch
    off = 0;
    struct Slot { float** p; size_t n; };
    std::vector<Slot> slots;
    auto want = [&slots](float** p, size_t n) { slots.push_back({p, n}); };
    want(&m->x0, N * C); want(&m->invf, N); want(&m->xf, N * C); want(&m->logits, N * (size_t)m->Vld);
    want(&m->ce_lse, N); want(&m->picked, N);
    want(&m->cosv, (size_t)cfg->sequence_len * (D / 2)); want(&m->sinv, (size_t)cfg->sequence_len * (D / 2));
    m->la.resize(cfg->n_layer);
    for (auto& a : m->la) {
        want(&a.inv1, N); want(&a.qkv, N * 3 * C); want(&a.o, N * C);
        want(&a.lse, N * cfg->n_head); want(&a.x1, N * C); want(&a.inv2, N);
        want(&a.r, N * Hm); want(&a.h, N * Hm); want(&a.x2, N * C);
    }
    for (auto& d : m->lg) {
        want(&d.dx, N * C); want(&d.dh, N * Hm); want(&d.dx1, N * C); want(&d.dqkv, N * 3 * C); want(&d.n1, N * C); want(&d.n2, N * C);
    }
    want(&m->dtmp, N * C);
    want(&m->loss_dev, 64);
    m->norm_dev = nullptr;
    size_t total = 0;
    for (auto& s : slots) total += align64(s.n);
    const size_t opt_bytes = deers_b200_optim_scratch_bytes();
    const size_t id_bytes = ((size_t)N * sizeof(long long) + 255) / 256 * 256;
    auto up256 = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t xf_h = up256(N * C * 2), w_h = up256(C * (size_t)m->Vld * 2), dl_h = up256(N * (size_t)m->Vld * 2);
    // K-split partial tiles of the head's input gradient: parts * tokens <= 148 * 128 * 128 / C + tokens, by pairs 74 * 256 * 192 / C
    const size_t x3 = m->tc_head ? up256(((size_t)148 * 16384 + N * C) * sizeof(float) * 2) : 0;
    m->x3_ws_bytes = x3;
    const size_t stats = up256(4 * ((V + 127) / 128) * N * sizeof(float2));
    const size_t tc_bytes = m->tc_head ? 2 * (xf_h + w_h + dl_h) + 2 * x3 + stats : 0;
    const size_t bytes = total * sizeof(float) + opt_bytes + 256 + 2 * id_bytes + tc_bytes;
    char* base = nullptr;
    if (!rc && cudaMalloc((void**)&base, bytes) != cudaSuccess) rc = DEERS_ERR_CUDA;
    if (!rc && cudaMemsetAsync(base, 0, bytes, ctx->stream) != cudaSuccess) rc = DEERS_ERR_CUDA;
    if (!rc) {
        m->act_base = (float*)base;
        float* p = (float*)base;
        for (auto& s : slots) { *s.p = p; p += align64(s.n); }
        m->norm_dev = m->loss_dev + 1;
        char* q = (char*)p;
        m->optim_scratch = q; q += (opt_bytes + 255) / 256 * 256;
        m->ids_dev = (long long*)q; q += id_bytes;
        m->tgt_dev = (long long*)q; q += id_bytes;
        if (m->tc_head) {
            m->xf_hi = q; q += xf_h; m->xf_lo = q; q += xf_h;
            m->w_hi = q; q += w_h; m->w_lo = q; q += w_h;
            m->dl_hi = q; q += dl_h; m->dl_lo = q; q += dl_h;
            m->x3_ws = q; q += x3;
            m->x3_ws_side = q; q += x3;
            m->ce_stats = (float2*)q; q += stats;
        }
        // rotary cache, f32 arithmetic of gpt.rs:12-46
        const int half = D / 2;
        std::vector<float> hc((size_t)cfg->sequence_len * half), hs(hc.size());
        for (int t = 0; t < cfg->sequence_len; ++t)
            for (int i = 0; i < half; ++i) {
                const float channel = (float)(2 * i);
                const float inv_freq = 1.0f / powf(cfg->rope_base, channel / (float)D);
                const float f = (float)t * inv_freq;
                hc[(size_t)t * half + i] = cosf(f);
                hs[(size_t)t * half + i] = sinf(f);
            }
        if (cudaMemcpyAsync(m->cosv, hc.data(), hc.size() * sizeof(float), cudaMemcpyHostToDevice, ctx->stream) != cudaSuccess ||
            cudaMemcpyAsync(m->sinv, hs.data(), hs.size() * sizeof(float), cudaMemcpyHostToDevice, ctx->stream) != cudaSuccess ||
            cudaStreamSynchronize(ctx->stream) != cudaSuccess)
            rc = DEERS_ERR_CUDA;
    }
    if (!rc && (cudaHostAlloc((void**)&m->ids_pin, 2 * (size_t)N * sizeof(long long), cudaHostAllocDefault) != cudaSuccess ||
                cudaHostAlloc((void**)&m->out_pin, 2 * sizeof(float), cudaHostAllocDefault) != cudaSuccess))
        rc = DEERS_ERR_CUDA;
    if (rc) {
        snprintf(ctx->last_error, sizeof(ctx->last_error), "gpt_create: %s", cudaGetErrorString(cudaGetLastError()));
        deers_b200_gpt_destroy(m);
        return rc;
    }
    *out = m;
    return DEERS_OK;
}

extern "C" void deers_b200_gpt_destroy(deers_gpt* m) {
    if (!m) return;
    cudaSetDevice(m->ctx->device);
    cudaStreamSynchronize(m->ctx->stream);
    drop_graph(m);
    if (m->side) { cudaStreamSynchronize(m->side); cudaStreamDestroy(m->side); }
    {
        cudaEvent_t evs[4] = {m->ev_fork, m->ev_join, m->ev_done[0], m->ev_done[1]};
        for (cudaEvent_t e : evs)
            if (e) cudaEventDestroy(e);
    }
    for (int a = 0; a < 4; ++a)
        if (m->arena[a]) cudaFree(m->arena[a]);
    if (m->act_base) cudaFree(m->act_base);
    if (m->ids_pin) cudaFreeHost(m->ids_pin);
    if (m->out_pin) cudaFreeHost(m->out_pin);
    delete m;
}

extern "C" int deers_b200_gpt_num_params(const deers_gpt* m) { return m ? 2 + 6 * m->cfg.n_layer : 0; }

extern "C" int deers_b200_gpt_param_info(const deers_gpt* m, int index, char* name, size_t name_bytes, int64_t* rows,
                                         int64_t* cols) {
    if (!m) return DEERS_ERR_NULL;
    float* p;
    long long r, c, ld;
    GPT_TRY(locate(m, index, 0, &p, &r, &c, &ld));
    if (rows) *rows = r;
    if (cols) *cols = c;
    if (name && name_bytes) {
        const int n = 2 + 6 * m->cfg.n_layer;
        if (index == 0) snprintf(name, name_bytes, "wte.weight");
        else if (index == n - 1) snprintf(name, name_bytes, "lm_head.weight");
        else snprintf(name, name_bytes, "blocks.%d.%s.weight", (index - 1) / 6, kBlockNames[(index - 1) % 6]);
    }
    return DEERS_OK;
}

extern "C" int deers_b200_gpt_param_set(deers_gpt* m, int index, int what, const float* host) {
    if (!m || !host) return DEERS_ERR_NULL;
    float* p;
    long long r, c, ld;
    GPT_TRY(locate(m, index, what, &p, &r, &c, &ld));
    m->head_pair_current = false;
    deers_ctx* ctx = m->ctx;
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    DEERS_CUDA_TRY(ctx, cudaMemcpy2DAsync(p, (size_t)ld * sizeof(float), host, (size_t)c * sizeof(float),
                                          (size_t)c * sizeof(float), (size_t)r, cudaMemcpyHostToDevice, ctx->stream));
    DEERS_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));          // the host array may be pageable and short-lived
    return DEERS_OK;
}

extern "C" int deers_b200_gpt_param_get(deers_gpt* m, int index, int what, float* host) {
    if (!m || !host) return DEERS_ERR_NULL;
    float* p;
    long long r, c, ld;
    GPT_TRY(locate(m, index, what, &p, &r, &c, &ld));
    deers_ctx* ctx = m->ctx;
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    DEERS_CUDA_TRY(ctx, cudaMemcpy2DAsync(host, (size_t)c * sizeof(float), p, (size_t)ld * sizeof(float),
                                          (size_t)c * sizeof(float), (size_t)r, cudaMemcpyDeviceToHost, ctx->stream));
    DEERS_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    return DEERS_OK;
}

extern "C" int deers_b200_gpt_set_graph(deers_gpt* m, int enable) {
    if (!m) return DEERS_ERR_NULL;
    m->graph_enabled = enable != 0;
    if (!enable) { drop_graph(m); m->graph_B = m->graph_T = -1; }
    return DEERS_OK;
}

extern "C" int deers_b200_gpt_graph_active(const deers_gpt* m) { return (m && m->graph_exec) ? 1 : 0; }

extern "C" int deers_b200_gpt_forward(deers_gpt* m, const int64_t* ids, int32_t B, int32_t T, float* logits) {
    if (!m || !ids) return DEERS_ERR_NULL;
    GPT_TRY(check_bt(m, B, T));
    deers_ctx* ctx = m->ctx;
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    const bool rec = recording(m), kept = m->head_pair_current && !m->captured_updates && !rec;
    const int V = m->cfg.vocab_size;
    // The tensor-core head writes the caller's dense rows itself; the small head's 16-byte stores want padded ones.
    const bool direct = logits && m->tc_head;
    GPT_TRY(forward(m, (const long long*)ids, B, T, !kept, false, direct ? logits : m->logits, direct ? V : m->Vld));
    if (!rec) m->head_pair_current = m->tc_head;
    if (logits && !direct) {
        const dim3 grid((unsigned)((V + 4095) / 4096), (unsigned)(B * T));
        DEERS_CUDA_TRY(ctx, launch_chained(ctx, copy_logits_kernel, grid, 256, 0, 1, m->logits, m->Vld, logits, V));
        ctx->launches += 1;
    }
    DEERS_CUDA_TRY(ctx, cudaGetLastError());
    return DEERS_OK;
}

extern "C" int deers_b200_gpt_forward_backward(deers_gpt* m, const int64_t* ids, const int64_t* targets, int32_t B,
                                               int32_t T, float* loss_dev) {
    if (!m || !ids || !targets) return DEERS_ERR_NULL;
    GPT_TRY(check_bt(m, B, T));
    deers_ctx* ctx = m->ctx;
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    GPT_TRY(stage_ids(m, ids, targets, (long long)B * T, cudaMemcpyDeviceToDevice));
    GPT_TRY(run_fwd_bwd(m, B, T, false));
    if (!recording(m)) m->head_pair_current = m->tc_head;
    if (loss_dev)
        DEERS_CUDA_TRY(ctx, cudaMemcpyAsync(loss_dev, m->loss_dev, sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream));
    return DEERS_OK;
}

static int train_step_common(deers_gpt* m, int B, int T, const deers_adamw_hyper* hyper, double max_grad_norm,
                             float* loss_out, float* norm_out) {
    GPT_TRY(run_fwd_bwd(m, B, T, true));
    m->head_pair_current = false;                                     // the update below changes the head weight
    m->captured_updates = m->captured_updates || recording(m);
    // clip_grad_norm + step_with_grads; "if grad_norm.is_finite() { step }" of tinystories_train.rs:213-216
    return launch_adamw(m->ctx, (int)m->opt.size(), m->opt.data(), hyper, m->norm_dev, max_grad_norm, true, StepSaid{m->loss_dev, loss_out, norm_out});
}

extern "C" int deers_b200_gpt_train_step(deers_gpt* m, const int64_t* ids, const int64_t* targets, int32_t B, int32_t T,
                                         const deers_adamw_hyper* hyper, double max_grad_norm, float* loss_dev,
                                         float* grad_norm_dev) {
    if (!m || !ids || !targets || !hyper) return DEERS_ERR_NULL;
    GPT_TRY(check_bt(m, B, T));
    if (hyper->step < 1) return DEERS_ERR_SHAPE;
    deers_ctx* ctx = m->ctx;
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    GPT_TRY(stage_ids(m, ids, targets, (long long)B * T, cudaMemcpyDeviceToDevice));
    float* const loss_out = loss_dev && plain_device(ctx, loss_dev, sizeof(float)) ? loss_dev : nullptr;
    float* const norm_out = grad_norm_dev && plain_device(ctx, grad_norm_dev, sizeof(float)) ? grad_norm_dev : nullptr;
    GPT_TRY(train_step_common(m, B, T, hyper, max_grad_norm, loss_out, norm_out));
    if (loss_dev && !loss_out)
        DEERS_CUDA_TRY(ctx, cudaMemcpyAsync(loss_dev, m->loss_dev, sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream));
    if (grad_norm_dev && !norm_out)
        DEERS_CUDA_TRY(ctx, cudaMemcpyAsync(grad_norm_dev, m->norm_dev, sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream));
    return DEERS_OK;
}

extern "C" int deers_b200_gpt_train_step_host(deers_gpt* m, const int64_t* ids_host, const int64_t* targets_host, int32_t B,
                                              int32_t T, const deers_adamw_hyper* hyper, double max_grad_norm,
                                              float* loss_host, float* grad_norm_host) {
    if (!m || !ids_host || !targets_host || !hyper) return DEERS_ERR_NULL;
    GPT_TRY(check_bt(m, B, T));
    if (hyper->step < 1) return DEERS_ERR_SHAPE;
    deers_ctx* ctx = m->ctx;
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    const long long N = (long long)B * T;
    memcpy(m->ids_pin, ids_host, (size_t)N * sizeof(long long));
    memcpy(m->ids_pin + m->max_tokens, targets_host, (size_t)N * sizeof(long long));
    GPT_TRY(stage_ids(m, (const int64_t*)m->ids_pin, (const int64_t*)(m->ids_pin + m->max_tokens), N, cudaMemcpyHostToDevice));
    GPT_TRY(train_step_common(m, B, T, hyper, max_grad_norm, nullptr, nullptr));
    DEERS_CUDA_TRY(ctx, cudaMemcpyAsync(m->out_pin, m->loss_dev, 2 * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    const int rc = deers_b200_sync(ctx);
    if (loss_host) *loss_host = m->out_pin[0];
    if (grad_norm_host) *grad_norm_host = m->out_pin[1];
    return rc;
}
