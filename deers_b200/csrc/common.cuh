// Shared internals of the deers_b200 library: the context object, status helpers
// and the launch prototypes each kernel file exports to the C-ABI layer.
#pragma once
#include <cuda_runtime.h>
#include <cuda.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <atomic>
#include <utility>

#include "../../include/deers_b200.h"

constexpr int DEERS_KT_RING = 512;

struct deers_ktimer {
    cudaEvent_t* start;     // DEERS_KT_RING events each, created when timing is first enabled
    cudaEvent_t* stop;
    int pending;            // recorded pairs not yet folded into total_ms
    double total_ms;
    uint64_t launches;
};

constexpr int DEERS_SCHED_CAP = 1 << 20;                 // ints per schedule table
constexpr int DEERS_SCHED_ENTRIES = 4;
struct deers_sched_entry {
    int key[5];             // key[0] < 0: empty
    int rows;
    int* dev;               // DEERS_SCHED_CAP ints of device memory
    int* host;              // pinned staging of the same size
    cudaEvent_t uploaded;   // recorded after the upload: the staging copy may be rewritten once it has fired
    uint64_t last_use;
};

struct deers_ctx {
    int device;
    cudaStream_t stream;
    bool owns_stream;
    int sm_count;
    // Error word the kernels write when a bounded wait gives up: dev_err in device
    // memory, host_err its pinned host mirror, refreshed by deers_b200_sync().
    unsigned int* host_err;
    unsigned int* dev_err;
    uint64_t launches;
    char last_error[256];
    // cuTensorMapEncodeTiled, fetched through the runtime so that the library
    // does not link against the driver.
    void* encode_tiled;
    bool timing;
    deers_ktimer kt[DEERS_K_COUNT];
    // Balanced work schedules of the persistent f16 kernels: table[n * grid + cta] = n-th work item
    // of that CTA (or -1), built on the host per (B, H, tiles, causal, grid).  A few shapes stay cached
    // (least recently used goes first), each with its own device table and pinned staging copy, so that a
    // caller alternating shapes (training / evaluation, the ragged last chunk of the host pipeline) neither
    // rebuilds nor waits: the upload is an asynchronous copy on the context's stream.
    deers_sched_entry sched[DEERS_SCHED_ENTRIES];
    uint64_t sched_clock;
    // Side streams and events of the host-tensor pipeline (created on first use).
    cudaStream_t h2d_stream, d2h_stream;
    cudaEvent_t pipe_ev[3][3];      // [buffer set][h2d done, compute done, d2h done]
    bool pipe_ready;
    bool no_chain;                  // launches follow work of another stream: nothing to overlap with (launch_chained)
    int cluster_capacity[9];        // [n]: clusters of n blocks the device holds at once (gemm_f32.cu; 0: not asked yet)
    int cluster_room_f16[9];        // the same for the f16 GEMM's CTAs (gemm_f16_sm100.cu)
};

// Brackets one kernel launch with events when timing is on.  A full ring drops the sample.
struct KernelTimerScope {
    deers_ctx* ctx;
    deers_ktimer* t;
    KernelTimerScope(deers_ctx* c, int kind) : ctx(c), t(nullptr) {
        if (c->timing && c->kt[kind].start && c->kt[kind].pending < DEERS_KT_RING) {
            t = &c->kt[kind];
            cudaEventRecord(t->start[t->pending], c->stream);
        }
    }
    ~KernelTimerScope() {
        if (t) {
            cudaEventRecord(t->stop[t->pending], ctx->stream);
            t->pending += 1;
        }
    }
};

// Returns DEERS_ERR_CUDA from the caller when `expr` fails.  The runtime keeps a failed call's error for the next
// cudaGetLastError(): it is taken here, or the next operator, which asks after its launches, would report it as its own.
#define DEERS_CUDA_TRY(ctx, expr)                                                            \
    do {                                                                                      \
        cudaError_t _e = (expr);                                                              \
        if (_e != cudaSuccess) {                                                              \
            snprintf((ctx)->last_error, sizeof((ctx)->last_error), "%s: %s", #expr,           \
                     cudaGetErrorString(_e));                                                 \
            cudaGetLastError();                                                               \
            return DEERS_ERR_CUDA;                                                            \
        }                                                                                     \
    } while (0)

// Opts a kernel into `bytes` of dynamic shared memory, once per call site (kernel instantiation) and device: the
// attribute stays with the function, and setting it on every launch costs the host about as much as a tensor map.
#define DEERS_SMEM_ONCE(ctx, kernel, bytes)                                                                         \
    do {                                                                                                            \
        static std::atomic<unsigned long long> _done{0};                                                            \
        const unsigned long long _bit = 1ull << ((ctx)->device & 63);                                               \
        if (!(_done.load(std::memory_order_acquire) & _bit)) {                                                      \
            DEERS_CUDA_TRY(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(bytes))); \
            _done.fetch_or(_bit, std::memory_order_release);                                                        \
        }                                                                                                           \
    } while (0)

// Back-to-back kernels.  A kernel launched by launch_chained() may be set up while the one before it still runs: it calls
// chain_wait() before its first access to global memory (the predecessor has finished and its writes are visible; every
// kernel of a chain waits, so this covers all before it) and chain_next() where its own successor may be set up.
// Saves the launch gap of a microsecond or two: 54 kernels (of then) of a GPT forward on a short prompt, replayed from a graph,
// 232 -> 206 us; launched one by one, where the host's time hides as well, 495 -> 214 us.  Where chain_next()
// stands matters: a successor set up at the start of a kernel of few large blocks takes the idle SMs unevenly (252 us), so
// those call it once their last loads are under way; kernels of small blocks call it first.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void chain_begin() { chain_next(); chain_wait(); }
// What a predecessor writes may change while a chained kernel is already resident, so its reads must be ordinary (coherent)
// loads behind the wait.  Pointers to such data are neither `const __restrict__` nor read by __ldg: both allow the read-only
// path, which promises the values of the kernel's start, and let the compiler move the load in front of the wait.  (Pointers
// that are only written may be __restrict__: it lets the loads of a loop run ahead of its stores.)
// One streaming (read once) float behind the wait.
__device__ __forceinline__ float ld_stream(const float* p) {
    float v;
    asm volatile("ld.global.cs.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}

// False while capturing, unless a kernel of this stream is the one predecessor (ctx.cu).
bool deers_can_chain(const deers_ctx* ctx);

// Every call looks at the result: the next kernel would work on what a refused one has not written.
template <typename... P, typename... A>
[[nodiscard]] cudaError_t launch_chained(deers_ctx* ctx, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, dim3 cluster, A&&... args) {
    cudaLaunchConfig_t lc{};
    lc.gridDim = grid;
    lc.blockDim = block;
    lc.dynamicSmemBytes = smem;
    lc.stream = ctx->stream;
    cudaLaunchAttribute at[2];
    unsigned n = 0;
    if (deers_can_chain(ctx)) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster.x * cluster.y * cluster.z > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = cluster.x; at[n].val.clusterDim.y = cluster.y; at[n++].val.clusterDim.z = cluster.z;
    }
    lc.attrs = at; lc.numAttrs = n;
    return cudaLaunchKernelEx(&lc, kernel, std::forward<A>(args)...);
}

// A long kernel of one block per SM gains nothing from an early start, and its blocks then land on the SMs in the order in
// which the predecessor's leave, not neighbours next to one another.  B64 H32 T2048 D128 forward and backward was never faster
// chained: 10870 us against 10470 unchained in one call, 11300 against 11180 and 11360 against 11220 in two more (runs of one
// side differ by 1.5 % and more there, so this is a choice between near equals); B2 H16 T8192 D128 2279 against 2264.
// steps: 128 x 128 score tiles (or the like, about half a microsecond) per block.
struct ChainScope {
    deers_ctx* ctx;
    bool was;
    ChainScope(deers_ctx* c, long long steps) : ctx(c), was(c->no_chain) { c->no_chain = was || steps > 128; }
    ~ChainScope() { ctx->no_chain = was; }
};

// Device-side error codes (upper byte: which kernel, lower bits: which wait).
enum {
    DEERS_KERR_FWD_F16 = 0x100,
    DEERS_KERR_BWD_F16 = 0x200,
    DEERS_KERR_SELFTEST = 0x300,
    DEERS_KERR_GEMM = 0x400,
    DEERS_KERR_GPT = 0x500,      // token id / target out of range
};

// Work schedule shared by the persistent f16 kernels (ctx.cu).  Work items are ordered in groups
// of 16 slices, heaviest tiles first inside a group (item -> (slot, slice), slot 0 heaviest, weight
// ntile - slot when causal).  The table hands the items, in that order, to whichever CTA is least
// loaded so far, which balances the causal triangle for any slice count.  Returns nullptr (plain
// strided assignment) when the table would not fit.
const int4* deers_get_schedule(deers_ctx* ctx, int B, int H, int ntile, int causal, int grid, int* rows);

// Argument validation shared by every attention entry point (ctx.cu)
int deers_check_desc(const deers_attn_desc* d);
int deers_check_tensor(const deers_attn_desc* d, const void* p, const int64_t* s, size_t esize);
int deers_check_bwd_args(const deers_attn_desc* d, const void* q, const void* k, const void* v, const void* o,
                         const float* lse, const void* d_o, void* dq, void* dk, void* dv);

// f32 attention, FFMA (attn_f32.cu)
int launch_attn_fwd_f32(deers_ctx* ctx, const deers_attn_desc* d, const float* q, const float* k,
                        const float* v, float* o, float* lse);
int launch_attn_bwd_f32(deers_ctx* ctx, const deers_attn_desc* d, const float* q, const float* k,
                        const float* v, const float* o, const float* lse, const float* d_o, float* dq,
                        float* dk, float* dv, const float* cosv = nullptr, const float* sinv = nullptr);

// f16 tcgen05 path (attn_fwd_f16_sm100.cu, attn_bwd_f16_sm100.cu)
int launch_attn_fwd_f16(deers_ctx* ctx, const deers_attn_desc* d, const void* q, const void* k,
                        const void* v, void* o, float* lse);
int launch_attn_bwd_f16(deers_ctx* ctx, const deers_attn_desc* d, const void* q, const void* k,
                        const void* v, const void* o, const float* lse, const void* d_o, void* dq,
                        void* dk, void* dv, void* workspace, bool keep_ds);
size_t attn_bwd_f16_workspace_bytes(const deers_attn_desc* d, bool keep_ds);
int run_selftest_umma(deers_ctx* ctx, float* max_abs_err);
int run_selftest_wait(deers_ctx* ctx, unsigned int limit_ms, int* result_host);

// f32 GEMM (gemm_f32.cu, gemm_f32_kernel.cuh)
int launch_gemm_f32(deers_ctx* ctx, int M, int N, int K, const float* a, long long lda, int a_mn, const float* b,
                    long long ldb, int b_mn, float* c, long long ldc, int epi, const float* r, long long ldr, float* aux);
// The same with the rows of A normalised on the way, C [M,N] = rmsnorm(A [M,K]) * B [K,N], all dense: what a block's pre-norms
// feed (launch_gemm_f32_norm).  inv (may be nullptr) receives the inverse norms.  Columns [0, rope_cols), heads of rope_d columns,
// may be rotated by position m % rope_t with the tables cosv, sinv [rope_t][rope_d / 2] (0 columns: none); *rotated tells whether
// they were.
struct GemmNorm {
    float eps;
    float* inv;
    const float* cosv; const float* sinv;
    int rope_cols, rope_d, rope_t;
};
int launch_gemm_f32_norm(deers_ctx* ctx, int M, int N, int K, const float* a, const float* b, float* c, int epi, float* aux, const GemmNorm& f,
                         bool* rotated);
// Products C_i [M_i,N_i] = A_i^T B_i with A_i [K,M_i], B_i [K,N_i], dense, in one launch.
constexpr int GEMM_GROUP_MAX = 4;
struct GemmTN { int M, N; const float* a; const float* b; float* c; };
int launch_gemm_f32_group(deers_ctx* ctx, int n, const GemmTN* t, int K);
bool gemm_f32_group_fits(deers_ctx* ctx, int n, const GemmTN* t, int K);
// RMSNorm (rmsnorm.cu)
int launch_rmsnorm_fwd(deers_ctx* ctx, long long rows, int C, double eps, const float* x, float* y, float* inv_norm);
int launch_rmsnorm_bwd(deers_ctx* ctx, long long rows, int C, const float* x, const float* inv_norm, const float* dy,
                       const float* add, float* dx, float* n_out = nullptr);
int launch_rmsnorm_split(deers_ctx* ctx, long long rows, int C, double eps, const float* x, float* inv_norm, void* hi, void* lo);
// embedding and cross-entropy (gpt_ops.cu)
int launch_embedding_fwd(deers_ctx* ctx, const float* weight, const long long* ids, long long n_ids, int C, long long V,
                         float* out);
int launch_embedding_bwd(deers_ctx* ctx, const float* dout, const long long* ids, long long n_ids, int C, long long V,
                         float* dweight, bool cleared = false);
int launch_cross_entropy_fwd(deers_ctx* ctx, const float* logits, long long ld, const long long* targets, long long rows,
                             long long V, float* lse, float* picked, float* loss);
int launch_cross_entropy_merge(deers_ctx* ctx, const float2* stats, int parts, const float* logits, long long ld, const long long* targets,
                               long long rows, long long V, float* lse, float* picked);
int launch_cross_entropy_rows(deers_ctx* ctx, const float* logits, long long ld, const long long* targets, long long rows, long long V, float* lse,
                              float* picked);
int launch_cross_entropy_loss(deers_ctx* ctx, const float* picked, long long rows, float* loss);
int launch_cross_entropy_bwd(deers_ctx* ctx, const float* logits, long long ld, const long long* targets, const float* lse,
                             long long rows, long long V, float upstream, float* dlogits, long long ldd);
// AdamW with the trainer's rule "no update when the gradient norm is not finite" (optim.cu).  said: what the caller wants to
// know of the step, written by the same launch.
struct StepSaid { const float* loss; float* loss_out; float* norm_out; };
int launch_adamw(deers_ctx* ctx, int n_tensors, const deers_optim_tensor* tensors, const deers_adamw_hyper* h,
                 const float* norm_dev, double max_norm, bool skip_nonfinite, const StepSaid& said = StepSaid{});
// f32-accurate tensor-core GEMM on split f16 operands (gemm_f16x3_sm100.cu) and the split writers
size_t gemm_f16x3_workspace_bytes(const deers_ctx* ctx, int M, int N, int K);
int launch_split_f16x3(deers_ctx* ctx, long long rows, int cols, const float* src, long long ld_src, float scale,
                       void* hi, void* lo, long long ld_dst);
int launch_gemm_f16x3(deers_ctx* ctx, int M, int N, int K, const void* a_hi, const void* a_lo, long long lda, int a_mn,
                      const void* b_hi, const void* b_lo, long long ldb, int b_mn, float* c, long long ldc, float out_scale,
                      void* workspace, size_t ws_bytes, float2* stats = nullptr, int* stat_parts = nullptr);
// (stats, stat_parts: with A in K and B in MN order the product may leave, per row and 32 columns, (maximum, sum of exponentials relative to
// it), [stat_parts][M]; 0 parts: it did not.  Room for 4 * ceil(N / 128) parts.)
int gemm_f16_pairs(deers_ctx* ctx, int* pairs);
int route_gemm_f16(deers_ctx* ctx, int M, int N, int K, deers_product_route* r);
int route_gemm_f16x3(deers_ctx* ctx, int M, int N, int K, int a_mn, int b_mn, int rows16, deers_product_route* r);
int launch_cross_entropy_bwd_split(deers_ctx* ctx, const float* logits, long long ld, const long long* targets,
                                   const float* lse, long long rows, long long V, float upstream, float scale, void* hi,
                                   void* lo, long long ldd);
