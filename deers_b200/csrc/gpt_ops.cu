// Embedding lookup and cross-entropy for the f32 GPT step: the ops around the transformer blocks that
// the reference builds from index_select / index_add (src/nn.rs:214-221, src/storage/cuda.rs:359-413)
// and from log_softmax + gather + sum (src/loss.rs:11-24, src/tensor.rs:408-425).
//
//   embedding_fwd   out[n, :] = weight[ids[n], :]
//   embedding_bwd   dweight = 0; dweight[ids[n], :] += dout[n, :] in token order.  The reference adds
//                   with atomics (scatter order undefined); here the first occurrence of a token id
//                   owns the row and adds the later occurrences in order, so the result is reproducible
//                   and equals the CPU backend's left-to-right sum.
//   cross_entropy   one block per row reads the logits once (running maximum / sum of exponentials),
//                   writes lse[row] and the picked log-probability (in the model these come from the head product's statistics
//                   per row and tile, merged in order); a one-block kernel adds the rows in a fixed order: loss = sum * (float)(-1/rows).
//   cross_entropy_bwd  dlogits = (onehot * g - softmax * g) * upstream, g = (float)(-1/rows): the chain
//                   gather backward -> log_softmax backward of src/ops.rs:210-214, 777-799, 1162-1175 in one
//                   element-wise pass (in place over the logits if asked).
// A token id or target outside [0, vocab) sets the context's error word (reported by deers_b200_sync as
// DEERS_ERR_KERNEL) and is skipped; nothing traps.
#include "common.cuh"

#include <cuda_fp16.h>

namespace {

__global__ void __launch_bounds__(256) embedding_fwd_kernel(const float* w, const long long* ids,
                                                            long long n_ids, int C, long long V, float* __restrict__ out,
                                                            int vec, unsigned int* err) {
    chain_begin();
    const int lane = threadIdx.x & 31;
    const long long n = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (n >= n_ids) return;
    const long long id = ids[n];
    float* o = out + n * C;
    if (id < 0 || id >= V) {
        if (lane == 0) atomicCAS(err, 0u, (unsigned)DEERS_KERR_GPT | 1u);
        for (int c = lane; c < C; c += 32) o[c] = 0.f;
        return;
    }
    const float* s = w + id * C;
    if (vec) {
        for (int c = lane; c < C / 4; c += 32) reinterpret_cast<float4*>(o)[c] = reinterpret_cast<const float4*>(s)[c];
    } else {
        for (int c = lane; c < C; c += 32) o[c] = s[c];
    }
}

// One block per token n.  The block whose token is the first occurrence of its id writes the row.
// What bounds it: latency, as the last kernel of a backward.  The ids are read once, several loads in flight, beside the token's own
// row; later occurrences are compacted by ballots into an ordered list whose rows are then loaded eight at a time.  (A walk over the flags
// of 256 tokens cost 4 us wherever a token repeats: 1024 tokens of 50257, C 192 13.5 us, 231 of 5003 12 us; now 5.1 and 3.3,
// traced in the step.)
__global__ void __launch_bounds__(256) embedding_bwd_kernel(const float* dout, const long long* ids, long long n_ids, int C,
                                                            long long V, float* __restrict__ dw) {
    chain_wait();
    constexpr int CH = 4;                                              // chunks of 256 ids looked at together
    __shared__ unsigned s_mask[CH * 8];
    __shared__ int s_list[CH * 256];
    const long long n = blockIdx.x;
    const long long id = ids[n];
    if (id < 0 || id >= V) return;                                     // reported by the forward
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // 8 channels per thread and sweep
    float acc[8];
    auto own = [&](int c0) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int c = c0 + k * 256 + threadIdx.x;
            acc[k] = c < C ? dout[n * C + c] : 0.f;
        }
    };
    own(0);
    int dup = 0, later = 0;
    for (long long j0 = 0; j0 < n_ids; j0 += CH * 256) {
        long long v[CH];
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            const long long j = j0 + i * 256 + threadIdx.x;
            v[i] = j < n_ids ? ids[j] : -1;
        }
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            const long long j = j0 + i * 256 + threadIdx.x;
            dup |= v[i] == id && j < n;
            later |= v[i] == id && j > n;
        }
    }
    if (__syncthreads_or(dup)) return;
    const bool more = __syncthreads_or(later);
    for (int c0 = 0; c0 < C; c0 += 256 * 8) {
        if (c0) own(c0);
        for (long long j0 = more ? n + 1 : n_ids; j0 < n_ids; j0 += CH * 256) {
            bool f[CH];
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                const long long j = j0 + i * 256 + threadIdx.x;
                f[i] = j < n_ids && ids[j] == id;
            }
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                const unsigned b = __ballot_sync(0xffffffffu, f[i]);
                if (lane == 0) s_mask[i * 8 + warp] = b;
            }
            __syncthreads();
            int total = 0;
#pragma unroll
            for (int i = 0; i < CH; ++i) {                             // place of the thread's tokens: those before them, in token order
                int before = total;
#pragma unroll
                for (int w = 0; w < 8; ++w) {
                    const int cnt = __popc(s_mask[i * 8 + w]);
                    if (w < warp) before += cnt;
                    total += cnt;
                }
                if (f[i]) s_list[before + __popc(s_mask[i * 8 + warp] & ((1u << lane) - 1u))] = (int)(j0 + i * 256 + threadIdx.x - n);
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int c = c0 + k * 256 + threadIdx.x;
                if (c >= C) break;
                const float* col = dout + n * C + c;
                int t = 0;
                for (; t + 8 <= total; t += 8) {
                    float v[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[e] = col[(long long)s_list[t + e] * C];
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[k] += v[e];
                }
                for (; t < total; ++t) acc[k] += col[(long long)s_list[t] * C];
            }
            __syncthreads();
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int c = c0 + k * 256 + threadIdx.x;
            if (c < C) dw[id * C + c] = acc[k];
        }
    }
}

// Row logsumexp + picked log-probability (src/storage/cpu.rs:759-770 computes the maximum first and then the
// sum of expf(x - max); the same value up to f32 rounding of a different summation order).
// Merges two (maximum, sum of exponentials relative to it) pairs.
__device__ __forceinline__ void lse_merge(float& m, float& s, float m2, float s2) {
    const float M = fmaxf(m, m2);
    if (M == -INFINITY) { s = 0.f; return; }                      // both parts empty
    s = s * expf(m - M) + s2 * expf(m2 - M);
    m = M;
}

// One pass over the row: every thread keeps a running maximum and the sum of exponentials relative to it (the
// sum is rescaled when the maximum grows), four values at a time when the row is 16-byte aligned; the 256 pairs
// are merged at the end.  A two-pass version (maximum, then sum) read the 206 MB of logits twice from DRAM.
__global__ void __launch_bounds__(256) cross_entropy_fwd_kernel(const float* logits, long long ld, const long long* targets, long long V,
                                                                float* __restrict__ lse, float* __restrict__ picked,
                                                                unsigned int* err) {
    chain_wait();
    __shared__ float red_m[8], red_s[8];
    const long long row = blockIdx.x;
    const float* x = logits + row * ld;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float m = -INFINITY, s = 0.f;
    const bool vec = (((uintptr_t)x) & 15u) == 0;
    const long long V4 = vec ? V / 4 : 0;
    for (long long j = threadIdx.x; j < V4; j += 256) {
        const float4 v = *reinterpret_cast<const float4*>(x + 4 * j);
        const float vm = fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w));
        if (vm > m) { s *= expf(m - vm); m = vm; }                // m = -inf at first: s = 0 * 0
        s += expf(v.x - m) + expf(v.y - m) + expf(v.z - m) + expf(v.w - m);
    }
    for (long long j = 4 * V4 + threadIdx.x; j < V; j += 256) {
        const float v = x[j];
        if (v > m) { s *= expf(m - v); m = v; }
        s += expf(v - m);
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1)
        lse_merge(m, s, __shfl_xor_sync(0xffffffffu, m, off), __shfl_xor_sync(0xffffffffu, s, off));
    if (lane == 0) { red_m[warp] = m; red_s[warp] = s; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) lse_merge(m, s, red_m[w], red_s[w]);
        const float l = logf(s) + m;
        lse[row] = l;
        const long long t = targets[row];
        if (t < 0 || t >= V) {
            atomicCAS(err, 0u, (unsigned)DEERS_KERR_GPT | 2u);
            picked[row] = 0.f;
        } else {
            picked[row] = x[t] - l;
        }
    }
}

// The same rows from what the head product has left of them: `parts` pairs (maximum, sum of exponentials relative to it) per row, [parts][rows].
// A block takes eight rows, 128 threads each, every thread eight loads at a time.  1024 rows of 1572 parts 7 us behind the product where the
// pass over the 206 MB of logits takes 42 (with 32 threads a row 18).
__global__ void __launch_bounds__(1024) cross_entropy_merge_kernel(const float2* stats, int parts, const float* logits, long long ld,
                                                                   const long long* targets,
                                                                   long long rows, long long V, float* __restrict__ lse, float* __restrict__ picked,
                                                                   unsigned int* err) {
    chain_wait();
    __shared__ float red_m[32][8], red_s[32][8];
    const int r = threadIdx.x & 7, seg = threadIdx.x >> 3, warp = threadIdx.x >> 5;
    const long long row = (long long)blockIdx.x * 8 + r;
    float m = -INFINITY, s = 0.f;
    if (row < rows) {
        for (int p0 = seg; p0 < parts; p0 += 8 * 128) {
            float2 v[8];
            float M = m;
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = p0 + q * 128 < parts ? stats[(long long)(p0 + q * 128) * rows + row] : make_float2(-INFINITY, 0.f);
#pragma unroll
            for (int q = 0; q < 8; ++q) M = fmaxf(M, v[q].x);
            const float ref = M == -INFINITY ? 0.f : M;               // (all empty so far: sums of zeros)
            s *= expf(m - ref);
#pragma unroll
            for (int q = 0; q < 8; ++q) s += v[q].y * expf(v[q].x - ref);
            m = M;
        }
    }
    chain_next();
    // lanes r, r + 8, r + 16, r + 24 of a warp, then the warps
#pragma unroll
    for (int off = 8; off <= 16; off *= 2) lse_merge(m, s, __shfl_xor_sync(0xffffffffu, m, off), __shfl_xor_sync(0xffffffffu, s, off));
    if ((threadIdx.x & 31) < 8) { red_m[warp][r] = m; red_s[warp][r] = s; }
    __syncthreads();
    if (warp) return;
    m = red_m[seg][r]; s = red_s[seg][r];
    for (int w = 4; w < 32; w += 4) lse_merge(m, s, red_m[w + seg][r], red_s[w + seg][r]);
#pragma unroll
    for (int off = 8; off <= 16; off *= 2) lse_merge(m, s, __shfl_xor_sync(0xffffffffu, m, off), __shfl_xor_sync(0xffffffffu, s, off));
    if (row >= rows || seg) return;
    const float l = logf(s) + m;
    lse[row] = l;
    const long long t = targets[row];
    if (t < 0 || t >= V) {
        atomicCAS(err, 0u, (unsigned)DEERS_KERR_GPT | 2u);
        picked[row] = 0.f;
    } else {
        picked[row] = logits[row * ld + t] - l;
    }
}

__global__ void __launch_bounds__(1024) cross_entropy_loss_kernel(const float* picked, long long rows,
                                                                  float neg_inv_rows, float* __restrict__ loss) {
    chain_wait();
    __shared__ float red[32];
    float s = 0.f;
    for (long long j = threadIdx.x; j < rows; j += 1024) s += picked[j];
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        s = red[threadIdx.x];
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (threadIdx.x == 0) loss[0] = s * neg_inv_rows;
    }
}

__global__ void __launch_bounds__(256) cross_entropy_bwd_kernel(const float* logits, long long ld, const long long* targets, const float* lse,
                                                                long long V, float g, float upstream, float* dlogits,
                                                                long long ldd, int vec) {         // dlogits may be logits
    chain_wait();
    const long long row = blockIdx.y;
    const float* x = logits + row * ld;
    float* d = dlogits + row * ldd;
    const float l = lse[row];
    const long long t = targets[row];
    const long long stride = (long long)gridDim.x * 256;
    if (vec) {
        for (long long q = (long long)blockIdx.x * 256 + threadIdx.x; q * 4 < V; q += stride) {
            const long long j = q * 4;
            if (j + 4 <= V) {
                const float4 v = *reinterpret_cast<const float4*>(x + j);
                float o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float p = expf(o[e] - l);
                    const float gj = (j + e == t) ? g : 0.f;
                    o[e] = __fmul_rn(__fsub_rn(gj, __fmul_rn(p, g)), upstream);
                }
                *reinterpret_cast<float4*>(d + j) = make_float4(o[0], o[1], o[2], o[3]);
            } else {
                for (long long e = j; e < V; ++e) {
                    const float p = expf(x[e] - l);
                    const float gj = (e == t) ? g : 0.f;
                    d[e] = __fmul_rn(__fsub_rn(gj, __fmul_rn(p, g)), upstream);
                }
            }
        }
    } else {
        for (long long j0 = (long long)blockIdx.x * 256 + threadIdx.x; j0 < V; j0 += 4 * stride) {
            float v[4];                                               // four loads in flight
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = j0 + e * stride < V ? x[j0 + e * stride] : 0.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const long long j = j0 + e * stride;
                const float p = expf(v[e] - l);
                const float gj = (j == t) ? g : 0.f;
                if (j < V) d[j] = __fmul_rn(__fsub_rn(gj, __fmul_rn(p, g)), upstream);
            }
        }
    }
}

// The same gradient written as the f16 pair the tensor-core head products read (gemm_f16x3_sm100.cu):
// v = dlogit * scale, hi = f16(v), lo = f16((v - hi) * 2^11).  |dlogit| <= 1/rows, so scale = rows * 4096 keeps
// hi within +-4096 and the smallest probabilities that matter well inside the f16 range.
__global__ void __launch_bounds__(256) cross_entropy_bwd_split_kernel(const float* logits, long long ld, const long long* targets,
                                                                      const float* lse, long long V, float g,
                                                                      float upstream, float scale, __half* __restrict__ hi,
                                                                      __half* __restrict__ lo, long long ldd) {
    chain_wait();
    const long long row = blockIdx.y;
    const float* x = logits + row * ld;
    __half* dh = hi + row * ldd;
    __half* dl = lo + row * ldd;
    const float l = lse[row];
    const long long t = targets[row];
    const long long stride = (long long)gridDim.x * 256;
    const bool vec = (ld % 4 == 0) && (ldd % 8 == 0) && ((((uintptr_t)logits) & 15u) == 0) &&
                     ((((uintptr_t)hi | (uintptr_t)lo) & 15u) == 0);
    for (long long q = (long long)blockIdx.x * 256 + threadIdx.x; q * 8 < V; q += stride) {
        const long long j = q * 8;
        float o[8];
        if (vec && j + 8 <= V) {
            const float4 a = *reinterpret_cast<const float4*>(x + j), b = *reinterpret_cast<const float4*>(x + j + 4);
            o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] = (j + e < V) ? x[j + e] : -INFINITY;
        }
        __half h8[8], l8[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float pr = expf(o[e] - l);
            const float gj = (j + e == t) ? g : 0.f;
            const float d = __fmul_rn(__fsub_rn(gj, __fmul_rn(pr, g)), upstream) * scale;
            h8[e] = __float2half_rn(d);
            l8[e] = __float2half_rn((d - __half2float(h8[e])) * 2048.0f);
        }
        if (vec && j + 8 <= V) {
            *reinterpret_cast<uint4*>(dh + j) = *reinterpret_cast<const uint4*>(h8);
            *reinterpret_cast<uint4*>(dl + j) = *reinterpret_cast<const uint4*>(l8);
        } else {
            for (int e = 0; e < 8 && j + e < V; ++e) { dh[j + e] = h8[e]; dl[j + e] = l8[e]; }
        }
    }
}

}  // namespace

int launch_cross_entropy_bwd_split(deers_ctx* ctx, const float* logits, long long ld, const long long* targets,
                                   const float* lse, long long rows, long long V, float upstream, float scale, void* hi,
                                   void* lo, long long ldd) {
    long long per_row = (V / 8 + 255) / 256;
    if (per_row < 1) per_row = 1;
    if (per_row > 64) per_row = 64;
    const dim3 grid((unsigned)per_row, (unsigned)rows);
    {
        KernelTimerScope ts(ctx, DEERS_K_GPT);
        DEERS_CUDA_TRY(ctx, launch_chained(ctx, cross_entropy_bwd_split_kernel, grid, 256, 0, 1, logits, ld, targets, lse, V, (float)(-1.0 / (double)rows),
                                                                      upstream, scale, (__half*)hi, (__half*)lo, ldd));
    }
    ctx->launches += 1;
    DEERS_CUDA_TRY(ctx, cudaGetLastError());
    return DEERS_OK;
}

int launch_embedding_fwd(deers_ctx* ctx, const float* weight, const long long* ids, long long n_ids, int C, long long V,
                         float* out) {
    if (n_ids == 0) return DEERS_OK;
    const int vec = C % 4 == 0 && (((uintptr_t)weight | (uintptr_t)out) & 15u) == 0;
    {
        KernelTimerScope ts(ctx, DEERS_K_GPT);
        DEERS_CUDA_TRY(ctx, launch_chained(ctx, embedding_fwd_kernel, (unsigned)((n_ids + 7) / 8), 256, 0, 1, weight, ids, n_ids, C, V, out, vec,
                                                                                  ctx->dev_err));
    }
    ctx->launches += 1;
    DEERS_CUDA_TRY(ctx, cudaGetLastError());
    return DEERS_OK;
}

int launch_embedding_bwd(deers_ctx* ctx, const float* dout, const long long* ids, long long n_ids, int C, long long V,
                         float* dweight, bool cleared) {
    if (!cleared) DEERS_CUDA_TRY(ctx, cudaMemsetAsync(dweight, 0, (size_t)V * C * sizeof(float), ctx->stream));
    if (n_ids == 0) return DEERS_OK;
    {
        KernelTimerScope ts(ctx, DEERS_K_GPT);
        DEERS_CUDA_TRY(ctx, launch_chained(ctx, embedding_bwd_kernel, (unsigned)n_ids, 256, 0, 1, dout, ids, n_ids, C, V, dweight));
    }
    ctx->launches += 1;
    DEERS_CUDA_TRY(ctx, cudaGetLastError());
    return DEERS_OK;
}

int launch_cross_entropy_merge(deers_ctx* ctx, const float2* stats, int parts, const float* logits, long long ld, const long long* targets,
                               long long rows, long long V, float* lse, float* picked) {
    {
        KernelTimerScope ts(ctx, DEERS_K_GPT);
        DEERS_CUDA_TRY(ctx, launch_chained(ctx, cross_entropy_merge_kernel, (unsigned)((rows + 7) / 8), 1024, 0, 1, stats, parts, logits, ld, targets,
                                           rows, V, lse, picked, ctx->dev_err));
    }
    ctx->launches += 1;
    return DEERS_OK;
}

int launch_cross_entropy_rows(deers_ctx* ctx, const float* logits, long long ld, const long long* targets, long long rows, long long V, float* lse,
                              float* picked) {
    {
        KernelTimerScope ts(ctx, DEERS_K_GPT);
        DEERS_CUDA_TRY(ctx, launch_chained(ctx, cross_entropy_fwd_kernel, (unsigned)rows, 256, 0, 1, logits, ld, targets, V, lse, picked, ctx->dev_err));
    }
    ctx->launches += 1;
    return DEERS_OK;
}

int launch_cross_entropy_loss(deers_ctx* ctx, const float* picked, long long rows, float* loss) {
    {
        KernelTimerScope ts(ctx, DEERS_K_GPT);
        DEERS_CUDA_TRY(ctx, launch_chained(ctx, cross_entropy_loss_kernel, 1, 1024, 0, 1, picked, rows, (float)(-1.0 / (double)rows), loss));
    }
    ctx->launches += 1;
    return DEERS_OK;
}

int launch_cross_entropy_fwd(deers_ctx* ctx, const float* logits, long long ld, const long long* targets, long long rows,
                             long long V, float* lse, float* picked, float* loss) {
    const int rc = launch_cross_entropy_rows(ctx, logits, ld, targets, rows, V, lse, picked);
    return rc ? rc : launch_cross_entropy_loss(ctx, picked, rows, loss);
}

int launch_cross_entropy_bwd(deers_ctx* ctx, const float* logits, long long ld, const long long* targets, const float* lse,
                             long long rows, long long V, float upstream, float* dlogits, long long ldd) {
    const int vec = ld % 4 == 0 && ldd % 4 == 0 && (((uintptr_t)logits | (uintptr_t)dlogits) & 15u) == 0;
    long long per_row = (V / 4 + 255) / 256;
    if (per_row < 1) per_row = 1;
    if (per_row > 64) per_row = 64;
    const dim3 grid((unsigned)per_row, (unsigned)rows);
    {
        KernelTimerScope ts(ctx, DEERS_K_GPT);
        DEERS_CUDA_TRY(ctx, launch_chained(ctx, cross_entropy_bwd_kernel, grid, 256, 0, 1, logits, ld, targets, lse, V, (float)(-1.0 / (double)rows),
                                                                upstream, dlogits, ldd, vec));
    }
    ctx->launches += 1;
    DEERS_CUDA_TRY(ctx, cudaGetLastError());
    return DEERS_OK;
}

extern "C" int deers_b200_embedding_fwd(deers_ctx* ctx, const float* weight, const int64_t* ids, int64_t n_ids, int32_t C,
                                        int64_t vocab, float* out) {
    if (!ctx || !weight || !ids || !out) return DEERS_ERR_NULL;
    if (n_ids < 0 || C < 1 || vocab < 1 || n_ids > 0x7fffffffLL) return DEERS_ERR_SHAPE;
    if ((((uintptr_t)weight | (uintptr_t)out) & 3u) || ((uintptr_t)ids & 7u)) return DEERS_ERR_LAYOUT;
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    return launch_embedding_fwd(ctx, weight, (const long long*)ids, n_ids, C, vocab, out);
}

extern "C" int deers_b200_embedding_bwd(deers_ctx* ctx, const float* dout, const int64_t* ids, int64_t n_ids, int32_t C,
                                        int64_t vocab, float* dweight) {
    if (!ctx || !dout || !ids || !dweight) return DEERS_ERR_NULL;
    if (n_ids < 0 || C < 1 || vocab < 1 || n_ids > 0x7fffffffLL) return DEERS_ERR_SHAPE;
    if ((((uintptr_t)dout | (uintptr_t)dweight) & 3u) || ((uintptr_t)ids & 7u)) return DEERS_ERR_LAYOUT;
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    return launch_embedding_bwd(ctx, dout, (const long long*)ids, n_ids, C, vocab, dweight);
}

extern "C" size_t deers_b200_cross_entropy_scratch_bytes(int64_t rows) {
    return rows > 0 ? (size_t)rows * sizeof(float) : 0;
}

extern "C" int deers_b200_cross_entropy_fwd(deers_ctx* ctx, int64_t rows, int64_t vocab, const float* logits, int64_t ld,
                                            const int64_t* targets, float* lse, float* loss, void* scratch,
                                            size_t scratch_bytes) {
    if (!ctx || !logits || !targets || !lse || !loss) return DEERS_ERR_NULL;
    if (rows < 1 || vocab < 1 || rows > 0x7fffffffLL) return DEERS_ERR_SHAPE;
    if (ld < vocab || (((uintptr_t)logits | (uintptr_t)lse | (uintptr_t)loss) & 3u) || ((uintptr_t)targets & 7u))
        return DEERS_ERR_LAYOUT;
    if (!scratch || scratch_bytes < deers_b200_cross_entropy_scratch_bytes(rows) || ((uintptr_t)scratch & 3u))
        return DEERS_ERR_WORKSPACE;
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    return launch_cross_entropy_fwd(ctx, logits, ld, (const long long*)targets, rows, vocab, lse, (float*)scratch, loss);
}

extern "C" int deers_b200_cross_entropy_bwd(deers_ctx* ctx, int64_t rows, int64_t vocab, const float* logits, int64_t ld,
                                            const int64_t* targets, const float* lse, float upstream, float* dlogits,
                                            int64_t ld_dlogits) {
    if (!ctx || !logits || !targets || !lse || !dlogits) return DEERS_ERR_NULL;
    if (rows < 1 || vocab < 1 || rows > 65535) return DEERS_ERR_SHAPE;
    if (ld < vocab || ld_dlogits < vocab || (((uintptr_t)logits | (uintptr_t)lse | (uintptr_t)dlogits) & 3u) ||
        ((uintptr_t)targets & 7u))
        return DEERS_ERR_LAYOUT;
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    return launch_cross_entropy_bwd(ctx, logits, ld, (const long long*)targets, lse, rows, vocab, upstream, dlogits,
                                    ld_dlogits);
}
