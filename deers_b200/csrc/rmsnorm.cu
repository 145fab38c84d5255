// RMSNorm forward and backward, f32, one pass each.
//
// The reference evaluates `x * (mean(x*x, last axis) + eps)^-0.5` (RMSNorm::forward,
// src/nn.rs:244-251) as six graph ops (multiply, sum, scalar multiply, scalar add, scalar power,
// broadcast multiply) and its backward as the autograd of those (src/ops.rs:210-214, 638-643,
// 675-679, 777-799): about fifteen launches and ten row- or tensor-sized temporaries per call, twice
// per transformer block plus once before the head.  Here a warp owns a row: it reads the row once,
// reduces x*x with shuffles, and writes y (and the row's inverse norm, kept for the backward like the
// row lse of the attention op); the backward reads x and dy once and writes dx:
//     inv = 1 / sqrt(sum(x*x) / n + eps)            y  = x * inv
//     dx  = dy * inv - x * (sum(dy * x) * inv^3 / n)
// Rows of up to 1024 elements are owned by a warp, up to 8192 by a block (both keep the row in registers: one
// pass over HBM); longer rows take two passes of 16-byte loads.
// HBM-bound: 8 bytes per element forward, 12 backward.  Sums are f32 shuffle trees (the reference
// sums left to right), so parity is to rounding, not to the bit.
#include <cuda_fp16.h>

#include "common.cuh"

namespace {

constexpr int RN_MAXV = 8;      // float4 pieces per lane: rows of up to 32 * 8 * 4 = 1024 elements stay in registers

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// Four elements of y as the f16 pair the split-f16 products read (hi = f16(v), lo = f16((v - hi) * 2^11); gemm_f16x3_sm100.cu).
__device__ __forceinline__ void put_pair(__half* hi, __half* lo, long long at, const float4& v) {
    const float x[4] = {v.x, v.y, v.z, v.w};
    __half h[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        h[e] = __float2half_rn(x[e]);
        l[e] = __float2half_rn((x[e] - __half2float(h[e])) * 2048.0f);
    }
    *reinterpret_cast<uint2*>(hi + at) = *reinterpret_cast<const uint2*>(h);
    *reinterpret_cast<uint2*>(lo + at) = *reinterpret_cast<const uint2*>(l);
}

// BWD = false: y = x * inv, inv_out[row] = inv (PAIR: y leaves as the f16 pair hi, lo, rows dense, instead of out).
// BWD = true: dx from x, dy and the saved inv_in; n_out (may be nullptr) receives y again for the weight gradient.
// NV: 16-byte pieces of a lane.  Of rows of up to 256 the backward requests everything at once, the residual and the norm too: behind the sum
// they were two more trips to L2 (22 M parameters, 1024 rows of 192, 13 a step: 4 steps and a forward 5057 -> 4996 us; 3 layers,
// 231 rows 1230 -> 1203).  Longer rows do not have the registers.
template <bool BWD, bool VEC, bool VEC2 = false, bool PAIR = false, int NV = RN_MAXV>
__global__ void __launch_bounds__(256) rmsnorm_kernel(const float* x, const float* dy, const float* add, const float* inv_in, float* __restrict__ out,
                                                      float* __restrict__ inv_out, long long rows, int C, float eps,
                                                      float inv_n, float* __restrict__ n_out, __half* __restrict__ hi,
                                                      __half* __restrict__ lo) {
    if (!BWD) chain_next();                                     // (backward: weight gradients run beside it, leave them the room; short rows below)
    chain_wait();
    const int lane = threadIdx.x & 31;
    const long long warp = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    const long long nwarps = (long long)gridDim.x * 8;
    for (long long row = warp; row < rows; row += nwarps) {
        const float* xr = x + row * C;
        float* orow = out + row * C;
        if (VEC) {
            const int nv = C / 4;                               // float4 pieces in the row (<= 32 * NV)
            float4 xv[NV], gv[NV], av[NV];
            constexpr bool EARLY = BWD && NV <= 2;
            float acc = 0.f, early_inv = 0.f;
            if (EARLY) early_inv = inv_in[row];
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const int p = lane + 32 * i;
                if (EARLY && add && p < nv) av[i] = reinterpret_cast<const float4*>(add + row * C)[p];
            }
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const int p = lane + 32 * i;
                if (p < nv) {
                    xv[i] = reinterpret_cast<const float4*>(xr)[p];
                    if (BWD) {
                        gv[i] = reinterpret_cast<const float4*>(dy + row * C)[p];
                        acc += xv[i].x * gv[i].x + xv[i].y * gv[i].y + xv[i].z * gv[i].z + xv[i].w * gv[i].w;
                    } else {
                        acc += xv[i].x * xv[i].x + xv[i].y * xv[i].y + xv[i].z * xv[i].z + xv[i].w * xv[i].w;
                    }
                }
            }
            if (EARLY && row + nwarps >= rows) chain_next();       // (a step of 3 layers, 231 rows, four of them and a forward: 1203 -> 1191 us)
            acc = warp_sum(acc);
            float inv, k = 0.f;
            if (BWD) {
                inv = EARLY ? early_inv : inv_in[row];
                k = acc * inv * inv * inv * inv_n;
            } else {
                inv = 1.0f / sqrtf(acc * inv_n + eps);
                if (lane == 0) inv_out[row] = inv;
            }
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const int p = lane + 32 * i;
                if (p < nv) {
                    float4 o;
                    if (BWD) {
                        o.x = gv[i].x * inv - xv[i].x * k; o.y = gv[i].y * inv - xv[i].y * k;
                        o.z = gv[i].z * inv - xv[i].z * k; o.w = gv[i].w * inv - xv[i].w * k;
                        if (add) {
                            const float4 r = EARLY ? av[i] : reinterpret_cast<const float4*>(add + row * C)[p];
                            o.x = r.x + o.x; o.y = r.y + o.y; o.z = r.z + o.z; o.w = r.w + o.w;
                        }
                        if (n_out) reinterpret_cast<float4*>(n_out + row * C)[p] = make_float4(xv[i].x * inv, xv[i].y * inv, xv[i].z * inv, xv[i].w * inv);
                    } else {
                        o.x = xv[i].x * inv; o.y = xv[i].y * inv; o.z = xv[i].z * inv; o.w = xv[i].w * inv;
                    }
                    if constexpr (PAIR) put_pair(hi, lo, row * C + 4 * p, o);
                    else reinterpret_cast<float4*>(orow)[p] = o;
                }
            }
        } else if (VEC2) {                                      // long aligned rows: two passes of 16-byte loads
            const int nv = C / 4;
            const float4* x4 = reinterpret_cast<const float4*>(xr);
            const float4* g4 = BWD ? reinterpret_cast<const float4*>(dy + row * C) : nullptr;
            float acc = 0.f;
            constexpr int U = BWD ? 8 : 16;                     // pieces of a lane in flight
            for (int p0 = lane; p0 < nv; p0 += 32 * U) {
                float4 a[U], b[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int p = p0 + 32 * u;
                    a[u] = b[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (p < nv) a[u] = x4[p];
                    if (BWD && p < nv) b[u] = g4[p];
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const float4 c = BWD ? b[u] : a[u];
                    acc += a[u].x * c.x + a[u].y * c.y + a[u].z * c.z + a[u].w * c.w;
                }
            }
            acc = warp_sum(acc);
            float inv, k = 0.f;
            if (BWD) {
                inv = inv_in[row];
                k = acc * inv * inv * inv * inv_n;
            } else {
                inv = 1.0f / sqrtf(acc * inv_n + eps);
                if (lane == 0) inv_out[row] = inv;
            }
            for (int p0 = lane; p0 < nv; p0 += 32 * U) {        // the row (<= a few KB per lane group) is still in L1 / L2
                float4 a[U], b[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int p = p0 + 32 * u;
                    if (p < nv) a[u] = x4[p];
                    if (BWD && p < nv) b[u] = g4[p];
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int p = p0 + 32 * u;
                    if (p >= nv) break;
                    float4 o;
                    if (BWD) {
                        o.x = b[u].x * inv - a[u].x * k; o.y = b[u].y * inv - a[u].y * k;
                        o.z = b[u].z * inv - a[u].z * k; o.w = b[u].w * inv - a[u].w * k;
                        if (add) {
                            const float4 r = reinterpret_cast<const float4*>(add + row * C)[p];
                            o.x = r.x + o.x; o.y = r.y + o.y; o.z = r.z + o.z; o.w = r.w + o.w;
                        }
                        if (n_out) reinterpret_cast<float4*>(n_out + row * C)[p] = make_float4(a[u].x * inv, a[u].y * inv, a[u].z * inv, a[u].w * inv);
                    } else {
                        o.x = a[u].x * inv; o.y = a[u].y * inv; o.z = a[u].z * inv; o.w = a[u].w * inv;
                    }
                    reinterpret_cast<float4*>(orow)[p] = o;
                }
            }
        } else {                                                // any C, any alignment: two passes over the row
            const float* gr = BWD ? dy + row * C : nullptr;
            float acc = 0.f;
            for (int c = lane; c < C; c += 32) acc += BWD ? xr[c] * gr[c] : xr[c] * xr[c];
            acc = warp_sum(acc);
            float inv, k = 0.f;
            if (BWD) {
                inv = inv_in[row];
                k = acc * inv * inv * inv * inv_n;
            } else {
                inv = 1.0f / sqrtf(acc * inv_n + eps);
                if (lane == 0) inv_out[row] = inv;
            }
            for (int c = lane; c < C; c += 32) {
                float o = BWD ? gr[c] * inv - xr[c] * k : xr[c] * inv;
                if (BWD && add) o = add[row * C + c] + o;
                if (BWD && n_out) n_out[row * C + c] = xr[c] * inv;
                orow[c] = o;
            }
        }
    }
}

// Rows of 1025 .. 8192 elements: a whole block owns a row, which still stays in registers (one pass over HBM).
template <bool BWD, bool PAIR = false>
__global__ void __launch_bounds__(256) rmsnorm_block_kernel(const float* x, const float* dy, const float* add, const float* inv_in, float* __restrict__ out,
                                                            float* __restrict__ inv_out, long long rows, int C, float eps,
                                                            float inv_n, float* __restrict__ n_out, __half* __restrict__ hi,
                                                            __half* __restrict__ lo) {
    if (!BWD) chain_next();                                     // (backward: weight gradients run beside it, leave them the room)
    chain_wait();
    __shared__ float part[8];
    const int nv = C / 4;                                       // <= 256 * RN_MAXV
    for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
        const float4* x4 = reinterpret_cast<const float4*>(x + row * C);
        const float4* g4 = BWD ? reinterpret_cast<const float4*>(dy + row * C) : nullptr;
        float4 xv[RN_MAXV], gv[RN_MAXV];
        float acc = 0.f;
#pragma unroll
        for (int i = 0; i < RN_MAXV; ++i) {
            const int p = threadIdx.x + 256 * i;
            if (p < nv) {
                xv[i] = x4[p];
                if (BWD) {
                    gv[i] = g4[p];
                    acc += xv[i].x * gv[i].x + xv[i].y * gv[i].y + xv[i].z * gv[i].z + xv[i].w * gv[i].w;
                } else {
                    acc += xv[i].x * xv[i].x + xv[i].y * xv[i].y + xv[i].z * xv[i].z + xv[i].w * xv[i].w;
                }
            }
        }
        acc = warp_sum(acc);
        __syncthreads();                                        // part[] of the previous row has been read
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
        __syncthreads();
        float tot = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) tot += part[w];
        float inv, k = 0.f;
        if (BWD) {
            inv = inv_in[row];
            k = tot * inv * inv * inv * inv_n;
        } else {
            inv = 1.0f / sqrtf(tot * inv_n + eps);
            if (threadIdx.x == 0) inv_out[row] = inv;
        }
        float4* o4 = reinterpret_cast<float4*>(out + row * C);
#pragma unroll
        for (int i = 0; i < RN_MAXV; ++i) {
            const int p = threadIdx.x + 256 * i;
            if (p < nv) {
                float4 o;
                if (BWD) {
                    o.x = gv[i].x * inv - xv[i].x * k; o.y = gv[i].y * inv - xv[i].y * k;
                    o.z = gv[i].z * inv - xv[i].z * k; o.w = gv[i].w * inv - xv[i].w * k;
                    if (add) {
                        const float4 r = reinterpret_cast<const float4*>(add + row * C)[p];
                        o.x = r.x + o.x; o.y = r.y + o.y; o.z = r.z + o.z; o.w = r.w + o.w;
                    }
                    if (n_out) reinterpret_cast<float4*>(n_out + row * C)[p] = make_float4(xv[i].x * inv, xv[i].y * inv, xv[i].z * inv, xv[i].w * inv);
                } else {
                    o.x = xv[i].x * inv; o.y = xv[i].y * inv; o.z = xv[i].z * inv; o.w = xv[i].w * inv;
                }
                if constexpr (PAIR) put_pair(hi, lo, row * C + 4 * p, o);
                else o4[p] = o;
            }
        }
    }
}

template <bool BWD>
int rms_launch(deers_ctx* ctx, long long rows, int C, float eps, const float* x, const float* dy, const float* inv_in, float* out, float* inv_out,
               const float* add = nullptr, float* n_out = nullptr) {
    if (rows == 0) return DEERS_OK;
    uintptr_t bits = (uintptr_t)x | (uintptr_t)out | (BWD ? (uintptr_t)dy : 0) | (uintptr_t)add | (uintptr_t)n_out;
    const bool aligned = (C % 4) == 0 && (bits & 15u) == 0;
    const bool vec = aligned && C <= 32 * RN_MAXV * 4;
    const long long want = (rows + 7) / 8;
    const long long cap = 16LL * ctx->sm_count;
    const unsigned grid = (unsigned)(want < cap ? want : cap);
    const float inv_n = (float)(1.0 / (double)C);               // mean = sum * (1/n as f64 -> f32), src/tensor.rs:461-465
    const auto launch = [&](auto kernel, unsigned blocks) -> int {
        KernelTimerScope ts(ctx, DEERS_K_NORM);
        DEERS_CUDA_TRY(ctx, launch_chained(ctx, kernel, blocks, 256, 0, 1, x, dy, add, inv_in, out, inv_out, rows, C, eps, inv_n, n_out, nullptr, nullptr));
        return DEERS_OK;
    };
    const int rc = BWD && vec && C <= 256              ? launch(rmsnorm_kernel<BWD, true, false, false, BWD ? 2 : RN_MAXV>, grid)
                 : vec                                 ? launch(rmsnorm_kernel<BWD, true>, grid)
                 : aligned && C <= 256 * RN_MAXV * 4   ? launch(rmsnorm_block_kernel<BWD>, (unsigned)(rows < cap ? rows : cap))
                 : aligned                             ? launch(rmsnorm_kernel<BWD, false, true>, grid)
                                                       : launch(rmsnorm_kernel<BWD, false>, grid);
    if (rc) return rc;
    ctx->launches += 1;
    DEERS_CUDA_TRY(ctx, cudaGetLastError());
    return DEERS_OK;
}

int rms_check(const deers_ctx* ctx, long long rows, int C, const void* a, const void* b, const void* c, const void* d) {
    if (!ctx || !a || !b || !c || !d) return DEERS_ERR_NULL;
    if (rows < 0 || C < 1) return DEERS_ERR_SHAPE;
    if (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)d) & 3u) return DEERS_ERR_LAYOUT;
    return DEERS_OK;
}

}  // namespace

extern "C" int deers_b200_rmsnorm_fwd(deers_ctx* ctx, int64_t rows, int32_t C, double eps, const float* x, float* y,
                                      float* inv_norm) {
    int rc = rms_check(ctx, rows, C, x, y, inv_norm, x);
    if (rc) return rc;
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    return rms_launch<false>(ctx, rows, C, (float)eps, x, nullptr, nullptr, y, inv_norm);
}

// Internal launchers for the model step (gpt_model.cu).
int launch_rmsnorm_fwd(deers_ctx* ctx, long long rows, int C, double eps, const float* x, float* y, float* inv_norm) {
    return rms_launch<false>(ctx, rows, C, (float)eps, x, nullptr, nullptr, y, inv_norm);
}
int launch_rmsnorm_bwd(deers_ctx* ctx, long long rows, int C, const float* x, const float* inv_norm, const float* dy,
                       const float* add, float* dx, float* n_out) {
    return rms_launch<true>(ctx, rows, C, 0.f, x, dy, inv_norm, dx, nullptr, add, n_out);
}
// y as an f16 pair, one pass where the row stays in registers.  DEERS_ERR_UNSUPPORTED otherwise: the caller normalises and
// splits in two.
int launch_rmsnorm_split(deers_ctx* ctx, long long rows, int C, double eps, const float* x, float* inv_norm, void* hi, void* lo) {
    if (C % 4 || C > 256 * RN_MAXV * 4 || (((uintptr_t)x | (uintptr_t)hi | (uintptr_t)lo) & 15u)) return DEERS_ERR_UNSUPPORTED;
    const long long cap = 16LL * ctx->sm_count, want = C <= 32 * RN_MAXV * 4 ? (rows + 7) / 8 : rows;
    const unsigned grid = (unsigned)(want < cap ? want : cap);
    const float inv_n = (float)(1.0 / (double)C);
    {
        KernelTimerScope ts(ctx, DEERS_K_NORM);
        if (C <= 32 * RN_MAXV * 4)
            DEERS_CUDA_TRY(ctx, launch_chained(ctx, rmsnorm_kernel<false, true, false, true>, grid, 256, 0, 1, x, nullptr, nullptr, nullptr, nullptr, inv_norm,
                                               rows, C, (float)eps, inv_n, nullptr, (__half*)hi, (__half*)lo));
        else
            DEERS_CUDA_TRY(ctx, launch_chained(ctx, rmsnorm_block_kernel<false, true>, grid, 256, 0, 1, x, nullptr, nullptr, nullptr, nullptr, inv_norm, rows, C,
                                               (float)eps, inv_n, nullptr, (__half*)hi, (__half*)lo));
    }
    ctx->launches += 1;
    DEERS_CUDA_TRY(ctx, cudaGetLastError());
    return DEERS_OK;
}

extern "C" int deers_b200_rmsnorm_bwd_add(deers_ctx* ctx, int64_t rows, int32_t C, const float* x, const float* inv_norm,
                                          const float* dy, const float* residual_grad, float* dx) {
    int rc = rms_check(ctx, rows, C, x, inv_norm, dy, dx);
    if (rc) return rc;
    if (!residual_grad) return DEERS_ERR_NULL;
    if ((uintptr_t)residual_grad & 3u) return DEERS_ERR_LAYOUT;
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    return rms_launch<true>(ctx, rows, C, 0.f, x, dy, inv_norm, dx, nullptr, residual_grad);
}

extern "C" int deers_b200_rmsnorm_bwd(deers_ctx* ctx, int64_t rows, int32_t C, const float* x, const float* inv_norm,
                                      const float* dy, float* dx) {
    int rc = rms_check(ctx, rows, C, x, inv_norm, dy, dx);
    if (rc) return rc;
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    return rms_launch<true>(ctx, rows, C, 0.f, x, dy, inv_norm, dx, nullptr);
}
