// Decode-time attention: a few new query rows against a long key / value cache (split-KV).
//
// The reference's mask helper already models queries that sit `seqlen_offset` positions into a longer
// key sequence (causal_mask, src/nn/functional.rs:12-55: key j is masked for query i iff
// j > i + seqlen_offset), but its sampling loop re-runs the whole prefix for every token
// (src/bin/tinystories_train.rs sampling: O(T^2) per token).  With a KV cache the step is
// `softmax(scale * q K^T + mask) V` for Tq new rows against Tk = Tq + offset cached rows: no tensor-core
// shape (M = Tq is tiny), purely bound by reading K and V once.
//
//   decode_vec_kernel       grid (splits, B*H): a block takes one chunk of the keys of one slice; its four
//                           warps stride over the chunk's keys; the lanes that share a key each own 16 bytes
//                           of its row (16-byte loads, four key groups in flight): dot product by shuffle
//                           reduction, online softmax, V accumulated in registers (f32); lane groups and
//                           warps are merged.  With up to eight chunks the blocks of a slice are one cluster: they merge
//                           through distributed shared memory and write O (and lse) themselves; one chunk needs no merge at
//                           all.  With more the block writes (max, sum, unnormalised O) of its chunk to the workspace.
//   decode_partial_kernel   the same with element loads, for rows that are not aligned 16-byte pieces.
//   decode_combine_kernel   merges the chunks of a (slice, query) pair from the workspace, normalises, writes O (and lse).
// What bounds it: a batch of long caches reads K and V at the copy bandwidth.  A single short sequence is launch and load
// latency: B1 H12 Tk777 D64 took 4.4 us + 2.6 us in two launches with 208 keys per block, 4.6 us in one.
// K and V are read once per query row (Tq is 1 in sampling); 2 * Tk * D * sizeof(T) bytes per slice.
#include <cuda_fp16.h>

#include "common.cuh"

#include <cooperative_groups.h>

namespace {

constexpr int DEC_MAXC = 8;             // channels per lane: head_dim <= 256
constexpr int DEC_MAX_SPLITS = 4 * 148;   // chunks of a slice (one slice on an otherwise idle device)
constexpr float DEC_LOG2E = 1.4426950408889634f;

struct DecodeParams {
    const void* q; const void* k; const void* v; void* o;
    float* lse;                          // [B*H*Tq] or nullptr
    float* part;                         // [B*H][Tq][splits][D + 2]
    long long sq[3], sk[3], sv[3], so[3];   // (b, h, t) strides in elements
    int B, H, Tq, Tk, D, causal, splits, chunk;
    float scale;
};

__device__ __forceinline__ float ld(const float* p) { return *p; }
__device__ __forceinline__ float ld(const __half* p) { return __half2float(*p); }
__device__ __forceinline__ void st(float* p, float v) { *p = v; }
__device__ __forceinline__ void st(__half* p, float v) { *p = __float2half_rn(v); }

template <typename T>
__global__ void __launch_bounds__(128) decode_partial_kernel(const DecodeParams p) {
    chain_begin();
    const int split = blockIdx.x, bh = blockIdx.y;
    const int b = bh / p.H, h = bh % p.H;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nc = (p.D + 31) / 32;                              // channels of this lane: lane, lane + 32, ...
    const int k_begin = split * p.chunk, k_end = min(p.Tk, k_begin + p.chunk);
    const int offset = p.Tk - p.Tq;
    const T* kb = static_cast<const T*>(p.k) + b * p.sk[0] + h * p.sk[1];
    const T* vb = static_cast<const T*>(p.v) + b * p.sv[0] + h * p.sv[1];
    const float sl2 = p.scale * DEC_LOG2E;
    __shared__ float sm_m[4], sm_l[4];
    __shared__ float sm_o[4][32 * DEC_MAXC];

    for (int i = 0; i < p.Tq; ++i) {
        const T* qr = static_cast<const T*>(p.q) + b * p.sq[0] + h * p.sq[1] + (long long)i * p.sq[2];
        float qv[DEC_MAXC], acc[DEC_MAXC];
#pragma unroll
        for (int c = 0; c < DEC_MAXC; ++c) {
            const int d = lane + 32 * c;
            qv[c] = (c < nc && d < p.D) ? ld(qr + d) : 0.f;
            acc[c] = 0.f;
        }
        const int last = p.causal ? min(k_end, i + offset + 1) : k_end;      // keys j <= i + offset
        float m = -INFINITY, l = 0.f;
        for (int j0 = k_begin + warp * 4; j0 < last; j0 += 16) {             // four keys per warp iteration
            float s[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int j = j0 + u;
                float dot = 0.f;
                if (j < last) {
                    const T* kr = kb + (long long)j * p.sk[2];
#pragma unroll
                    for (int c = 0; c < DEC_MAXC; ++c) {
                        const int d = lane + 32 * c;
                        if (c < nc && d < p.D) dot = fmaf(qv[c], ld(kr + d), dot);
                    }
                }
                s[u] = dot;
            }
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) {
#pragma unroll
                for (int u = 0; u < 4; ++u) s[u] += __shfl_xor_sync(0xffffffffu, s[u], off);
            }
            float mx = m;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                s[u] = (j0 + u < last) ? s[u] * sl2 : -INFINITY;
                mx = fmaxf(mx, s[u]);
            }
            const float corr = exp2f(m - mx);                                // 0 on the first keys (m = -inf)
            l *= corr;
#pragma unroll
            for (int c = 0; c < DEC_MAXC; ++c) acc[c] *= corr;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int j = j0 + u;
                if (j < last) {
                    const float pj = exp2f(s[u] - mx);
                    l += pj;
                    const T* vr = vb + (long long)j * p.sv[2];
#pragma unroll
                    for (int c = 0; c < DEC_MAXC; ++c) {
                        const int d = lane + 32 * c;
                        if (c < nc && d < p.D) acc[c] = fmaf(pj, ld(vr + d), acc[c]);
                    }
                }
            }
            m = mx;
        }
        // merge the four warps (a warp without keys has m = -inf, l = 0)
        __syncthreads();                                                     // shared arrays of the previous query are free
        if (lane == 0) { sm_m[warp] = m; sm_l[warp] = l; }
#pragma unroll
        for (int c = 0; c < DEC_MAXC; ++c) sm_o[warp][lane + 32 * c] = acc[c];
        __syncthreads();
        if (warp == 0) {
            float mm = fmaxf(fmaxf(sm_m[0], sm_m[1]), fmaxf(sm_m[2], sm_m[3]));
            const float ms = (mm == -INFINITY) ? 0.f : mm;
            float w[4], ll = 0.f;
#pragma unroll
            for (int x = 0; x < 4; ++x) { w[x] = exp2f(sm_m[x] - ms); ll += w[x] * sm_l[x]; }
            float* out = p.part + (((long long)bh * p.Tq + i) * p.splits + split) * (p.D + 2);
#pragma unroll
            for (int c = 0; c < DEC_MAXC; ++c) {
                const int d = lane + 32 * c;
                if (c < nc && d < p.D) {
                    float o = 0.f;
#pragma unroll
                    for (int x = 0; x < 4; ++x) o += w[x] * sm_o[x][d];
                    out[d] = o;
                }
            }
            if (lane == 0) { out[p.D] = mm; out[p.D + 1] = ll; }
        }
    }
}

// 16-byte path: LPK lanes (a power of two) share a key and own 16 bytes of its row each (those beyond the row's pieces idle),
// so a warp instruction covers 32 / LPK keys; four such groups of keys are in flight per iteration.  Needs 16-byte aligned rows.
enum DecodeEnd { DEC_TO_WORKSPACE = 0, DEC_ONE_CHUNK = 1, DEC_CLUSTER = 2 };   // what a block does with its chunk's result
// Seven blocks per SM (72 registers) where a batch of caches streams: what is in flight counts; at 96 registers B64 H32
// Tk2048 D128 takes 336 us instead of 323.
template <typename T, int LPK, int END>
__global__ void __launch_bounds__(128, END == DEC_CLUSTER ? 6 : 7) decode_vec_kernel(const DecodeParams p) {
    chain_wait();
    constexpr int VEC = 16 / (int)sizeof(T);                     // channels per lane
    constexpr int KPW = 32 / LPK;                                // keys per warp instruction
    constexpr int U = 4;                                         // key groups in flight
    const int split = blockIdx.x, bh = blockIdx.y;
    const int b = bh / p.H, h = bh % p.H;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sub = lane / LPK, cl = lane % LPK;
    const bool mine = cl * VEC < p.D;                            // this lane has a piece of the row
    const int k_begin = split * p.chunk, k_end = min(p.Tk, k_begin + p.chunk);
    const int offset = p.Tk - p.Tq;
    const T* kb = static_cast<const T*>(p.k) + b * p.sk[0] + h * p.sk[1] + cl * VEC;
    const T* vb = static_cast<const T*>(p.v) + b * p.sv[0] + h * p.sv[1] + cl * VEC;
    const float sl2 = p.scale * DEC_LOG2E;
    __shared__ float sm_m[4], sm_l[4];
    __shared__ float sm_o[4][32 * DEC_MAXC];
    __shared__ float sm_part[END == DEC_CLUSTER ? 2 : 1][END == DEC_CLUSTER ? 32 * DEC_MAXC + 2 : 1];   // this chunk's O, max and sum (two queries in turn)

    auto unpack = [](const uint4& r, float (&f)[VEC]) {
        if constexpr (sizeof(T) == 2) {
            const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&w[e]));
                f[2 * e] = t.x; f[2 * e + 1] = t.y;
            }
        } else {
            f[0] = __uint_as_float(r.x); f[1] = __uint_as_float(r.y); f[2] = __uint_as_float(r.z); f[3] = __uint_as_float(r.w);
        }
    };

    for (int i = 0; i < p.Tq; ++i) {
        const T* qr = static_cast<const T*>(p.q) + b * p.sq[0] + h * p.sq[1] + (long long)i * p.sq[2] + cl * VEC;
        float qv[VEC], acc[VEC];
        unpack(mine ? *reinterpret_cast<const uint4*>(qr) : make_uint4(0u, 0u, 0u, 0u), qv);
#pragma unroll
        for (int c = 0; c < VEC; ++c) acc[c] = 0.f;
        const int last = p.causal ? min(k_end, i + offset + 1) : k_end;
        float m = -INFINITY, l = 0.f;
        // this lane group's keys: k_begin + (warp * U + u) * KPW + sub, stepping 4 warps * U * KPW
        for (int j0 = k_begin + warp * U * KPW; j0 < last; j0 += 4 * U * KPW) {
            uint4 kr[U], vr[U];
            bool ok[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int j = j0 + u * KPW + sub;
                ok[u] = j < last;
                kr[u] = make_uint4(0u, 0u, 0u, 0u);
                vr[u] = kr[u];
                if (ok[u] && mine) {
                    kr[u] = *reinterpret_cast<const uint4*>(kb + (long long)j * p.sk[2]);
                    vr[u] = *reinterpret_cast<const uint4*>(vb + (long long)j * p.sv[2]);
                }
            }
            float s[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                float kf[VEC];
                unpack(kr[u], kf);
                float dot = 0.f;
#pragma unroll
                for (int c = 0; c < VEC; ++c) dot = fmaf(qv[c], kf[c], dot);
                s[u] = dot;
            }
#pragma unroll
            for (int off = LPK / 2; off >= 1; off >>= 1) {
#pragma unroll
                for (int u = 0; u < U; ++u) s[u] += __shfl_xor_sync(0xffffffffu, s[u], off);
            }
            float mx = m;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                s[u] = ok[u] ? s[u] * sl2 : -INFINITY;
                mx = fmaxf(mx, s[u]);
            }
            // The maximum is -inf before this lane group's first key, but also while all its scores are NaN (fmaxf passes over
            // them): those must reach the sums, so no step is skipped.
            const float ms = mx == -INFINITY ? 0.f : mx, corr = exp2f(m - ms);
            l *= corr;
#pragma unroll
            for (int c = 0; c < VEC; ++c) acc[c] *= corr;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float pj = exp2f(s[u] - ms);               // 0 for keys that do not exist
                l += pj;
                float vf[VEC];
                unpack(vr[u], vf);
#pragma unroll
                for (int c = 0; c < VEC; ++c) acc[c] = fmaf(pj, vf[c], acc[c]);
            }
            m = mx;
        }
        // merge the lane groups of the warp (they saw different keys), then the four warps
#pragma unroll
        for (int off = LPK; off < 32; off <<= 1) {
            const float mo = __shfl_xor_sync(0xffffffffu, m, off), lo = __shfl_xor_sync(0xffffffffu, l, off);
            const float mn = fmaxf(m, mo);
            const float ms = (mn == -INFINITY) ? 0.f : mn;
            const float wa = exp2f(m - ms), wb = exp2f(mo - ms);
#pragma unroll
            for (int c = 0; c < VEC; ++c) acc[c] = wa * acc[c] + wb * __shfl_xor_sync(0xffffffffu, acc[c], off);
            l = wa * l + wb * lo;
            m = mn;
        }
        __syncthreads();
        if (lane == 0) { sm_m[warp] = m; sm_l[warp] = l; }
        if (i == p.Tq - 1) chain_next();
        if (sub == 0 && mine) {
#pragma unroll
            for (int c = 0; c < VEC; ++c) sm_o[warp][cl * VEC + c] = acc[c];
        }
        __syncthreads();
        if (warp == 0) {
            const float mm = fmaxf(fmaxf(sm_m[0], sm_m[1]), fmaxf(sm_m[2], sm_m[3]));
            const float ms = (mm == -INFINITY) ? 0.f : mm;
            float w[4], ll = 0.f;
#pragma unroll
            for (int x = 0; x < 4; ++x) { w[x] = exp2f(sm_m[x] - ms); ll += w[x] * sm_l[x]; }
            if constexpr (END == DEC_ONE_CHUNK) {                    // the chunk is the whole cache: this is the result
                const float inv = 1.f / ll;
                T* orow = static_cast<T*>(p.o) + b * p.so[0] + h * p.so[1] + (long long)i * p.so[2];
                for (int d = lane; d < p.D; d += 32) {
                    float o = 0.f;
#pragma unroll
                    for (int x = 0; x < 4; ++x) o += w[x] * sm_o[x][d];
                    st(orow + d, o * inv);
                }
                if (p.lse && lane == 0) p.lse[(long long)bh * p.Tq + i] = (mm + log2f(ll)) * 0.6931471805599453f;
            } else {
                float* out = END == DEC_CLUSTER ? sm_part[i & 1] : p.part + (((long long)bh * p.Tq + i) * p.splits + split) * (p.D + 2);
                for (int d = lane; d < p.D; d += 32) {
                    float o = 0.f;
#pragma unroll
                    for (int x = 0; x < 4; ++x) o += w[x] * sm_o[x][d];
                    out[d] = o;
                }
                if (lane == 0) { out[p.D] = mm; out[p.D + 1] = ll; }
            }
        }
        if constexpr (END == DEC_CLUSTER) {
            // The cluster's blocks share the channels; the next query's partial goes to the other buffer, so one cluster
            // barrier per query keeps writers off what is still being read.
            cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
            cluster.sync();
            const float* part[8];
            float w[8], mx = -INFINITY, l_all = 0.f;
#pragma unroll
            for (int z = 0; z < 8; ++z) {
                part[z] = cluster.map_shared_rank(sm_part[i & 1], z < p.splits ? z : 0);
                w[z] = z < p.splits ? part[z][p.D] : -INFINITY;
                mx = fmaxf(mx, w[z]);
            }
            const float mxs = (mx == -INFINITY) ? 0.f : mx;
#pragma unroll
            for (int z = 0; z < 8; ++z) {
                w[z] = exp2f(w[z] - mxs);
                if (z < p.splits) l_all = fmaf(w[z], part[z][p.D + 1], l_all);
            }
            const float inv = 1.f / l_all;
            const int share = (p.D + p.splits - 1) / p.splits, d_end = min(p.D, (split + 1) * share);
            T* orow = static_cast<T*>(p.o) + b * p.so[0] + h * p.so[1] + (long long)i * p.so[2];
            for (int d = split * share + (int)threadIdx.x; d < d_end; d += 128) {
                float o = 0.f;
#pragma unroll
                for (int z = 0; z < 8; ++z)
                    if (z < p.splits) o = fmaf(w[z], part[z][d], o);
                st(orow + d, o * inv);
            }
            if (p.lse && split == 0 && threadIdx.x == 0) p.lse[(long long)bh * p.Tq + i] = (mx + log2f(l_all)) * 0.6931471805599453f;
        }
    }
    if constexpr (END == DEC_CLUSTER) {
        cooperative_groups::this_cluster().sync();               // nobody leaves while a peer still reads its part
    }
}

template <typename T>
__global__ void __launch_bounds__(128) decode_combine_kernel(const DecodeParams p) {
    chain_begin();
    const long long row = blockIdx.x;                                        // (bh, i)
    const int bh = (int)(row / p.Tq), i = (int)(row % p.Tq);
    const int b = bh / p.H, h = bh % p.H;
    const float* part = p.part + row * p.splits * (p.D + 2);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ float sm_w[DEC_MAX_SPLITS], sm_r[8];
    // every thread takes some chunks' maximum and sum; weights go to shared memory
    float mm = -INFINITY;
    for (int z = threadIdx.x; z < p.splits; z += 128) {
        sm_w[z] = part[z * (p.D + 2) + p.D];
        mm = fmaxf(mm, sm_w[z]);
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, off));
    if (lane == 0) sm_r[warp] = mm;
    __syncthreads();
    mm = fmaxf(fmaxf(sm_r[0], sm_r[1]), fmaxf(sm_r[2], sm_r[3]));
    const float ms = (mm == -INFINITY) ? 0.f : mm;
    float l = 0.f;
    for (int z = threadIdx.x; z < p.splits; z += 128) {
        const float w = exp2f(sm_w[z] - ms);
        sm_w[z] = w;
        l = fmaf(w, part[z * (p.D + 2) + p.D + 1], l);
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
    if (lane == 0) sm_r[4 + warp] = l;
    __syncthreads();
    l = (sm_r[4] + sm_r[5]) + (sm_r[6] + sm_r[7]);
    const float inv = 1.f / l;
    T* orow = static_cast<T*>(p.o) + b * p.so[0] + h * p.so[1] + (long long)i * p.so[2];
    for (int d = threadIdx.x; d < p.D; d += 128) {
        float o[4] = {0.f, 0.f, 0.f, 0.f};                                   // four chains of independent loads
        int z = 0;
        for (; z + 4 <= p.splits; z += 4) {
#pragma unroll
            for (int u = 0; u < 4; ++u) o[u] = fmaf(sm_w[z + u], part[(z + u) * (p.D + 2) + d], o[u]);
        }
        for (; z < p.splits; ++z) o[0] = fmaf(sm_w[z], part[z * (p.D + 2) + d], o[0]);
        st(orow + d, ((o[0] + o[1]) + (o[2] + o[3])) * inv);
    }
    if (p.lse && threadIdx.x == 0) p.lse[row] = (mm + log2f(l)) * 0.6931471805599453f;   // natural log, like the forward op
}

// 16-byte path when a row is 1..32 whole pieces and every stride keeps rows aligned (base pointers are checked at launch).
bool decode_vec_ok(const deers_decode_desc* d) {
    const int64_t es = d->dtype == DEERS_F16 ? 2 : 4;
    if ((d->D * es) % 16 != 0 || d->D * es / 16 > 32) return false;
    for (int i = 0; i < 3; ++i)
        if ((d->q_strides[i] * es) % 16 != 0 || (d->k_strides[i] * es) % 16 != 0 || (d->v_strides[i] * es) % 16 != 0) return false;
    return true;
}

// How the keys are cut.  *cluster: the chunks of a slice run as one cluster of up to 8 blocks and need no workspace.  That is
// the choice when the slices alone fill the device, and for caches of up to 8192 keys, where 8 chunks of at least 64 keys
// cost less than a second launch (12 slices of 4096 x 64: 8.3 us against 12.4); longer caches of few slices take four blocks per
// SM in all and the combining launch.
int decode_splits(const deers_decode_desc* d, int* chunk, bool* cluster) {
    const long long slices = (long long)d->B * d->H;
    long long want = (4LL * 148 + slices - 1) / slices;                        // about four blocks per SM in all
    const long long by256 = (d->Tk + 255) / 256, by64 = (d->Tk + 63) / 64;
    *cluster = decode_vec_ok(d) && ((want < by256 ? want : by256) <= 8 || d->Tk <= 8192);
    if (*cluster) {
        if (want > by64) want = by64;
        if (want > 8) want = 8;
    } else if (want > by256) {
        want = by256;                                                          // at least 256 keys per block
    }
    if (want < 1) want = 1;
    long long c = (d->Tk + want - 1) / want;
    c = (c + 15) / 16 * 16;
    *chunk = (int)c;
    return (int)((d->Tk + c - 1) / c);
}

int decode_check(const deers_decode_desc* d) {
    if (!d) return DEERS_ERR_NULL;
    if (d->dtype != DEERS_F16 && d->dtype != DEERS_F32) return DEERS_ERR_DTYPE;
    if (d->B < 1 || d->H < 1 || d->Tq < 1 || d->Tk < d->Tq || d->D < 1) return DEERS_ERR_SHAPE;
    if (d->D > 32 * DEC_MAXC || d->Tq > 128 || d->Tk > (1 << 24)) return DEERS_ERR_UNSUPPORTED;
    if ((long long)d->B * d->H > 65535) return DEERS_ERR_UNSUPPORTED;           // grid.y
    if (!(d->scale == d->scale)) return DEERS_ERR_SHAPE;
    const int64_t* ss[4] = {d->q_strides, d->k_strides, d->v_strides, d->o_strides};
    for (const int64_t* s : ss) {
        if (s[3] != 1) return DEERS_ERR_LAYOUT;
        for (int i = 0; i < 3; ++i)
            if (s[i] < 0) return DEERS_ERR_LAYOUT;
    }
    return DEERS_OK;
}

}  // namespace

extern "C" size_t deers_b200_attn_decode_workspace_bytes(const deers_decode_desc* d) {
    if (decode_check(d) != DEERS_OK) return 0;
    int chunk;
    bool cluster;
    const int splits = decode_splits(d, &chunk, &cluster);
    // (the element-load kernel may have to stand in when a base pointer is misaligned: its partials need the room too)
    return (size_t)d->B * d->H * d->Tq * splits * (d->D + 2) * sizeof(float);
}

template <typename T, int LPK>
static int decode_launch_vec(deers_ctx* ctx, const DecodeParams& p, const dim3& grid, bool cluster) {
    if (!cluster || p.splits == 1) {
        if (cluster) DEERS_CUDA_TRY(ctx, launch_chained(ctx, decode_vec_kernel<T, LPK, DEC_ONE_CHUNK>, grid, 128, 0, 1, p));
        else DEERS_CUDA_TRY(ctx, launch_chained(ctx, decode_vec_kernel<T, LPK, DEC_TO_WORKSPACE>, grid, 128, 0, 1, p));
        return DEERS_OK;
    }
    DEERS_CUDA_TRY(ctx, launch_chained(ctx, decode_vec_kernel<T, LPK, DEC_CLUSTER>, grid, 128, 0, p.splits, p));
    return DEERS_OK;
}

template <typename T>
static int decode_launch(deers_ctx* ctx, const DecodeParams& p, const dim3& grid, bool vec, bool cluster) {
    const int pieces = p.D * (int)sizeof(T) / 16;
    int rc = DEERS_OK;
    if (!vec) DEERS_CUDA_TRY(ctx, launch_chained(ctx, decode_partial_kernel<T>, grid, 128, 0, 1, p));
    else if (pieces > 16) rc = decode_launch_vec<T, 32>(ctx, p, grid, cluster);
    else if (pieces > 8) rc = decode_launch_vec<T, 16>(ctx, p, grid, cluster);
    else if (pieces > 4) rc = decode_launch_vec<T, 8>(ctx, p, grid, cluster);
    else rc = decode_launch_vec<T, 4>(ctx, p, grid, cluster);
    if (rc || (vec && cluster)) return rc;
    DEERS_CUDA_TRY(ctx, launch_chained(ctx, decode_combine_kernel<T>, (unsigned)((long long)p.B * p.H * p.Tq), 128, 0, 1, p));
    ctx->launches += 1;
    return DEERS_OK;
}

extern "C" int deers_b200_attn_decode(deers_ctx* ctx, const deers_decode_desc* d, const void* q, const void* k_cache,
                                      const void* v_cache, void* o, float* lse, void* workspace, size_t workspace_bytes) {
    if (!ctx || !q || !k_cache || !v_cache || !o) return DEERS_ERR_NULL;
    int rc = decode_check(d);
    if (rc) return rc;
    const size_t es = d->dtype == DEERS_F16 ? 2 : 4;
    if (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)o) & (es - 1)) return DEERS_ERR_LAYOUT;
    DecodeParams p;
    bool cluster;
    p.splits = decode_splits(d, &p.chunk, &cluster);
    const size_t need = (size_t)d->B * d->H * d->Tq * p.splits * (d->D + 2) * sizeof(float);
    const bool vec = decode_vec_ok(d) && (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache) & 15u) == 0;
    if (!(vec && cluster) && (!workspace || workspace_bytes < need || ((uintptr_t)workspace & 3u))) return DEERS_ERR_WORKSPACE;
    DEERS_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
    p.q = q; p.k = k_cache; p.v = v_cache; p.o = o; p.lse = lse; p.part = (float*)workspace;
    for (int i = 0; i < 3; ++i) { p.sq[i] = d->q_strides[i]; p.sk[i] = d->k_strides[i]; p.sv[i] = d->v_strides[i]; p.so[i] = d->o_strides[i]; }
    p.B = d->B; p.H = d->H; p.Tq = d->Tq; p.Tk = d->Tk; p.D = d->D; p.causal = d->causal; p.scale = d->scale;
    const dim3 grid(p.splits, d->B * d->H);
    {
        KernelTimerScope ts(ctx, DEERS_K_DECODE);
        rc = d->dtype == DEERS_F16 ? decode_launch<__half>(ctx, p, grid, vec, cluster) : decode_launch<float>(ctx, p, grid, vec, cluster);
        if (rc) return rc;
    }
    ctx->launches += 1;
    DEERS_CUDA_TRY(ctx, cudaGetLastError());
    return DEERS_OK;
}
