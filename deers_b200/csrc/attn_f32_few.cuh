// f32 causal attention in blocks of 16 and 8 stationary rows, for calls of few blocks (the kernels: attn_f32_kernel.cuh).  A module per tile width:
// the first call of a process loads all kernels of its module, and a program has one width as a rule.
#pragma once
#include "attn_f32_kernel.cuh"

namespace {

template <int DP, int RM>
int fwd_few(deers_ctx* ctx, const F32Params& p, int groups, int stream) {
    if constexpr (DP <= 32) {
        if (groups == 8) return fwd_launch_f32<DP, 8, 32, RM>(ctx, p);
    }
    if constexpr (DP == 64) {
        if (stream == 64) return fwd_launch_f32<DP, 4, 64, RM>(ctx, p);
    }
    return fwd_launch_f32<DP, 4, 32, RM>(ctx, p);
}

template <int DP, int RM>
int bwd_few(deers_ctx* ctx, const F32Params& p, int groups) {
    if constexpr (DP <= 64) {
        if (groups == 8) return bwd_launch_f32<DP, 8, RM>(ctx, p);
    }
    return bwd_launch_f32<DP, 4, RM>(ctx, p);
}

template <int DP>
int fwd_few_rows(deers_ctx* ctx, const F32Params& p, int groups, int stream, int rm) {
    return rm == 2 ? fwd_few<DP, 2>(ctx, p, groups, stream) : fwd_few<DP, 1>(ctx, p, groups, stream);
}
template <int DP>
int bwd_few_rows(deers_ctx* ctx, const F32Params& p, int groups, int rm) {
    return rm == 2 ? bwd_few<DP, 2>(ctx, p, groups) : bwd_few<DP, 1>(ctx, p, groups);
}

}  // namespace
