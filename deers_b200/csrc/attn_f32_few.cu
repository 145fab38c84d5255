// f32 causal attention in blocks of 16 and 8 stationary rows, for calls of few blocks (the kernels: attn_f32_kernel.cuh).
#include "attn_f32_kernel.cuh"

namespace {

template <int DP, int RM>
int fwd_few(deers_ctx* ctx, const F32Params& p, int groups, int stream) {
    if constexpr (DP <= 32) {
        if (groups == 8) return fwd_launch_f32<DP, 8, 32, RM>(ctx, p);
    }
    if constexpr (DP <= 64) {
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

template <int RM>
int fwd_few_dp(deers_ctx* ctx, const F32Params& p, int dp, int groups, int stream) {
    return dp == 32 ? fwd_few<32, RM>(ctx, p, groups, stream) : dp == 64 ? fwd_few<64, RM>(ctx, p, groups, stream)
         : dp == 96 ? fwd_few<96, RM>(ctx, p, groups, stream) : fwd_few<128, RM>(ctx, p, groups, stream);
}
template <int RM>
int bwd_few_dp(deers_ctx* ctx, const F32Params& p, int dp, int groups) {
    return dp == 32 ? bwd_few<32, RM>(ctx, p, groups) : dp == 64 ? bwd_few<64, RM>(ctx, p, groups)
         : dp == 96 ? bwd_few<96, RM>(ctx, p, groups) : bwd_few<128, RM>(ctx, p, groups);
}

}  // namespace

int launch_attn_fwd_f32_few(deers_ctx* ctx, const F32Params& p, int dp, int groups, int stream, int rm) {
    return rm == 2 ? fwd_few_dp<2>(ctx, p, dp, groups, stream) : fwd_few_dp<1>(ctx, p, dp, groups, stream);
}
int launch_attn_bwd_f32_few(deers_ctx* ctx, const F32Params& p, int dp, int groups, int rm) {
    return rm == 2 ? bwd_few_dp<2>(ctx, p, dp, groups) : bwd_few_dp<1>(ctx, p, dp, groups);
}
