// f32 causal attention, few blocks, heads of up to 128 columns (attn_f32_few.cuh).
#include "attn_f32_few.cuh"

int launch_attn_fwd_f32_few128(deers_ctx* ctx, const F32Params& p, int groups, int stream, int rm) {
    return fwd_few_rows<128>(ctx, p, groups, stream, rm);
}
int launch_attn_bwd_f32_few128(deers_ctx* ctx, const F32Params& p, int groups, int rm) { return bwd_few_rows<128>(ctx, p, groups, rm); }
