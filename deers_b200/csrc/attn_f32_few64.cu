// f32 causal attention, few blocks, heads of up to 64 columns (attn_f32_few.cuh).
#include "attn_f32_few.cuh"

int launch_attn_fwd_f32_few64(deers_ctx* ctx, const F32Params& p, int groups, int stream, int rm) {
    return fwd_few_rows<64>(ctx, p, groups, stream, rm);
}
int launch_attn_bwd_f32_few64(deers_ctx* ctx, const F32Params& p, int groups, int rm) { return bwd_few_rows<64>(ctx, p, groups, rm); }
