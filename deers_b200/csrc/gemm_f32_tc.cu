// f32 GEMM on the tensor core, rows of both operands on 16-byte boundaries (the tile: gemm_f32_tc.cuh).
#include "gemm_f32_tc.cuh"

int launch_gemm_f32_tc(deers_ctx* ctx, int parts, const GemmArgs& g, int a_mn, int b_mn, bool fused) {
    if (fused) return launch_tc_order<false, true, true, false>(ctx, parts, g);
    return launch_tc_orders<false>(ctx, parts, g, a_mn, b_mn);
}
