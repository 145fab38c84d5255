// f32 GEMM on the tensor core, rows on any 4-byte boundary: a module of its own, as most programs never need it (see gemm_f32_kernel.cuh).
#include "gemm_f32_tc.cuh"

int launch_gemm_f32_tc_loose(deers_ctx* ctx, int parts, const GemmArgs& g, int a_mn, int b_mn) {
    return launch_tc_orders<true>(ctx, parts, g, a_mn, b_mn);
}
