// The kernels of gemm_f32_kernel.cuh for operands whose rows lie on no 16-byte boundary.
#include "gemm_f32_kernel.cuh"

int launch_gemm_f32_loose(deers_ctx* ctx, const GemmPlan& p, const GemmArgs& g, int a_mn, int b_mn, bool fused) {
    return launch_tiles<true>(ctx, p, g, a_mn, b_mn, fused);
}
