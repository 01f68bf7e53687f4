// Q8_0 weights of the f32-accurate prefill GEMM (a translation unit of its own: they compile side by side).
#include "gemm_exact.cuh"

namespace zc {

cudaError_t launch_exact_q8(const ExactGemm& p, const XPlan& plan, const ExactPrep& prep, cudaStream_t s) {
    // rows have a 16-byte pitch, as a tensor map needs, only where K % 256 == 0
    if (p.K & 255u) return x_launch_bn<T_Q8_0, true>(p, plan, prep, s);
    return x_launch_bn<T_Q8_0, false>(p, plan, prep, s);
}

}  // namespace zc
