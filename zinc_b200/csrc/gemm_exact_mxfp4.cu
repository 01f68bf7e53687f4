// MXFP4 weights of the f32-accurate prefill GEMM (a translation unit of its own: they compile side by side).
#include "gemm_exact.cuh"

namespace zc {

cudaError_t launch_exact_mxfp4(const ExactGemm& p, const XPlan& plan, const ExactPrep& prep, cudaStream_t s) {
    return x_launch_bn<T_MXFP4, true>(p, plan, prep, s);
}

}  // namespace zc
