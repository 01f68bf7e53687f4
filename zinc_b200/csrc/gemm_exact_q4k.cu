// Q4_K weights of the f32-accurate prefill GEMM (a translation unit of its own: they compile side by side).
#include "gemm_exact.cuh"

namespace zc {

cudaError_t launch_exact_q4k(const ExactGemm& p, const XPlan& plan, const ExactPrep& prep, cudaStream_t s) {
    return x_launch_bn<T_Q4_K, false>(p, plan, prep, s);
}

}  // namespace zc
