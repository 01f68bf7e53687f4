// Q5_K weights of the f32-accurate prefill GEMM (a translation unit of its own: they compile side by side).
#include "gemm_exact.cuh"

namespace zc {

cudaError_t launch_exact_q5k(const ExactGemm& p, const XPlan& plan, bool dry, cudaStream_t s, ExactGrid* grid) {
    return x_launch_bn<T_Q5_K, false>(p, plan, dry, s, grid);
}

}  // namespace zc
