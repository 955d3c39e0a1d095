// Adjoint-first derivative kernels, bra classes (4,0), (4,1), (4,2).
#include "dfb_grad_tmpl.cuh"

namespace dfb {
cudaError_t grad_run_40(const GradLaunch& L) { return grad_launch_lc<4, 0>(L); }
cudaError_t grad_run_41(const GradLaunch& L) { return grad_launch_lc<4, 1>(L); }
cudaError_t grad_run_42(const GradLaunch& L) { return grad_launch_lc<4, 2>(L); }
}  // namespace dfb
