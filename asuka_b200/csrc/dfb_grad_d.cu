// Adjoint-first derivative kernels, bra classes (2,0), (2,1).
#include "dfb_grad_tmpl.cuh"

namespace dfb {
cudaError_t grad_run_20(const GradLaunch& L) { return grad_launch_lc<2, 0>(L); }
cudaError_t grad_run_21(const GradLaunch& L) { return grad_launch_lc<2, 1>(L); }
}  // namespace dfb
