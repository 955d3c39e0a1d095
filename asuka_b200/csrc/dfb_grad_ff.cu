// Adjoint-first derivative kernels, bra classes (3,2), (3,3).
#include "dfb_grad_tmpl.cuh"

namespace dfb {
cudaError_t grad_run_32(const GradLaunch& L) { return grad_launch_lc<3, 2>(L); }
cudaError_t grad_run_33(const GradLaunch& L) { return grad_launch_lc<3, 3>(L); }
}  // namespace dfb
