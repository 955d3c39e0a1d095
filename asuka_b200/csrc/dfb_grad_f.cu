// Adjoint-first derivative kernels, bra classes (3,0), (3,1).
#include "dfb_grad_tmpl.cuh"

namespace dfb {
cudaError_t grad_run_30(const GradLaunch& L) { return grad_launch_lc<3, 0>(L); }
cudaError_t grad_run_31(const GradLaunch& L) { return grad_launch_lc<3, 1>(L); }
}  // namespace dfb
