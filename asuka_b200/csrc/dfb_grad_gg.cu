// Adjoint-first derivative kernels, bra classes (4,3), (4,4).
#include "dfb_grad_tmpl.cuh"

namespace dfb {
cudaError_t grad_run_43(const GradLaunch& L) { return grad_launch_lc<4, 3>(L); }
cudaError_t grad_run_44(const GradLaunch& L) { return grad_launch_lc<4, 4>(L); }
}  // namespace dfb
