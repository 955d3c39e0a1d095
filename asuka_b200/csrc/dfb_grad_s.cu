// Adjoint-first derivative kernels, bra classes (0,0), (1,0).
#include "dfb_grad_tmpl.cuh"

namespace dfb {
cudaError_t grad_run_00(const GradLaunch& L) { return grad_launch_lc<0, 0>(L); }
cudaError_t grad_run_10(const GradLaunch& L) { return grad_launch_lc<1, 0>(L); }
}  // namespace dfb
