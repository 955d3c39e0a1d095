// Adjoint-first derivative kernels, bra classes (2,2).
#include "dfb_grad_tmpl.cuh"

namespace dfb {
cudaError_t grad_run_22(const GradLaunch& L) { return grad_launch_lc<2, 2>(L); }
}  // namespace dfb
