// Adjoint-first derivative kernels, bra classes (1,1).
#include "dfb_grad_tmpl.cuh"

namespace dfb {
cudaError_t grad_run_11(const GradLaunch& L) { return grad_launch_lc<1, 1>(L); }
}  // namespace dfb
