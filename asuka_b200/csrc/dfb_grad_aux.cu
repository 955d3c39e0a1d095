// Adjoint-first derivative kernels of the metric for aux shells above g (bra = one primitive aux function).
#include "dfb_grad_tmpl.cuh"

namespace dfb {
cudaError_t grad_run_50(const GradLaunch& L) { return grad_launch_f<5, 0, 0>(L); }
cudaError_t grad_run_60(const GradLaunch& L) { return grad_launch_f<6, 0, 0>(L); }
cudaError_t grad_run_70(const GradLaunch& L) { return grad_launch_f<7, 0, 0>(L); }
cudaError_t grad_run_80(const GradLaunch& L) { return grad_launch_f<8, 0, 0>(L); }
}  // namespace dfb
