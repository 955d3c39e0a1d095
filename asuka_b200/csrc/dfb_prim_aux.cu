// Primitive-group integral kernels of the metric for aux shells above g (bra = one primitive aux function).
#include "dfb_prim_tmpl.cuh"

namespace dfb {
cudaError_t prim_int_50(const PrimLaunch& L) { return prim_launch_f<5, 0>(L); }
cudaError_t prim_int_60(const PrimLaunch& L) { return prim_launch_f<6, 0>(L); }
cudaError_t prim_int_70(const PrimLaunch& L) { return prim_launch_f<7, 0>(L); }
cudaError_t prim_int_80(const PrimLaunch& L) { return prim_launch_f<8, 0>(L); }
}  // namespace dfb
