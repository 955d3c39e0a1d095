// Primitive-group integral kernels, bra classes (2,0), (2,1).
#include "dfb_prim_tmpl.cuh"

namespace dfb {
cudaError_t prim_out_20(const PrimLaunch& L) { return prim_launch_out<2, 0>(L); }
cudaError_t prim_int_20(const PrimLaunch& L) { return prim_launch_int<2, 0>(L); }
cudaError_t prim_out_21(const PrimLaunch& L) { return prim_launch_out<2, 1>(L); }
cudaError_t prim_int_21(const PrimLaunch& L) { return prim_launch_int<2, 1>(L); }
}  // namespace dfb
