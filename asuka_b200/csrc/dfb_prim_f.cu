// Primitive-group integral kernels, bra classes (3,0), (3,1).
#include "dfb_prim_tmpl.cuh"

namespace dfb {
cudaError_t prim_out_30(const PrimLaunch& L) { return prim_launch_out<3, 0>(L); }
cudaError_t prim_int_30(const PrimLaunch& L) { return prim_launch_int<3, 0>(L); }
cudaError_t prim_out_31(const PrimLaunch& L) { return prim_launch_out<3, 1>(L); }
cudaError_t prim_int_31(const PrimLaunch& L) { return prim_launch_int<3, 1>(L); }
}  // namespace dfb
