// Primitive-group integral kernels, bra classes (3,2), (3,3).
#include "dfb_prim_tmpl.cuh"

namespace dfb {
cudaError_t prim_out_32(const PrimLaunch& L) { return prim_launch_out<3, 2>(L); }
cudaError_t prim_int_32(const PrimLaunch& L) { return prim_launch_int<3, 2>(L); }
cudaError_t prim_out_33(const PrimLaunch& L) { return prim_launch_out<3, 3>(L); }
cudaError_t prim_int_33(const PrimLaunch& L) { return prim_launch_int<3, 3>(L); }
}  // namespace dfb
