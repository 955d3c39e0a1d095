// Primitive-group integral kernels, bra classes (4,3), (4,4).
#include "dfb_prim_tmpl.cuh"

namespace dfb {
cudaError_t prim_out_43(const PrimLaunch& L) { return prim_launch_out<4, 3>(L); }
cudaError_t prim_int_43(const PrimLaunch& L) { return prim_launch_int<4, 3>(L); }
cudaError_t prim_out_44(const PrimLaunch& L) { return prim_launch_out<4, 4>(L); }
cudaError_t prim_int_44(const PrimLaunch& L) { return prim_launch_int<4, 4>(L); }
}  // namespace dfb
