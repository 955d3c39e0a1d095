// Primitive-group integral kernels, bra classes (2,2).
#include "dfb_prim_tmpl.cuh"

namespace dfb {
cudaError_t prim_out_22(const PrimLaunch& L) { return prim_launch_out<2, 2>(L); }
cudaError_t prim_int_22(const PrimLaunch& L) { return prim_launch_int<2, 2>(L); }
}  // namespace dfb
