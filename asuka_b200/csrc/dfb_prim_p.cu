// Primitive-group integral kernels, bra classes (1,1).
#include "dfb_prim_tmpl.cuh"

namespace dfb {
cudaError_t prim_out_11(const PrimLaunch& L) { return prim_launch_out<1, 1>(L); }
cudaError_t prim_int_11(const PrimLaunch& L) { return prim_launch_int<1, 1>(L); }
}  // namespace dfb
