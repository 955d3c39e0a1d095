// Primitive-group integral kernels, bra classes (0,0), (1,0).
#include "dfb_prim_tmpl.cuh"

namespace dfb {
cudaError_t prim_out_00(const PrimLaunch& L) { return prim_launch_out<0, 0>(L); }
cudaError_t prim_int_00(const PrimLaunch& L) { return prim_launch_int<0, 0>(L); }
cudaError_t prim_out_10(const PrimLaunch& L) { return prim_launch_out<1, 0>(L); }
cudaError_t prim_int_10(const PrimLaunch& L) { return prim_launch_int<1, 0>(L); }
}  // namespace dfb
