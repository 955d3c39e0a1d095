// Primitive-group integral kernels, bra classes (4,0), (4,1), (4,2).
#include "dfb_prim_tmpl.cuh"

namespace dfb {
cudaError_t prim_out_40(const PrimLaunch& L) { return prim_launch_out<4, 0>(L); }
cudaError_t prim_int_40(const PrimLaunch& L) { return prim_launch_int<4, 0>(L); }
cudaError_t prim_out_41(const PrimLaunch& L) { return prim_launch_out<4, 1>(L); }
cudaError_t prim_int_41(const PrimLaunch& L) { return prim_launch_int<4, 1>(L); }
cudaError_t prim_out_42(const PrimLaunch& L) { return prim_launch_out<4, 2>(L); }
cudaError_t prim_int_42(const PrimLaunch& L) { return prim_launch_int<4, 2>(L); }
}  // namespace dfb
