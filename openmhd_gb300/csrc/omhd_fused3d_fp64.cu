// omhd_fused3d_fp64.cu -- 3D fused stage kernels, arithmetic variant "fp64"
// (face arithmetic in double).
#define OMHD_VARIANT v_fp64
#define OMHD_FAST true
#include "omhd_fused3d.cuh"
#include "omhd_fused3d_pipe.cuh"
#include "omhd_tma.h"

namespace omhd {
// HLLD with minmod or MC where it is selected: the warp-specialised kernel; else the
// one-role kernel
namespace {
bool takes_pipe(const StageArgs& a) {
  return a.flux_type == FX_HLLD && (a.lm_type == LM_MINMOD || a.lm_type == LM_MC) && pipe3d_enabled();
}
}  // namespace
Tiling tiling3d_fp64(const StageArgs& a, int nsm) {
  using namespace v_fp64;
  return takes_pipe(a) ? Tiling{d3p::TX, d3p::TY, d3p::ZC, 1} : d3::tiling3d<double>(a, nsm);
}
int launch_stage3d_fp64(const StageArgs& a, cudaStream_t s) {
  if (takes_pipe(a))
    return v_fp64::d3p::launch_pipe3d<FX_HLLD>(a, s);
  return v_fp64::d3::launch_variant3d<double>(a, s);
}
}  // namespace omhd
