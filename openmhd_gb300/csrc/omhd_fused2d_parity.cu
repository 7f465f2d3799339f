// omhd_fused2d_parity.cu -- 2D fused stage kernels, arithmetic variant "parity"
// (face arithmetic in double; built with --fmad=false so the op sequence is the reference's).
#define OMHD_VARIANT v_parity
#define OMHD_FAST false
#include "omhd_fused2d.cuh"

namespace omhd {
int fill_eta2d_parity(const StageArgs& a, double* etax, double* etay, cudaStream_t s) {
  return v_parity::fill_eta2d(a, etax, etay, s);
}
Tiling tiling2d_parity(const StageArgs& a, int nsm) { return v_parity::tiling_one<double>(a, nsm); }
int launch_stage2d_parity(const StageArgs& a, cudaStream_t s) { return v_parity::launch_variant<double>(a, s); }
}  // namespace omhd
