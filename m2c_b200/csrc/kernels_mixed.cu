// Mixed-precision instantiations of the fused stage kernel: reconstruction
// and fluxes in FP32 (FP32 accumulation), while the conserved-state RK
// update, the conservative-to-primitive pressure recovery and the residual
// sum stay FP64 (the recovery p = (gamma-1) rho e - gamma p_inf cancels
// ~1e9 Pa terms down to ~1e5 Pa for water and must not be done in FP32).
#include "launch.h"

namespace m2c {

cudaError_t launch_stage_mixed(const StageArgs& a, const StageVariant& v, cudaStream_t s) {
  return stage_variant<float>(v, &a, s, nullptr);
}

cudaError_t prepare_stage_mixed(const StageVariant& v, int* resident) {
  return stage_variant<float>(v, nullptr, nullptr, resident);
}

}  // namespace m2c
