// FP64 instantiations of the fused stage kernel. Built with -fmad=false:
// every multiply and add rounds separately, as in the reference's x86-64
// build, which keeps the FP64 path bit-compatible with it.
#include "launch.h"

namespace m2c {

cudaError_t launch_stage_fp64(const StageArgs& a, const StageVariant& v, cudaStream_t s) {
  return stage_variant<double>(v, &a, s, nullptr);
}

cudaError_t prepare_stage_fp64(const StageVariant& v, int* resident) {
  return stage_variant<double>(v, nullptr, nullptr, resident);
}

}  // namespace m2c
