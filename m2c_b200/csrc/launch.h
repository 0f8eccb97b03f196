// Host-side launchers for the stage kernels, one translation unit per
// precision. The FP64 instantiations live in a unit compiled without FMA
// contraction (-fmad=false) so that their arithmetic rounds like the
// reference's x86-64 build; the mixed instantiations keep contraction on.
#pragma once
#include <cuda_runtime.h>

#include "stage.cuh"

namespace m2c {

// The kernel variant of a stage: two materials (or cut faces), non-primitive
// reconstruction, faces cut by an embedded surface, stiffened gases only.
struct StageVariant {
  int flux;
  bool multi, cons, walls, sg;
};

// Launch one stage on a persistent grid of a.nitems CTAs sharing the work
// evenly; the variant was prepared.
cudaError_t launch_stage_fp64(const StageArgs& a, const StageVariant& v, cudaStream_t s);
cudaError_t launch_stage_mixed(const StageArgs& a, const StageVariant& v, cudaStream_t s);
// Make the variant launchable on the current device (its shared memory) and
// report the CTAs of it that the device holds at once.
cudaError_t prepare_stage_fp64(const StageVariant& v, int* resident);
cudaError_t prepare_stage_mixed(const StageVariant& v, int* resident);

template <typename T, int FLUX, bool MULTI, bool CONS, bool WALLS, bool SG>
cudaError_t stage_one(const StageArgs* a, cudaStream_t s, int* resident) {
  auto k = stage_kernel<T, FLUX, MULTI, CONS, WALLS, SG>;
  const size_t smem = sizeof(StageSmem<T, StageShape<T>::ty, MULTI>);
  const dim3 block(TX, StageShape<T>::warps);
  if (a) {
    k<<<a->nitems, block, smem, s>>>(*a);
    return cudaGetLastError();
  }
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int dev = 0, nsm = 0, per_sm = 0;
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, block.x * block.y, smem);
  if (e == cudaSuccess && per_sm < 1) e = cudaErrorInvalidConfiguration;
  *resident = per_sm * nsm;
  return e;
}

template <typename T, int FLUX>
cudaError_t stage_flux(const StageVariant& v, const StageArgs* a, cudaStream_t s, int* r) {
  if (v.cons) {  // compiled for any equation of state
    if (v.walls) return stage_one<T, FLUX, true, true, true, false>(a, s, r);
    return v.multi ? stage_one<T, FLUX, true, true, false, false>(a, s, r)
                   : stage_one<T, FLUX, false, true, false, false>(a, s, r);
  }
  if (v.walls)
    return v.sg ? stage_one<T, FLUX, true, false, true, true>(a, s, r)
                : stage_one<T, FLUX, true, false, true, false>(a, s, r);
  if (v.multi)
    return v.sg ? stage_one<T, FLUX, true, false, false, true>(a, s, r)
                : stage_one<T, FLUX, true, false, false, false>(a, s, r);
  return v.sg ? stage_one<T, FLUX, false, false, false, true>(a, s, r)
              : stage_one<T, FLUX, false, false, false, false>(a, s, r);
}

// a: launch it; NULL: prepare the variant.
template <typename T>
cudaError_t stage_variant(const StageVariant& v, const StageArgs* a, cudaStream_t s, int* r) {
  switch (v.flux) {
    case FLUX_ROE: return stage_flux<T, FLUX_ROE>(v, a, s, r);
    case FLUX_LLF: return stage_flux<T, FLUX_LLF>(v, a, s, r);
    default: return stage_flux<T, FLUX_HLLC>(v, a, s, r);
  }
}

}  // namespace m2c
