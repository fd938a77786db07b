// gvh_stage_launch.h -- launching one RK substep over one lattice (gvh_rk2_step and
// gvh_rk2_step_noalloc). The stage kernels of each equation of state and precision are compiled
// in a translation unit of their own (gvh_stage_*.cu).
#pragma once

#include <cuda_runtime.h>

#include "../../include/gvh.h"

namespace gvh {

struct StageArgs;

// Raises the stage kernels' shared-memory limits on the current device (once per device, before
// any launch or capture).
cudaError_t prepare_qcd_fp64();
cudaError_t prepare_qcd_mixed();
cudaError_t prepare_conformal_fp64();
cudaError_t prepare_conformal_mixed();
inline cudaError_t prepare_stage_kernels() {
  cudaError_t e = prepare_qcd_fp64();
  if (e == cudaSuccess) e = prepare_qcd_mixed();
  if (e == cudaSuccess) e = prepare_conformal_fp64();
  if (e == cudaSuccess) e = prepare_conformal_mixed();
  return e;
}

// One substep. wave: the cells of one wave of the one-thread-per-cell kernel on this device
// (stage_wave_cells).
cudaError_t launch_qcd_fp64(const StageArgs &a, int shear, int bulk, bool stage2, long long wave, cudaStream_t st);
cudaError_t launch_qcd_mixed(const StageArgs &a, int shear, int bulk, bool stage2, long long wave, cudaStream_t st);
cudaError_t launch_conformal_fp64(const StageArgs &a, int shear, int bulk, bool stage2, long long wave,
                                  cudaStream_t st);
cudaError_t launch_conformal_mixed(const StageArgs &a, int shear, int bulk, bool stage2, long long wave,
                                   cudaStream_t st);
inline cudaError_t launch_stage(int eos, int shear, int bulk, int precision, const StageArgs &a, bool stage2,
                                long long wave, cudaStream_t st) {
  const bool mixed = precision == GVH_PRECISION_MIXED;
  if (eos == GVH_EOS_CONFORMAL)
    return mixed ? launch_conformal_mixed(a, shear, bulk, stage2, wave, st)
                 : launch_conformal_fp64(a, shear, bulk, stage2, wave, st);
  return mixed ? launch_qcd_mixed(a, shear, bulk, stage2, wave, st) : launch_qcd_fp64(a, shear, bulk, stage2, wave, st);
}

}  // namespace gvh
