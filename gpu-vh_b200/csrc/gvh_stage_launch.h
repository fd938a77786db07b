// gvh_stage_launch.h -- launching one RK substep over one lattice (gvh_rk2_step and
// gvh_rk2_step_noalloc). The stage kernels of each equation of state and precision are compiled
// in a translation unit of their own (gvh_stage_*.cu).
#pragma once

#include <cuda_runtime.h>

#include "../../include/gvh.h"

namespace gvh {

struct StageArgs;

// Raises the shared-memory limit of the two stage kernels that a lattice of ncells takes on the
// current device; before any launch or capture of them. Doing so loads a kernel (0.05 ms and 50 KB
// of device memory each), so a handle prepares its own and not all 96.
cudaError_t prepare_qcd_fp64(int shear, int bulk, long long ncells, long long wave);
cudaError_t prepare_qcd_mixed(int shear, int bulk, long long ncells, long long wave);
cudaError_t prepare_conformal_fp64(int shear, int bulk, long long ncells, long long wave);
cudaError_t prepare_conformal_mixed(int shear, int bulk, long long ncells, long long wave);
inline cudaError_t prepare_stage(int eos, int shear, int bulk, int precision, long long ncells, long long wave) {
  const bool mixed = precision == GVH_PRECISION_MIXED;
  if (eos == GVH_EOS_CONFORMAL)
    return mixed ? prepare_conformal_mixed(shear, bulk, ncells, wave) : prepare_conformal_fp64(shear, bulk, ncells, wave);
  return mixed ? prepare_qcd_mixed(shear, bulk, ncells, wave) : prepare_qcd_fp64(shear, bulk, ncells, wave);
}
// The same for every lattice (gvh_rk2_step_noalloc: its first call on a device is the only one that
// may load kernels). The four sizes are one of each rule in stage_parts.
inline cudaError_t prepare_all_stages(long long wave) {
  cudaError_t e = cudaSuccess;
  for (int eos : {GVH_EOS_QCD, GVH_EOS_CONFORMAL})
    for (int precision : {GVH_PRECISION_FP64, GVH_PRECISION_MIXED})
      for (int physics = 0; physics < 3; ++physics)  // ideal, shear, shear + bulk
        for (long long ncells : {wave / 8, wave / 4, wave / 2, wave})
          if (e == cudaSuccess) e = prepare_stage(eos, physics > 0, physics > 1, precision, ncells, wave);
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
