// gvh_stage_conformal_fp64.cu -- the stage kernels of the conformal equation of state, plain FP64.
#include "gvh_stage_launch.cuh"

namespace gvh {

cudaError_t prepare_conformal_fp64(int shear, int bulk, long long ncells, long long wave) {
  return prepare_stage_of<EOS_CONFORMAL, false>(shear, bulk, ncells, wave);
}
cudaError_t launch_conformal_fp64(const StageArgs &a, int shear, int bulk, bool stage2, long long wave, cudaStream_t st) {
  return launch_stage_of<EOS_CONFORMAL, false>(a, shear, bulk, stage2, wave, st);
}

}  // namespace gvh
