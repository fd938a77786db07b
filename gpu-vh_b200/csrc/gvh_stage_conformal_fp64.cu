// gvh_stage_conformal_fp64.cu -- the stage kernels of the conformal equation of state, plain FP64.
#include "gvh_stage_launch.cuh"

namespace gvh {

cudaError_t prepare_conformal_fp64() { return prepare_stages_of<EOS_CONFORMAL, false>(); }
cudaError_t launch_conformal_fp64(const StageArgs &a, int shear, int bulk, bool stage2, long long wave, cudaStream_t st) {
  return launch_stage_of<EOS_CONFORMAL, false>(a, shear, bulk, stage2, wave, st);
}

}  // namespace gvh
