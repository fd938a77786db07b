// gvh_stage_qcd_mixed.cu -- the stage kernels of the QCD equation of state, mixed precision.
#include "gvh_stage_launch.cuh"

namespace gvh {

cudaError_t prepare_qcd_mixed(int shear, int bulk, long long ncells, long long wave) {
  return prepare_stage_of<EOS_QCD, true>(shear, bulk, ncells, wave);
}
cudaError_t launch_qcd_mixed(const StageArgs &a, int shear, int bulk, bool stage2, long long wave, cudaStream_t st) {
  return launch_stage_of<EOS_QCD, true>(a, shear, bulk, stage2, wave, st);
}

}  // namespace gvh
