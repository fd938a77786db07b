// gvh_stage_qcd_mixed.cu -- the stage kernels of the QCD equation of state, mixed precision.
#include "gvh_stage_launch.cuh"

namespace gvh {

cudaError_t prepare_qcd_mixed() { return prepare_stages_of<EOS_QCD, true>(); }
cudaError_t launch_qcd_mixed(const StageArgs &a, int shear, int bulk, bool stage2, long long wave, cudaStream_t st) {
  return launch_stage_of<EOS_QCD, true>(a, shear, bulk, stage2, wave, st);
}

}  // namespace gvh
