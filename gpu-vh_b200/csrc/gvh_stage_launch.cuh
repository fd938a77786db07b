// gvh_stage_launch.cuh -- the body of a gvh_stage_*.cu: the stage kernels of one equation of state
// and precision, and which of them a lattice takes.
#pragma once

#include "gvh_stage.cuh"
#include "gvh_stage_launch.h"

namespace gvh {

// A lattice smaller than one wave of the one-thread-per-cell kernel (75,776 cells on 148 SMs) takes
// the kernel whose waves it fills best: a wave of PARTS threads per cell holds 1/PARTS of the
// cells and takes about 0.033 ms per step (PARTS = 4), 0.056 (2), 0.097 (1) for QCD with shear
// and bulk, FP64. Measured, ms per step with 4 / 2 / 1: 18,513 cells 0.034 / 0.042 / 0.057;
// 35,301 cells 0.063 / 0.055 / 0.066; 46,575 cells 0.087 / 0.089 / 0.092; 59,823 cells
// 0.121 / 0.105 / 0.101; 81,608 cells 0.150 / 0.136 / 0.130. Eight warps per 32 cells
// (kt_stage_faces_kernel) fill their wave with an eighth: 720 cells 0.0164 ms against 0.0238 with
// PARTS = 4, 3,721 (2+1D) 0.0185 / 0.0260, 9,261 cells 0.0221 / 0.0284. Mixed and conformal order
// alike.
inline int stage_parts(long long ncells, long long wave) {
  if (8 * ncells <= wave) return 8;
  if (4 * ncells <= wave) return 4;
  if (2 * ncells <= wave) return 2;
  if (4 * ncells <= 3 * wave) return 4;
  return 1;
}

template <int EOS, bool SHEAR, bool BULK, bool STAGE2, bool MIXED>
void launch_stage_kernel(const StageArgs &a, int parts, cudaStream_t st) {
  const size_t smem = stage_smem_bytes<SHEAR, BULK>();
  if (parts == 8)
    launch_overlapped(kt_stage_faces_kernel<EOS, SHEAR, BULK, STAGE2, MIXED>, faces_grid(a.ncells), kFaceBlock,
                      faces_smem_bytes<SHEAR, BULK>(), st, a);
  else if (parts == 4)
    launch_overlapped(kt_stage_split_kernel<EOS, SHEAR, BULK, STAGE2, MIXED, 4>, split_grid(a.ncells, 4), kBlock, smem,
                      st, a);
  else if (parts == 2)
    launch_overlapped(kt_stage_split_kernel<EOS, SHEAR, BULK, STAGE2, MIXED, 2>, split_grid(a.ncells, 2), kBlock, smem,
                      st, a);
  else
    launch_overlapped(kt_stage_kernel<EOS, SHEAR, BULK, STAGE2, MIXED>, stage_grid(a.ncells), kBlock, smem, st, a);
}

template <int EOS, bool SHEAR, bool BULK, bool MIXED>
void launch_stage_physics(const StageArgs &a, bool stage2, int parts, cudaStream_t st) {
  if (stage2) launch_stage_kernel<EOS, SHEAR, BULK, true, MIXED>(a, parts, st);
  else launch_stage_kernel<EOS, SHEAR, BULK, false, MIXED>(a, parts, st);
}

template <int EOS, bool MIXED>
cudaError_t launch_stage_of(const StageArgs &a, int shear, int bulk, bool stage2, long long wave, cudaStream_t st) {
  const int parts = stage_parts(a.ncells, wave);
  if (!shear) launch_stage_physics<EOS, false, false, MIXED>(a, stage2, parts, st);
  else if (!bulk) launch_stage_physics<EOS, true, false, MIXED>(a, stage2, parts, st);
  else launch_stage_physics<EOS, true, true, MIXED>(a, stage2, parts, st);
  return cudaGetLastError();
}

template <int EOS, bool MIXED, bool SHEAR, bool BULK, bool STAGE2>
cudaError_t prepare_stage_kernel(int parts) {
  const size_t smem = stage_smem_bytes<SHEAR, BULK>();
  if (parts == 8)
    return allow_stage_smem(kt_stage_faces_kernel<EOS, SHEAR, BULK, STAGE2, MIXED>, faces_smem_bytes<SHEAR, BULK>());
  if (parts == 4) return allow_stage_smem(kt_stage_split_kernel<EOS, SHEAR, BULK, STAGE2, MIXED, 4>, smem);
  if (parts == 2) return allow_stage_smem(kt_stage_split_kernel<EOS, SHEAR, BULK, STAGE2, MIXED, 2>, smem);
  return allow_stage_smem(kt_stage_kernel<EOS, SHEAR, BULK, STAGE2, MIXED>, smem);
}

template <int EOS, bool MIXED, bool SHEAR, bool BULK>
cudaError_t prepare_stage_physics(int parts) {
  const cudaError_t e = prepare_stage_kernel<EOS, MIXED, SHEAR, BULK, false>(parts);
  return e == cudaSuccess ? prepare_stage_kernel<EOS, MIXED, SHEAR, BULK, true>(parts) : e;
}

template <int EOS, bool MIXED>
cudaError_t prepare_stage_of(int shear, int bulk, long long ncells, long long wave) {
  const int parts = stage_parts(ncells, wave);
  if (!shear) return prepare_stage_physics<EOS, MIXED, false, false>(parts);
  if (!bulk) return prepare_stage_physics<EOS, MIXED, true, false>(parts);
  return prepare_stage_physics<EOS, MIXED, true, true>(parts);
}

}  // namespace gvh
