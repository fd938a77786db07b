// gvh_stage_launch.cuh -- the body of a gvh_stage_*.cu: the stage kernels of one equation of state
// and precision, and which of them a lattice takes.
#pragma once

#include "gvh_stage.cuh"
#include "gvh_stage_launch.h"

namespace gvh {

// A lattice smaller than one wave of the one-thread-per-cell kernel (75,776 cells on 148 SMs) takes
// the kernel whose waves it fills best: a wave of PARTS threads per cell holds 1/PARTS of the cells.
// Measured on a B200, us per step with 8 / 4 / 2 / 1, smooth state:
//    cells    QCD shear + bulk, FP64        mixed                         conformal shear, FP64
//      720     16.3 /  21.9 /  32.5 /  46.1   14.8 /  20.1 /  28.6 /  40.4   13.1 / 18.3 / 26.1 / 38.1
//    9,261     26.6 /  33.1 /  44.5 /  62.1   26.3 /  33.1 /  43.7 /  59.6   16.6 / 21.4 / 28.5 / 41.8
//   13,728     38.1 /  35.3 /  45.4 /  59.4   37.4 /  33.1 /  43.5 /  57.1   28.3 / 24.1 / 30.6 / 43.5
//   18,513     39.0 /  33.6 /  45.7 /  58.8   36.3 /  31.0 /  42.2 /  55.5   30.0 / 24.4 / 31.7 / 43.1
//   26,825     55.4 /  49.1 /  58.7 /  67.0   51.4 /  45.9 /  55.7 /  64.6   42.7 / 40.9 / 37.5 / 47.1
//   35,301     71.9 /  59.0 /  58.9 /  67.6   66.7 /  54.6 /  55.9 /  65.4   55.9 / 44.3 / 37.9 / 47.7
//   46,575     92.1 /  77.1 /  78.3 /  95.7   86.0 /  70.6 /  74.1 /  88.4   69.6 / 59.9 / 59.8 / 63.0
//   59,850    133.1 / 112.7 / 102.5 /  95.8  133.0 / 110.2 /  97.7 /  88.6   92.5 / 76.9 / 64.6 / 63.1
// Past the wave of PARTS = 4 (18,944 cells) its second wave is short and runs with few blocks per SM, so
// it stays the fastest for a while. How long depends on the physics and the state: with bulk up to
// about 3/8 of a wave (28,336 cells, 4 against 2: smooth 56.7 / 58.5, nearly uniform 54.7 / 52.0; 24,000:
// 48.6 / 58.4 and 52.2 / 52.3, hotspots 110 / 117), with shear alone up to 17/64 (20,090 cells: QCD
// 41.0 / 40.1, 45.7 / 48.1, hotspots 49.1 / 54.0), for an ideal fluid not at all (19,440 cells:
// 21.4 / 18.5, hotspots 28.5 / 33.1). An ideal fluid's one-thread kernel is as fast as two threads, or
// up to 18% faster, from 26,825 cells on; the rule does not follow that.
inline int stage_parts(long long ncells, long long wave, int shear, int bulk) {
  if (8 * ncells <= wave) return 8;
  if (64 * ncells <= (bulk ? 24 : shear ? 17 : 16) * wave) return 4;
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
  const int parts = stage_parts(a.ncells, wave, shear, bulk);
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
  const int parts = stage_parts(ncells, wave, shear, bulk);
  if (!shear) return prepare_stage_physics<EOS, MIXED, false, false>(parts);
  if (!bulk) return prepare_stage_physics<EOS, MIXED, true, false>(parts);
  return prepare_stage_physics<EOS, MIXED, true, true>(parts);
}

}  // namespace gvh
