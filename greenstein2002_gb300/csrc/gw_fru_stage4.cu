// FP64 cleft-parallel FRU stage kernel (the plain method): the substep loop
// of gw_fru_cleft.cuh instantiated in double.  Compiled with -fmad=false so
// every floating-point operation is the reference's own, rounded once.
//
// Reference: simfru_local.c:32-278 (see gw_fru_cleft.cuh for the mapping).
#include "gw_fru_cleft.cuh"

namespace gw {

// Two builds of the fixed-layout kernel: with the registers it asks for (178:
// two warps per sub-partition, eight per SM) for launches of about one wave,
// and capped at 128 (sixteen per SM) for more (gw_stage_shape.h).  Five stages
// at the peak of release, dense and roomy: 12,500 FRUs 6.82 and 6.07 ms, 250
// FRUs alike.
__global__ void __launch_bounds__(kMaxStageWarps * 32, 1) fru_stage4_kernel(DevState s, StageParams p) {
  cleft::stage_body<double>(s, p, blockIdx.x, s.res);
}
// Two FRUs per warp, sixteen lanes each: the FP64 chain of a substep is shorter
// by the local ODE's (104 to about 55 instructions for an FRU alone in its
// warp), for four times the warps.  Five stages at the peak of release, this
// and the fixed layout (8 FRUs per warp; 4 below 2,500): 250 FRUs 2.36 and 2.79
// ms, 1,250 2.98 and 3.71, 2,500 3.08 and 3.73, 3,000 3.83 and 4.13, 4,000 4.17
// and 4.08.
__global__ void __launch_bounds__(kMaxStageWarps * 32, 1) fru_stage4_wide_kernel(DevState s, StageParams p) {
  cleft::stage_body<double, cleft::WideGroup>(s, p, blockIdx.x, s.res, 2);
}
__global__ void __launch_bounds__(kMaxStageWarps * 32, 2) fru_stage4_dense_kernel(DevState s, StageParams p) {
  cleft::stage_body<double>(s, p, blockIdx.x, s.res);
}

cudaError_t launch_stage4(const DevState& s, const StageParams& p, int warps, bool wide, bool dense, cudaStream_t st) {
  const int blocks = stage_blocks(s.nfru, warps, wide ? 2 : 8);
  static const cudaError_t attr = stage_cache_attributes(fru_stage4_kernel);
  static const cudaError_t attr_dense = stage_cache_attributes(fru_stage4_dense_kernel);
  if (attr != cudaSuccess) return attr;
  if (attr_dense != cudaSuccess) return attr_dense;
  static const cudaError_t attr_wide = stage_cache_attributes(fru_stage4_wide_kernel);
  if (attr_wide != cudaSuccess) return attr_wide;
  if (wide) fru_stage4_wide_kernel<<<blocks, 32 * warps, 0, st>>>(s, p);
  else if (dense) fru_stage4_dense_kernel<<<blocks, 32 * warps, 0, st>>>(s, p);
  else fru_stage4_kernel<<<blocks, 32 * warps, 0, st>>>(s, p);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(kMaxStageWarps * 32) fru_stage4_batch_kernel(BatchArgs a) { cleft::batch_body<double>(a); }

cudaError_t launch_stage4_batch(const BatchArgs& a, int nblocks, int warps, cudaStream_t st) {
  static const cudaError_t attr = stage_cache_attributes(fru_stage4_batch_kernel);
  if (attr != cudaSuccess) return attr;
  fru_stage4_batch_kernel<<<nblocks, 32 * warps, 0, st>>>(a);
  return cudaGetLastError();
}

// A bound of thirteen blocks or more makes the compiler take 128 registers
// (sixteen single-warp blocks per SM; 56 bytes spilled at 13, 28 at 14 and 15, 4
// at 16), of eleven or twelve 168 (twelve blocks).  16 cells of 12,500 FRUs for 2 ms,
// 32 FRUs per warp, at 11 / 12 / 13 / 14 / 15 / 16: 617 / 604 / 584 / 592 / 591 /
// 595 ms; the last four differ by spills and noise.
__global__ void __launch_bounds__(32, 13) fru_stage4_packed_kernel(DevState s, StageParams p) {
  cleft::stage_body_packed<double>(s, p, s.res);
}

cudaError_t launch_stage4_packed(const DevState& s, const StageParams& p, int warps, cudaStream_t st) {
  static const cudaError_t attr = stage_cache_attributes(fru_stage4_packed_kernel);
  if (attr != cudaSuccess) return attr;
  fru_stage4_packed_kernel<<<warps, 32, 0, st>>>(s, p);
  return cudaGetLastError();
}

}  // namespace gw
