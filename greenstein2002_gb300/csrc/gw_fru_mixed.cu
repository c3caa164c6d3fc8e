// Mixed-precision cleft-parallel FRU stage kernel: transition rates and the
// FRU-local Ca ODE in FP32 (FP32 issues 64x faster than FP64 on GB300); the
// FRU Ca state, the FRU clock, its step and the cross-FRU flux sums stay FP64.
// The channel algorithm, its MT19937 draw order and the transition rules are
// the FP64 method's (gw_fru_cleft.cuh), so both share every random number.
//
// Reference: simfru_local.c:32-278, fru_rates_local.c:30-798, fcn_fru.c:23-137.
#define GW_CONTRACT
#include "gw_fru_cleft.cuh"

namespace gw {

// Two builds, as in gw_fru_stage4.cu: 178 registers (eight warps per SM) and
// 128 (sixteen).  Alone, five stages with 128 and 178: 1,251 FRUs 0.532 and
// 0.505 ms, 12,500 FRUs 1.415 and 1.370 ms; 16 cells of 12,500 FRUs at once for
// 10 ms: 580 and 891 ms.
__global__ void __launch_bounds__(kMaxStageWarps * 32, 1) fru_stage_mixed_kernel(DevState s, StageParams p, int fpw) {
  cleft::stage_body<float>(s, p, blockIdx.x, s.res, fpw);
}
__global__ void __launch_bounds__(kMaxStageWarps * 32, 2) fru_stage_mixed_dense_kernel(DevState s, StageParams p, int fpw) {
  cleft::stage_body<float>(s, p, blockIdx.x, s.res, fpw);
}

cudaError_t launch_stage_mixed(const DevState& s, const StageParams& p, int warps, int fpw, bool dense, cudaStream_t st) {
  const int blocks = stage_blocks(s.nfru, warps, fpw);
  static const cudaError_t attr = stage_cache_attributes(fru_stage_mixed_kernel);
  static const cudaError_t attr_dense = stage_cache_attributes(fru_stage_mixed_dense_kernel);
  if (attr != cudaSuccess) return attr;
  if (attr_dense != cudaSuccess) return attr_dense;
  if (dense) fru_stage_mixed_dense_kernel<<<blocks, 32 * warps, 0, st>>>(s, p, fpw);
  else fru_stage_mixed_kernel<<<blocks, 32 * warps, 0, st>>>(s, p, fpw);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(kMaxStageWarps * 32) fru_stage_mixed_batch_kernel(BatchArgs a) { cleft::batch_body<float>(a); }

cudaError_t launch_stage_mixed_batch(const BatchArgs& a, int nblocks, int warps, cudaStream_t st) {
  static const cudaError_t attr = stage_cache_attributes(fru_stage_mixed_batch_kernel);
  if (attr != cudaSuccess) return attr;
  fru_stage_mixed_batch_kernel<<<nblocks, 32 * warps, 0, st>>>(a);
  return cudaGetLastError();
}

// 124 registers, sixteen single-warp blocks per SM.  16 cells of 12,500 FRUs
// for 10 ms, 32 FRUs per warp, with a bound of 12 / 14 / 16 / 18 / 20 blocks (151 /
// 124 / 124 / 96 / 96 registers): 528 / 487 / 501 / 562 / 545 ms; equal builds
// differ by 3%, the noise of these figures.
__global__ void __launch_bounds__(32, 14) fru_stage_mixed_packed_kernel(DevState s, StageParams p) {
  cleft::stage_body_packed<float>(s, p, s.res);
}

cudaError_t launch_stage_mixed_packed(const DevState& s, const StageParams& p, int warps, cudaStream_t st) {
  static const cudaError_t attr = stage_cache_attributes(fru_stage_mixed_packed_kernel);
  if (attr != cudaSuccess) return attr;
  fru_stage_mixed_packed_kernel<<<warps, 32, 0, st>>>(s, p);
  return cudaGetLastError();
}

}  // namespace gw
