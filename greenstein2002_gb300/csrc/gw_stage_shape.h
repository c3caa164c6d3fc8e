/* Which build of the fixed-layout stage kernels a launch takes, and how many
 * FRUs share a warp.  Every choice gives the same bits. */
#pragma once

namespace gw {

struct StageShape {
  bool dense;  /* the build capped at 128 registers (16 warps per SM), else the roomy one (8 warps) */
  bool wide;   /* FP64: two FRUs per warp, sixteen lanes each (8 warps per SM) */
  int fpw;     /* mixed: FRUs per warp */
};

/* groups: 8-FRU groups in flight over all cells of the device; sms: its
 * multiprocessors; warps: warps per block; advance: the launch runs substeps.
 *
 * Dense and wide.  The roomy and the wide build hold 178 registers, two warps
 * per sub-partition, so 8 warps per SM are resident, and blocks of 2, 4 or 8
 * warps take them up to there: a stage at the peak of release with 10 groups
 * per SM in blocks of 2 / 4 / 8, roomy and dense, FP64 3.57 and 2.86 / 3.72 and
 * 3.01 / 4.18 and 3.83 ms, mixed 0.660 and 0.541 / 0.673 and 0.538 / 0.729 and
 * 0.573; with 10 wide warps per SM, wide and roomy, 2.16 and 1.98 / 2.33 and
 * 1.99 / 2.52 and 2.44.  A launch of single-warp blocks somewhat larger than
 * one wave still loses less with its late blocks than to the denser build:
 * roomy and dense at 8.6 / 10 / 10.9 groups per SM FP64 3.01 and 3.61 / 3.51 and
 * 3.87 / 3.59 and 3.93 ms (at rest 0.319 and 0.367 / 0.421 and 0.437 / 0.411 and
 * 0.401), mixed 0.586 and 0.616 / 0.656 and 0.693 / 0.596 and 0.625; five wide
 * and roomy stages at 9.9 wide warps per SM (3,000 FRUs) 3.83 and 4.13 ms, at
 * 13.2 (4,000) 4.17 and 4.08.
 *
 * fpw.  Fewer FRUs per warp as long as that makes at most four warps per SM
 * (one per sub-partition), because the FRUs of a warp execute each other's
 * branches: five stages at the peak of release with 8, 4, 2 and 1 per warp, 250
 * FRUs 0.651 / 0.630 / 0.614 / 0.609 ms, 1,250 FRUs 0.792 / 0.762 / 0.759 /
 * 0.778, 2,500 FRUs 0.791 / 0.765 / 0.807 / 0.960. */
static inline StageShape stage_shape(int groups, int sms, int warps, bool advance) {
  const int roomy = warps == 1 ? 11 : 8, wide = warps == 1 ? 10 : 8;
  StageShape s;
  s.dense = groups > roomy * sms;
  s.wide = advance && 4 * groups <= wide * sms;
  s.fpw = !advance ? 8 : 4 * groups <= 4 * sms ? 2 : 2 * groups <= 4 * sms ? 4 : 8;
  return s;
}

}  // namespace gw
