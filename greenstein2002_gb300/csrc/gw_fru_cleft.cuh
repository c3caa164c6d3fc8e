// Cleft-parallel FRU substep loop, shared by the FP64 and the mixed-precision
// stage kernels: each FRU is advanced by a group of four lanes, one per
// dyadic cleft (8 FRUs per warp).
//
// Why four lanes per FRU: on GB300 every SM sub-partition issues one FP64
// warp instruction per 64 cycles whatever the active-lane mask, so a stage
// lasts as long as the FP64 instruction chain of its slowest FRU.  Spreading an
// FRU over its clefts divides that chain by about four at the same total work.
//
// R = double: the plain FP64 method.  Every operation is the reference's, in
// its order, arranged to issue few FP64 instructions (what bounds the
// kernels).  Sums and products are rounded as the reference rounds them;
//   - quotients, reciprocals and exponentials are those of gw_fp64_math.cuh:
//     quotients correctly rounded unless within 2^-37 of a last place of a
//     midpoint, exponentials to 0.52 of a last place;
//   - max/min/compares of non-negative doubles on their bit patterns;
//   - rates are estimated in FP32 and formed in FP64 only where the estimate
//     leaves a decision open: which rate is the largest (when 0.1 over it is
//     below the substep's cap) and which side of its threshold a draw is on;
//     there 1 - dt*rate is compared with the draw in the integer domain
//     (u = y/2^32 > P  <=>  y > floor(P*2^32));
//   - products with 0/1 flags are selections, halvings are folded into FMAs
//     (both exact), the three interpolated voltages/concentrations are
//     computed one per lane, and exp(2VF/RT) at the end of a substep is reused
//     at the start of the next (and at the stage start computed once per
//     lane, not per FRU).
// R = float: the mixed-precision method.  Transition rates, the local Ca ODE
// and the FRU clock are evaluated in FP32, the Ca states and the clock
// accumulated as compensated FP32 pairs; FP64 is kept for the FRU arrays in
// memory and for the cross-FRU flux sums.  Channel transitions use the
// complement form 1 - u < dt*rate, which keeps full resolution near u = 1.
//
// MT19937 rows are drawn from and regenerated in place, in the FRU's own
// row in global memory (L1-cached; the kernels use no shared memory): on
// GB300 this ran as fast as staging the eight rows of a warp in shared
// memory for FP64 and 15% faster for mixed precision, whose warps the
// staging's 20 KB per warp had held to eleven per SM.
//
// Reference: simfru_local.c:32-278, fru_rates_local.c:30-798, fcn_fru.c:23-137,
// mt19937_local.c:97-240.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "gw_fp64_math.cuh"
#include "gw_fru_core.cuh"
#include "gw_fru_model.cuh"
#include "gw_kernels.h"

namespace gw {
namespace cleft {

// ---- type-specific operations ----------------------------------------------
__device__ __forceinline__ long long ord(double a) { return __double_as_longlong(a); }
__device__ __forceinline__ int ord(float a) { return __float_as_int(a); }
// max/min of values known to be >= 0 (or of a negative value against a
// positive constant): IEEE order equals the signed integer order of the bits;
// ties return the first argument like the reference's macros
template <typename R>
__device__ __forceinline__ R imax(R a, R b) { return ord(a) < ord(b) ? b : a; }
template <typename R>
__device__ __forceinline__ R imin(R a, R b) { return ord(a) < ord(b) ? a : b; }
template <typename R>
__device__ __forceinline__ bool ilt(R a, R b) { return ord(a) < ord(b); }
// |v| < c for a positive constant c, on the integer pipe
__device__ __forceinline__ bool abs_lt(double v, double c) {
  return (__double_as_longlong(v) & 0x7fffffffffffffffLL) < __double_as_longlong(c);
}
__device__ __forceinline__ bool abs_lt(float v, float c) { return (__float_as_int(v) & 0x7fffffff) < __float_as_int(c); }

// FP32 (the mixed-precision method): division by a constant as a product,
// rdiv the fast approximate quotient, qdiv the correctly rounded one.
__device__ __forceinline__ float divc(float x, float d, float r) { return x * r; }
__device__ __forceinline__ float rdiv(float a, float b) { return __fdividef(a, b); }
__device__ __forceinline__ float qdiv(float a, float b) { return a / b; }
__device__ __forceinline__ float rexp(float x) { return expf(x); }
// e = exp(x) and the GHK denominator e - 1 by expm1f, because expf(x) - 1
// keeps almost no relative precision for the |x| < 1e-5 of membrane
// potentials within a few tenths of a mV of zero, and is exactly 0 for
// potentials of a few uV (just above the 1e-6 mV of the reference's V = 0
// branch), which made the GHK factor infinite.
__device__ __forceinline__ void exp_em1(float x, float& e, float& em1) {
  em1 = expm1f(x);
  e = 1.0f + em1;
}

// FP64: u = y/2^32 compared with P = 1 - dt*R in the integer domain.
__device__ __forceinline__ void thresh(double P, uint64_t& fl, bool& exact) {
  const uint64_t b = (uint64_t)__double_as_longlong(P);
  const int e = (int)((b >> 52) & 0x7ff) - 1023;
  const uint64_t M = (b & 0xfffffffffffffull) | (1ull << 52);
  const int sh = 20 - e;  // floor(P * 2^32) = M >> (52 - 32 - e)
  if (sh >= 64) {
    fl = 0;
    exact = false;
  } else {
    fl = M >> sh;
    exact = (M & ((1ull << sh) - 1ull)) == 0ull;
  }
}
__device__ __forceinline__ bool nonpos(double P) { return __double_as_longlong(P) <= 0LL; }  // P <= 0 (not NaN)
// y/2^32 > P (LCC, RyR) and y/2^32 >= P (VDI gate, Cl channel)
__device__ __forceinline__ bool u_above(uint32_t y, double P) {
  if (nonpos(P)) return true;  // never on valid input (dt*rate <= 0.1)
  uint64_t fl;
  bool ex;
  thresh(P, fl, ex);
  return (uint64_t)y > fl;
}
__device__ __forceinline__ bool u_reaches(uint32_t y, double P) {
  if (nonpos(P)) return true;
  uint64_t fl;
  bool ex;
  thresh(P, fl, ex);
  return (uint64_t)y > fl || (ex && (uint64_t)y == fl);
}
// 2^32 - y rounded to FP32, from a 32-bit conversion: the same value as
// converting the 33-bit integer, without a 64-bit integer conversion, which
// runs on the FP64 pipe.  (0 - y is 2^32 - y for y > 0; for y = 0, y = 1 rounds
// to 2^32 too.)
__device__ __forceinline__ float comp_u32(uint32_t y) { return (float)(0u - max(y, 1u)); }
// FP32: complement form, 1 - u = (2^32 - y)/2^32 against dt*R, dts = dt 2^32
__device__ __forceinline__ bool leave_gt(uint32_t y, float dts, float R) { return comp_u32(y) < dts * R; }
__device__ __forceinline__ bool leave_ge(uint32_t y, float dts, float R) { return comp_u32(y) <= dts * R; }

// Destination of a channel that leaves its state (simfru_local.c:215-253) in
// FP32: walks the remaining exit mass against 1 - u = (2^32 - y)/2^32, which
// keeps full resolution near u = 1 where the walk happens.
__device__ __forceinline__ int choose_dest(const float r[4], const int d[4], int len, float dt, uint32_t y) {
  const float c = comp_u32(y) * 2.3283064365386963e-10f;
  float rem = dt * r[0] - dt * r[1];
  int n = 1;
  while (c < rem && n + 1 < len) {
    n++;
    rem = rem - dt * r[n];
  }
  return d[n];
}

// u = y/2^32 < p for 0 < p < 1 (pseudo-state draws, fru_rates_local.c):
// FP64 in the integer domain (u < p <=> y < p*2^32); FP32 directly
__device__ __forceinline__ bool u_below(uint32_t y, double p) {
  if (nonpos(p)) return false;
  uint64_t fl;
  bool ex;
  thresh(p, fl, ex);
  return ex ? (uint64_t)y < fl : (uint64_t)y <= fl;
}
__device__ __forceinline__ bool u_below(uint32_t y, float p) { return (float)y * 2.3283064365386963e-10f < p; }

// LCC exit total = (cX*bX + cY*bY) + cZ*bZ with bases {1, alpha, beta,
// gamma, alpha', beta'}: the sums of fru_rates_local.c:176-340 in their order.
__constant__ float c_lcc_coef[13][3] = {
    {0.0f, 0.0f, 0.0f},
    {4.0f, 1.0f, 0.0f},                     // 1: 4a + g
    {1.0f, 3.0f, (float)(aL)},                      // 2: b + 3a + aL g
    {2.0f, 2.0f, (float)(aL * aL)},                 // 3
    {3.0f, 1.0f, (float)(aL * aL * aL)},            // 4
    {4.0f, (float)(fL), (float)(aL * aL * aL * aL)},        // 5
    {(float)(gL), 0.0f, 0.0f},                      // 6
    {4.0f, (float)(CCa0_to_C0), 0.0f},              // 7: 4a' + omega
    {1.0f, 3.0f, (float)(CCa1_to_C1)},              // 8: b' + 3a' + omega/bL
    {2.0f, 2.0f, (float)(CCa2_to_C2)},              // 9
    {3.0f, 1.0f, (float)(CCa3_to_C3)},              // 10
    {4.0f, (float)(CCa4_to_C4), (float)(fLprime)},          // 11
    {(float)(gLprime), 0.0f, 0.0f},                 // 12
};
// basis index of each term, packed 3 x 4 bits per state:
// 0 = 1, 1 = alpha, 2 = beta, 3 = gamma, 4 = alpha', 5 = beta'
__constant__ uint16_t c_lcc_basis[13] = {
    0x000, 0x031, 0x312, 0x312, 0x312, 0x302, 0x000, 0x004, 0x045, 0x045, 0x045, 0x005, 0x000,
};

template <typename R>
__device__ __forceinline__ R pick_basis(int i, R al, R be, R ga, R ap, R bp) {
  R v = R(1);
  v = (i == 1) ? al : v;
  v = (i == 2) ? be : v;
  v = (i == 3) ? ga : v;
  v = (i == 4) ? ap : v;
  v = (i == 5) ? bp : v;
  return v;
}

struct Group {
  int c;           // cleft of this lane (0..3)
  int base;        // lane index of cleft 0 of this FRU within the warp
  unsigned mask;   // the lanes of this FRU
  int q = 0;       // sixteen lanes per FRU: this lane's copy of the cleft (0..3)
};
// Sixteen lanes per FRU (FP64 launches of few FRUs, whose other lanes would
// idle): four copies of each cleft's lane run the substep alike and share the
// FP64 work of the local ODE; copy 0 stores.
struct WideGroup : Group {};
template <typename G>
struct is_wide {
  static constexpr bool value = false;
};
template <>
struct is_wide<WideGroup> {
  static constexpr bool value = true;
};

// group-local shuffles (the four lanes of one FRU may run while other
// groups of the warp have finished their substeps)
template <typename T>
__device__ __forceinline__ T from(const Group& g, T v, int c) {
  return __shfl_sync(g.mask, v, g.base + c);
}
template <typename R>
__device__ __forceinline__ R gmax(const Group& g, R v) {
  v = imax(v, __shfl_xor_sync(g.mask, v, 1));
  v = imax(v, __shfl_xor_sync(g.mask, v, 2));
  return v;
}

// Words k0 .. k0 + 32*STEPS - 1 of a row's regeneration (below 624), by the
// warp: every lane reads all its words before the barrier and writes after it.
template <int STEPS>
__device__ __forceinline__ void regen_chunk(uint32_t* m, int k0, int lane) {
  uint32_t nw[STEPS];
#pragma unroll
  for (int j = 0; j < STEPS; j++) {
    const int k = k0 + 32 * j + lane;
    if (k < kMtN) {
      const uint32_t cur = m[k];
      const uint32_t nxt = m[(k + 1 == kMtN) ? 0 : k + 1];
      const uint32_t far = m[(k + kMtM < kMtN) ? k + kMtM : k + kMtM - kMtN];
      const uint32_t y = (cur & 0x80000000u) | (nxt & 0x7fffffffu);
      nw[j] = far ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
    }
  }
  __syncwarp();
#pragma unroll
  for (int j = 0; j < STEPS; j++) {
    const int k = k0 + 32 * j + lane;
    if (k < kMtN) m[k] = nw[j];
  }
  __syncwarp();
}
// In-place regeneration of one FRU's 624 words (mt19937_local.c:97-154) by
// all 32 lanes of the warp, in three chunks of 224, 224 and 176 words whose
// loads are all in flight together: word k < 227 reads the old word k + 397,
// word k >= 227 the new word k - 227, which is in an earlier chunk, and word
// 623 the new words 0 and 396, as in the sequential loop.  (One step of 32
// words after another waited for 20 loads in turn.)
__device__ __forceinline__ void regen32(uint32_t* m, int lane) {
  regen_chunk<7>(m, 0, lane);
  regen_chunk<7>(m, 224, lane);
  regen_chunk<6>(m, 448, lane);
}
// 624 words in 16-byte pieces by the group's 4 lanes (rows 16-byte aligned)
__device__ __forceinline__ void copy_row16(uint32_t* dst, const uint32_t* src, const Group& g) {
  const uint4* s4 = reinterpret_cast<const uint4*>(src);
  uint4* d4 = reinterpret_cast<uint4*>(dst);
  for (int i = g.c; i < kMtN / 4; i += 4) d4[i] = s4[i];
  __syncwarp(g.mask);
}

// The five RyR states of a channel word as masks over their nibbles (bit 0 of
// nibble i set when RyR i is in the state).
struct RyrMasks {
  uint32_t s1, s2, s3, s4, s5, s6, s7, s8;
};
__device__ __forceinline__ RyrMasks ryr_masks(uint32_t w) {
  const uint32_t r = w >> 8;
  const uint32_t b0 = r & 0x11111u, b1 = (r >> 1) & 0x11111u, b2 = (r >> 2) & 0x11111u;
  RyrMasks m;
  m.s1 = b0 & ~b1 & ~b2;
  m.s2 = ~b0 & b1 & ~b2;
  m.s3 = b0 & b1 & ~b2;
  m.s4 = ~b0 & ~b1 & b2;
  m.s5 = b0 & ~b1 & b2;
  m.s6 = ~b0 & b1 & b2;
  m.s7 = b0 & b1 & b2;
  m.s8 = (r >> 3) & 0x11111u;
  return m;
}
// The extra draws of a substep: regime 0 resolves RyR states 7 and 8,
// regime 1 resolves 7 (in cleft, then RyR order).  exmask: this lane's RyRs
// that draw (bit 0 of their nibbles), ne their number, pre the draws of the
// clefts before, etot the FRU's.  The four counts travel as the bytes of one
// word, and with them two flags of each cleft; any: their union over the FRU.
// (Votes of the four lanes are taken by one group of the warp after another;
// with the flags here instead of two votes an FP64 substep is 2% faster.)
__device__ __forceinline__ void draw_layout(const Group& g, uint32_t w, int regime, uint32_t flags, uint32_t& exmask,
                                            int& ne, int& pre, int& etot, uint32_t& any) {
  const RyrMasks m = ryr_masks(w);
  exmask = (regime == 0) ? (m.s7 | m.s8) : (regime == 1) ? m.s7 : 0u;
  ne = __popc(exmask);
  uint32_t n = ((uint32_t)ne | (flags << 4)) << (8 * g.c);
  n |= __shfl_xor_sync(g.mask, n, 1);
  n |= __shfl_xor_sync(g.mask, n, 2);
  any = ((n & 0x10101010u) ? 1u : 0u) | ((n & 0x20202020u) ? 2u : 0u);
  n &= 0x07070707u;
  etot = (int)((n * 0x01010101u) >> 24);
  pre = (int)(((n & ((1u << (8 * g.c)) - 1u)) * 0x01010101u) >> 24);
}
// merged RyR states: 3, 4 -> 7 in regime 2; 5, 6 -> 8 in regimes 1 and 2
__device__ __forceinline__ uint32_t merge_ryr(uint32_t w, int regime) {
  const RyrMasks m = ryr_masks(w);
  const uint32_t c7 = (regime == 2) ? (m.s3 | m.s4) << 8 : 0u, c8 = (regime != 0) ? (m.s5 | m.s6) << 8 : 0u;
  return (w & ~((c7 | c8) * 15u)) | (c7 * 7u) | (c8 << 3);
}
__device__ __forceinline__ int ryr_open_masked(uint32_t w) {
  const RyrMasks m = ryr_masks(w);
  return __popc(m.s3 | m.s4 | m.s7);
}

// The launch's view of one warp's 8 FRUs: each lane's FRU row (in place,
// global memory) and the copy-on-twist rows of the cell.
struct StageCtx {
  const StageParams* p;
  uint32_t* m;               // this lane's FRU row
  uint32_t* hold_base;       // copy-on-twist rows of the cell, FRU-major
  uint32_t* hold_epoch_base; // their epochs
  uint32_t* my_hold_epoch;   // the epoch of this lane's FRU
  int f;                     // this lane's FRU (any value for a group without one)
};

// Point the group at its FRU's row; on a resume whose epoch's snapshot
// holds the row's words from before its last regeneration, put them back
// first (send_resume_state's MT restore, mpi_slave.c:150-184).
__device__ __forceinline__ void use_row(StageCtx& sc, uint32_t* row, const uint32_t* hold, bool restore,
                                        const Group& g) {
  if (restore) copy_row16(row, hold, g);
  sc.m = row;
}

// The words of one substep are E_tot extra draws (lane c owns positions
// pre .. pre+ne-1) followed by the 32 batch draws (lane c owns 8c .. 8c+7).
// fetch_old reads those below word 624; regen_crossing then regenerates, with
// the whole warp, the rows whose draws run past it; fetch_new reads the rest
// from the new generation, tempers, and advances mti.
__device__ __forceinline__ void fetch_old(const StageCtx& sc, const Group& g, int mti, int pre, int ne, int etot,
                                          uint32_t ex[kRyR], uint32_t bw[8]) {
  if (ne) {
#pragma unroll
    for (int i = 0; i < kRyR; i++) {
      const int pos = mti + pre + i;
      if (i < ne && pos < kMtN) ex[i] = sc.m[pos];
    }
  }
  const uint32_t* m = sc.m + (mti + etot + 8 * g.c);
  if (mti + etot + 32 <= kMtN) {
#pragma unroll
    for (int k = 0; k < 8; k++) bw[k] = m[k];
  } else {
#pragma unroll
    for (int k = 0; k < 8; k++)
      if (mti + etot + 8 * g.c + k < kMtN) bw[k] = m[k];
  }
}

// cross / copy: the bit of a group's first lane (regen_step's ballots) is set
// when the group regenerates its row / first copies its words of before to its
// hold row in this epoch.
__device__ __forceinline__ void regen_crossing(const StageCtx& sc, int lane, unsigned cross, unsigned copy) {
  while (cross) {
    const int l0 = __ffs(cross) - 1;
    cross &= cross - 1u;
    uint32_t* row = reinterpret_cast<uint32_t*>(__shfl_sync(0xffffffffu, (unsigned long long)sc.m, l0));
    const int fg = __shfl_sync(0xffffffffu, sc.f, l0);  // the FRU of lane l0's group
    __syncwarp();  // the group has read its old words
    if (copy & (1u << l0)) {
      const uint4* s4 = reinterpret_cast<const uint4*>(row);
      uint4* d4 = reinterpret_cast<uint4*>(sc.hold_base + (size_t)fg * kMtStride);
      for (int i = lane; i < kMtN / 4; i += 32) d4[i] = s4[i];
      if (lane == 0) sc.hold_epoch_base[fg] = sc.p->epoch;
    }
    regen32(row, lane);
  }
}

__device__ __forceinline__ void fetch_new(const StageCtx& sc, const Group& g, int& mti, int pre, int ne, int etot,
                                          uint32_t ex[kRyR], uint32_t bw[8]) {
  const int W = etot + 32;
  if (mti + W > kMtN) {
#pragma unroll
    for (int i = 0; i < kRyR; i++) {
      const int pos = mti + pre + i;
      if (i < ne && pos >= kMtN) ex[i] = sc.m[pos - kMtN];
    }
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int pos = mti + etot + 8 * g.c + k;
      if (pos >= kMtN) bw[k] = sc.m[pos - kMtN];
    }
    mti = mti + W - kMtN;
  } else {
    mti = mti + W;
  }
  if (ne) {
#pragma unroll
    for (int i = 0; i < kRyR; i++) ex[i] = mt_temper(ex[i]);
  }
#pragma unroll
  for (int k = 0; k < 8; k++) bw[k] = mt_temper(bw[k]);
}

// JRyRmax * (R)n for n = 0..5 open RyRs, by selection instead of a
// conversion and a multiply (the products are the same rounded values)
template <typename R>
__device__ __forceinline__ R jryr_coef(int n) {
  R v = R(0);
  v = (n == 1) ? R(JRyRmax) * R(1) : v;
  v = (n == 2) ? R(JRyRmax) * R(2) : v;
  v = (n == 3) ? R(JRyRmax) * R(3) : v;
  v = (n == 4) ? R(JRyRmax) * R(4) : v;
  v = (n == 5) ? R(JRyRmax) * R(5) : v;
  return v;
}

// Local Ca ODE of one cleft (fcn_fru.c:23-137) evaluated by the FRU's four
// lanes.  Each lane returns dCaSS of its cleft; every lane returns the same
// dCaJSR.  e2 = exp(2 V F/RT) and a2j are passed in (shared by all lanes).
template <typename R>
__device__ __forceinline__ void fcn_fru4(const Group& g, R cajsr, R cass, const R dep[3], R e2, R a2j, bool small,
                                         R lopen, int nopen, R pca_scale, R& dJSR, R& dSS) {
  constexpr double JDHconstant = 1.0 / (2.0 * VSS * Faraday * 1000.0);
  constexpr double KJDHsmall = -PCa * 2.0 * 1000.0 * Faraday;
  const R Cai = dep[1], CaNSR = dep[2];
  // JRyR of every cleft, summed in cleft order
  const R jcoef = jryr_coef<R>(nopen);
  const R JRyR = jcoef * (cajsr - cass);
  const R j0 = from(g, JRyR, 0), j1 = from(g, JRyR, 1), j2 = from(g, JRyR, 2), j3 = from(g, JRyR, 3);
  const R JRyRtot = j0 + j1 + j2 + j3;
  const R cnext = from(g, cass, (g.c + 1) & 3);
  const R Jss = divc(cass - cnext, R(tauss2ss), R(1.0 / tauss2ss));
  const R Jss_prev = from(g, Jss, (g.c + 3) & 3);
  const R Jxfer = divc(cass - Cai, R(tauxfer), R(1.0 / tauxfer));
  R JDH;
  if (small) JDH = R(KJDHsmall) * pca_scale * (cass - R(Cao * 0.341)) * lopen * R(JDHconstant);
  else JDH = -(cass * e2 - R(Cao * 0.341)) * a2j * lopen;
  R a1 = rdiv(R(BSRtot * KBSR), (cass + R(KBSR)) * (cass + R(KBSR)));
  R a2 = rdiv(R(BSLtot * KBSL), (cass + R(KBSL)) * (cass + R(KBSL)));
  const R bSS = rdiv(R(1), R(1) + a1 + a2);
  dSS = bSS * (JDH + JRyR - Jxfer - Jss + Jss_prev);
  const R Jtr = divc(CaNSR - cajsr, R(tautr), R(1.0 / tautr));
  a1 = rdiv(R(CSQNtot * KmCSQN), (cajsr + R(KmCSQN)) * (cajsr + R(KmCSQN)));
  const R bJSR = rdiv(R(1), R(1) + a1);
  dJSR = bJSR * (Jtr - R(VSS / VJSR) * JRyRtot);
}

// exp(2 V F / RT) and the GHK factor a2 of fcn_fru.c:78-101 for voltage V
template <typename R>
__device__ __forceinline__ void ghk_terms(R V, R pca_scale, R& e2, R& a2j, bool& small) {
  constexpr double JDHconstant = 1.0 / (2.0 * VSS * Faraday * 1000.0);
  const R VFRT = divc(V, R(RT_over_F), R(1.0 / RT_over_F));
  const R VFsqRT = R(1000.0 * Faraday) * VFRT;
  R em1;
  exp_em1(R(2) * VFRT, e2, em1);
  small = abs_lt(V, R(1.e-6));
  if (small) a2j = R(0);
  else a2j = rdiv(R(PCa * 4.0) * pca_scale * VFsqRT, em1) * R(JDHconstant);
}

// The constants of one lane for a stage (the same for every FRU of it).
template <typename R>
struct LaneStage {
  R dep0[3], span[3], pca_scale, rinterval;
  double t0, tf, interval;
  float ihi, ilo;  // the interval as a compensated FP32 pair (the mixed-precision clock)
  // per-lane voltage exponential of the rates: alpha, beta, yCa_inf, tau_yCa
  //   lane 0: alphacf*exp(0.012*(V-35))     lane 1: betacf*exp(-0.05*(V-35))
  //   lane 2: 0.4/(1+exp((V+12.5)/5)) + 0.6  lane 3: 60 + 340/(1+exp((V+30)/12))
  bool isdiv;
  R cA, cR, cD, cCF, cK, cM;
};

template <typename R>
__device__ __forceinline__ void lane_stage(const StageParams& p, const Group& g, LaneStage<R>& L) {
#pragma unroll
  for (int i = 0; i < 3; i++) {
    L.dep0[i] = (R)p.dep0[i];
    L.span[i] = (R)p.span[i];
  }
  L.pca_scale = (R)p.pca_scale;
  L.t0 = p.t0;
  L.tf = p.tf;
  L.interval = p.tf - p.t0;
  L.rinterval = (R)(1.0 / L.interval);
  L.ihi = (float)L.interval;
  L.ilo = (float)(L.interval - (double)L.ihi);
  L.isdiv = g.c >= 2;
  L.cA = L.isdiv ? (g.c == 2 ? R(12.5) : R(30.0)) : R(-35.0);
  L.cR = L.isdiv ? (g.c == 2 ? R(1.0 / 5.0) : R(1.0 / 12.0)) : (g.c == 0 ? R(0.012) : R(-0.05));
  L.cD = L.isdiv ? (g.c == 2 ? R(5.0) : R(12.0)) : R(1.0);
  L.cCF = L.isdiv ? R(0.0) : (g.c == 0 ? R(alphacf) : R(betacf));
  L.cK = L.isdiv ? (g.c == 2 ? R(0.4) : R(340.0)) : R(1.0);
  L.cM = L.isdiv ? (g.c == 2 ? R(1.0 - 0.4) : R(60.0)) : R(0.0);
}

// FP64: exp(2VF/RT) and the GHK factor a2 of fcn_fru.c:78-101 for voltage V
// (any V and scale: beyond +-500 mV or a scale near the ends of the exponent
// range the hardware's division).  The reference's LCC flux is a product with
// the open flag, NaN for closed channels too where a factor is not finite; the
// local ODE selects by the flag, so there Cai, which every cleft's flux takes,
// becomes NaN instead (the product or a test in the ODE cost 1% of a stage).
__device__ __forceinline__ void ghk_terms(double V, double pca4, double& e2, double& a2j, bool& small, double& cai) {
  constexpr double JDHconstant = 1.0 / (2.0 * VSS * Faraday * 1000.0);
  // 2VF/RT is V over half the divisor and 1000 F VF/RT half of 1000 F times
  // it: exact scalings by two of the reference's products
  const double VF2 = fma(V, 2.0 * kDivRTF.rhi, V * (2.0 * kDivRTF.rlo));
  const double VFsqRT = (500.0 * Faraday) * VF2;
  e2 = fexp(VF2);
  small = abs_lt(V, 1.e-6);
  a2j = 0.0;
  if (!small) {
    const double num = pca4 * VFsqRT, em1 = e2 - 1.0;
    if (abs_lt(V, 500.0) && fits(pca4)) {
      a2j = fast_div(num, em1) * JDHconstant;
    } else {
      a2j = num / em1 * JDHconstant;
      if (!isfinite(e2) || !isfinite(a2j)) cai = __longlong_as_double(0x7ff8000000000000ll);
    }
  }
}

template <>
struct LaneStage<double> {
  double dep0[3], myspan, mydep0;  // V, Cai, CaNSR at t0; the one this lane interpolates (cleft % 3)
  double pca4, pca2;               // LCC permeability factors of the GHK and the V = 0 form
  double t0, tf, interval, rhi, rlo;  // rhi + rlo = 1/interval to about 105 bits
  double e2, a2j;                  // ghk_terms at t0
  bool small, isdiv, tpos;         // tpos: times are >= 0 (and tf is not NaN)
  float cA, cR, cCF, cK, cM;       // per-lane voltage exponential in FP32 (see LaneStage<R>)
};
__device__ __forceinline__ void lane_stage(const StageParams& p, const Group& g, LaneStage<double>& L) {
#pragma unroll
  for (int i = 0; i < 3; i++) L.dep0[i] = p.dep0[i];
  L.mydep0 = g.c == 1 ? p.dep0[1] : g.c == 2 ? p.dep0[2] : p.dep0[0];
  L.myspan = g.c == 1 ? p.span[1] : g.c == 2 ? p.span[2] : p.span[0];
  L.pca4 = (PCa * 4.0) * p.pca_scale;
  L.pca2 = (-PCa * 2.0 * 1000.0 * Faraday) * p.pca_scale;
  L.t0 = p.t0;
  L.tf = p.tf;
  L.tpos = ord(p.t0) >= 0 && p.tf >= 0.0;
  L.interval = p.tf - p.t0;
  L.rhi = 1.0 / L.interval;
  L.rlo = fma(-L.interval, L.rhi, 1.0) * L.rhi;
  ghk_terms(L.dep0[0], L.pca4, L.e2, L.a2j, L.small, L.dep0[1]);
  L.isdiv = g.c >= 2;
  L.cA = L.isdiv ? (g.c == 2 ? 12.5f : 30.0f) : -35.0f;
  L.cR = L.isdiv ? (g.c == 2 ? 1.0f / 5.0f : 1.0f / 12.0f) : (g.c == 0 ? 0.012f : -0.05f);
  L.cCF = g.c == 0 ? (float)alphacf : (float)betacf;
  L.cK = g.c == 2 ? 0.4f : 340.0f;
  L.cM = g.c == 2 ? 0.6f : 60.0f;
}

// Accumulator of an FRU Ca concentration over the substeps.  FP64: a double,
// updated as the reference does.  Mixed precision: a compensated FP32 pair
// (Neumaier's summation: hi + lo carries about 48 bits), so the FP32
// increments accumulate without FP64 instructions or conversions in the
// substep loop; the FRU arrays stay FP64 (split on load, joined on store).
template <typename R>
struct CaAcc;
template <>
struct CaAcc<double> {
  double v;
  __device__ __forceinline__ void set(double x) { v = x; }
  __device__ __forceinline__ double get() const { return v; }
  __device__ __forceinline__ double r() const { return v; }
  __device__ __forceinline__ void add(double inc) { v = v + inc; }
};
template <>
struct CaAcc<float> {
  float hi, lo;
  __device__ __forceinline__ void set(double x) {
    hi = (float)x;
    lo = (float)(x - (double)hi);
  }
  __device__ __forceinline__ double get() const { return (double)hi + (double)lo; }
  __device__ __forceinline__ float r() const { return hi + lo; }
  __device__ __forceinline__ void add(float inc) {
    const float t = hi + inc;
    lo = lo + ((fabsf(hi) >= fabsf(inc)) ? (hi - t) + inc : (inc - t) + hi);
    hi = t;
  }
};

// The FRU's clock over [t0, tf] (simfru_local.c:135-146, :161): the step of
// a substep is dt = min(dt_rate, tf - t), so the last substep lands on tf.
// FP64: the reference's time_FRU, an FP64 time (t + (tf - t) is exactly tf,
// as both are close).  Mixed precision: the time since t0 as a compensated
// FP32 pair (about 48 bits, far finer than any substep of a stage of at most
// 0.1 ms), the last substep taking exactly the time that remains -- no FP64
// instruction or conversion in the substep loop.
template <typename R>
struct FruClock;
template <>
struct FruClock<double> {
  double t;
  __device__ __forceinline__ void begin(const LaneStage<double>& L) { t = L.t0; }
  // t < tf; for times >= 0 on their bit patterns
  __device__ __forceinline__ bool running(const LaneStage<double>& L) const {
    return L.tpos ? ilt(t, L.tf) : t < L.tf;
  }
  __device__ __forceinline__ double advance(double dtr, const LaneStage<double>& L) {
    const double dt64 = imin(dtr, L.tf - t);
    t = t + dt64;
    return dt64;
  }
  // (t - t0) / interval, by the two-instruction division with the stage's own
  // reciprocal: the quotient is known to 2^-105 before its last rounding
  __device__ __forceinline__ double frac(const LaneStage<double>& L) const {
    const double x = t - L.t0;
    return fma(x, L.rhi, x * L.rlo);
  }
};
template <>
struct FruClock<float> {
  float hi, lo;  // time since t0
  bool fin;      // the FRU has reached tf
  __device__ __forceinline__ void begin(const LaneStage<float>& L) {
    hi = 0.0f;
    lo = 0.0f;
    fin = !(L.interval > 0.0);
  }
  __device__ __forceinline__ bool running(const LaneStage<float>&) const { return !fin; }
  __device__ __forceinline__ float advance(float dtr, const LaneStage<float>& L) {
    const float rem = (L.ihi - hi) + (L.ilo - lo);
    if (!(dtr < rem)) {
      fin = true;
      hi = L.ihi;
      lo = L.ilo;
      return rem;
    }
    const float s = hi + dtr;  // Knuth's two-sum of hi and dtr
    const float b = s - hi;
    lo = lo + ((hi - (s - b)) + (dtr - b));
    hi = s;
    return dtr;
  }
  __device__ __forceinline__ float frac(const LaneStage<float>& L) const { return (hi + lo) * L.rinterval; }
};

// One FRU's state in the substep loop, as seen by one lane (its cleft):
// the FRU Ca state and clock, channel word, MT position, and the values
// carried from one substep to the next.
template <typename R>
struct Fru4 {
  FruClock<R> clk;
  CaAcc<R> jsr, ss;  // CaJSR and this cleft's CaSS
  uint32_t w, nsub;
  int mti, nopen;
  R dep[3], e2, a2j, lopen;
  bool small;
};

// the FRU at the stage start (t0, voltages dep0)
template <typename R>
__device__ __forceinline__ void fru_begin(Fru4<R>& F, const LaneStage<R>& L) {
#pragma unroll
  for (int i = 0; i < 3; i++) F.dep[i] = L.dep0[i];
  F.lopen = lcc_open(F.w) ? R(1) : R(0);
  F.nopen = ryr_open_count(F.w);
  F.clk.begin(L);
  ghk_terms(F.dep[0], L.pca_scale, F.e2, F.a2j, F.small);
}

// Values of one substep carried from its first half (rates, extra-draw
// layout, words below 624) to its second (words past 624, Heun step,
// transitions), between which the warp regenerates MT rows.
template <typename R>
struct Sub4 {
  R cajsr, cass, alpha, beta, bp, gam, k12, k23, k34, k54, k25, k56, p34, R0[8];
  int regime, ne, pre, etot;
  uint32_t exmask;  // RyRs that draw an extra uniform (bit 0 of their nibbles)
  uint32_t exw[kRyR], bw[8];
};

// First half of one substep of the FRU (simfru_local.c:83-146 up to the
// draws): the layout of the extra draws and the words that precede word 624,
// then voltage terms, exit totals and the RyR constants.
template <typename R>
__device__ __forceinline__ void substep_a(Fru4<R>& F, Sub4<R>& S, const LaneStage<R>& L, const Group& g,
                                          const StageCtx& sc) {
  uint32_t& w = F.w;
  const int mti = F.mti;
  const R* dep = F.dep;
  R &cajsr = S.cajsr, &cass = S.cass, &alpha = S.alpha, &beta = S.beta, &bp = S.bp, &gam = S.gam;
  R &k12 = S.k12, &k23 = S.k23, &k34 = S.k34, &k54 = S.k54, &k25 = S.k25, &k56 = S.k56;
  R* R0 = S.R0;
  int &regime = S.regime, &ne = S.ne, &pre = S.pre, &etot = S.etot;
  const bool isdiv = L.isdiv;
  const R cA = L.cA, cR = L.cR, cD = L.cD, cCF = L.cCF, cK = L.cK, cM = L.cM;
  cajsr = F.jsr.r();
  cass = F.ss.r();
  // the layout of the extra draws and the words that precede word 624 first:
  // their loads overlap the rest
  {
    const R cc = imin(cass, R(threshMAXCa));
    regime = ilt(cc, R(threshCa56to8)) ? 0 : (ilt(cc, R(threshCa34to7)) ? 1 : 2);
  }
  uint32_t any;
  draw_layout(g, w, regime, 0u, S.exmask, ne, pre, etot, any);
  fetch_old(sc, g, mti, pre, ne, etot, S.exw, S.bw);
  // ---- voltage terms at the substep start, one exponential per lane ----
  const R x = dep[0] + cA;
  R q = x * cR;
  if (isdiv) q = divc(x, cD, cR);
  const R ev = rexp(q);
  const R r01 = cCF * ev;
  const R r23 = rdiv(cK, R(1) + ev) + cM;
  const R vterm = isdiv ? r23 : r01;
  alpha = from(g, vterm, 0);
  beta = from(g, vterm, 1);
  const R yinf = from(g, vterm, 2), tau = from(g, vterm, 3);
  bp = divc(beta, R(bL * kappa), R(1.0 / (bL * kappa)));
  const R ap = R(aL) * alpha;
  // ---- exit totals of this cleft's 8 channels ----
  gam = R(gammacf) * cass;
  {
    const int s = lcc_of(w);
    const uint16_t bi = c_lcc_basis[s];
    const R X = c_lcc_coef[s][0] * pick_basis(bi & 15, alpha, beta, gam, ap, bp);
    const R Y = c_lcc_coef[s][1] * pick_basis((bi >> 4) & 15, alpha, beta, gam, ap, bp);
    const R Z = c_lcc_coef[s][2] * pick_basis((bi >> 8) & 15, alpha, beta, gam, ap, bp);
    R0[0] = X + Y + Z;
  }
  {
    const R num = (vdi_of(w) == 2) ? (R(1) - yinf) : yinf;
    R0[1] = rdiv(num, tau);
  }
  // RyR constants of the cleft and the pseudo-state draws
  const R c2 = cass * cass;
  const R sat = imin(R(threshMAX), divc(c2, R(k_rate), R(1.0 / k_rate)));
  const R sat2 = imin(R(threshMAX), divc(c2, R(k_rate2), R(1.0 / k_rate2)));
  k12 = R(k12cf) * sat2;
  k23 = R(k23cf) * sat;
  k34 = R(k34cf) * sat;
  k54 = R(k54cf) * sat;
  k25 = R(k25cf) * sat;
  k56 = R(k56cf) * sat;
}

// Second half: the remaining words, the RyR pseudo-states, the substep size,
// the Heun step of the local Ca ODE and the transitions (:135-277).
template <typename R>
__device__ __forceinline__ void substep_b(Fru4<R>& F, Sub4<R>& S, const LaneStage<R>& L, const Group& g,
                                          StageCtx& sc) {
  uint32_t& w = F.w;
  int& mti = F.mti;
  R* dep = F.dep;
  R &e2 = F.e2, &a2j = F.a2j, &lopen = F.lopen;
  bool& small = F.small;
  int& nopen = F.nopen;
  const R cajsr = S.cajsr, cass = S.cass, alpha = S.alpha, beta = S.beta, bp = S.bp, gam = S.gam;
  const R k12 = S.k12, k23 = S.k23, k34 = S.k34, k54 = S.k54, k25 = S.k25, k56 = S.k56;
  R& p34 = S.p34;
  R* R0 = S.R0;
  const int regime = S.regime, ne = S.ne, pre = S.pre, etot = S.etot;
  uint32_t* exw = S.exw;
  uint32_t* bw = S.bw;
  const R pca_scale = L.pca_scale;
  fetch_new(sc, g, mti, pre, ne, etot, exw, bw);
  {
    // k34/(k34+k43) is formed once, for the draws of regimes 0/1 or for the
    // merged state 7 of regime 2 (never both)
    const RyrMasks m = ryr_masks(w);
    if (m.s7 | (regime == 2 ? m.s3 | m.s4 : 0u)) p34 = qdiv(k34, k34 + R(k43));
    uint32_t ex = S.exmask;
    while (ex) {
      const int b = __ffs(ex) - 1;  // the RyR's nibble
      ex &= ex - 1u;
      const uint32_t y = exw[0];  // in RyR order, from a shifting window (static register indices)
      exw[0] = exw[1];
      exw[1] = exw[2];
      exw[2] = exw[3];
      exw[3] = exw[4];
      int s;
      if (((w >> (8 + b)) & 15u) == 7u) s = u_below(y, p34) ? 4 : 3;
      else s = u_below(y, qdiv(k56, k56 + R(k65))) ? 6 : 5;
      w = set_field(w, 8 + b, s);
    }
    w = merge_ryr(w, regime);
  }
  {
    const RyrMasks m = ryr_masks(w);
    const bool need7 = m.s7 != 0u, need8 = m.s8 != 0u;
    const R T2 = R(k21) + k23 + k25, T3 = R(k32) + k34, T5 = R(k52) + k54 + k56;
    const R T4 = R(k43 + k45);
    R T7 = R(0), T8 = R(0);
    if (need7) {
      const R a1 = p34;  // k34 / (k43 + k34)
      T7 = (R(1) - a1) * R(k32) + a1 * R(k45);
    }
    if (need8) {
      const R a1 = qdiv(R(k65), k56 + R(k65));
      T8 = a1 * R(k52) + a1 * k54;
    }
  #pragma unroll
    for (int i = 0; i < kRyR; i++) {
      // by the bits of the state, 1 .. 8
      const bool b0 = (w >> (8 + 4 * i)) & 1u, b1 = (w >> (9 + 4 * i)) & 1u, b2 = (w >> (10 + 4 * i)) & 1u;
      const R lo = b1 ? (b0 ? T3 : T2) : (b0 ? k12 : T8), hi = b1 ? (b0 ? T7 : R(k65)) : (b0 ? T5 : T4);
      const R r = b2 ? hi : lo;
      R0[2 + i] = r;
    }
  }
  R0[7] = (cl_of(w) == 1) ? R(kfIto2) * cass : R(kbIto2);
  R mx = R(0);
  #pragma unroll
  for (int j = 0; j < 8; j++) mx = imax(mx, R0[j]);
  mx = gmax(g, mx);
  // ---- substep size (simfru_local.c:135-146) ----
  R dtr = imin(rdiv(R(0.1), mx), R(10.001e-3));
  const R cmax = gmax(g, imax(R(0.e-3), cass));
  if (ilt(R(1.5e-3), cmax)) dtr = imin(dtr, R(5.001e-3));
  const R dt = F.clk.advance(dtr, L);
  // which channels leave (:215-276), beside the Heun step
  const R dts = dt * R(4294967296.0);
  const bool lcc_leaves = leave_gt(bw[0], dts, R0[0]), vdi_leaves = leave_ge(bw[1], dts, R0[1]),
             cl_leaves = leave_ge(bw[7], dts, R0[7]);
  unsigned pend = 0u;
  #pragma unroll
  for (int i = 0; i < kRyR; i++) pend |= leave_gt(bw[2 + i], dts, R0[2 + i]) ? (1u << i) : 0u;
  // ---- Heun step (simfru_local.c:149-173) ----
  R dJ, dS;
  fcn_fru4(g, cajsr, cass, dep, e2, a2j, small, lopen, nopen, pca_scale, dJ, dS);
  const R k1J = dt * dJ, k1S = dt * dS;
  const R y1J = cajsr + k1J, y1S = cass + k1S;
  const R frac = F.clk.frac(L);
  #pragma unroll
  for (int i = 0; i < 3; i++) dep[i] = L.dep0[i] + frac * L.span[i];
  ghk_terms(dep[0], pca_scale, e2, a2j, small);
  fcn_fru4(g, y1J, y1S, dep, e2, a2j, small, lopen, nopen, pca_scale, dJ, dS);
  F.jsr.add((k1J + dt * dJ) / R(2));
  F.ss.add((k1S + dt * dS) / R(2));
  // ---- transitions of this cleft's 8 channels (:215-276) ----
  bool moved = false;
  if (lcc_leaves) {
    const LccBasisT<R> lb{alpha, beta, bp};
    R r[4];
    int d[4];
    const int len = lcc_row(lcc_of(w), lb, gam, r, d);
    w = set_field(w, 0, choose_dest(r, d, len, dt, bw[0]));
  }
  if (vdi_leaves) w = set_field(w, 4, 3 - vdi_of(w));
  // The RyRs that leave their state, then one pass per leaving RyR: the
  // lanes of a warp share the pass (one rate row and destination walk per
  // pass for every lane that has a RyR left), instead of one divergent body
  // per RyR index taken whenever any lane's RyR of that index leaves.  Each
  // RyR's row depends only on its own state and its cleft's constants, so
  // the order of the passes does not matter.
  moved = pend != 0u;
  while (pend) {
    const int i = __ffs(pend) - 1;
    pend &= pend - 1u;
    uint32_t y = bw[2];  // the RyR's uniform, by selection (no dynamic register indexing)
    y = (i == 1) ? bw[3] : y;
    y = (i == 2) ? bw[4] : y;
    y = (i == 3) ? bw[5] : y;
    y = (i == 4) ? bw[6] : y;
    const RyrKT<R> k{k12, k23, k34, k54, k25, k56, regime};
    R r[4];
    int d[4];
    const int len = ryr_row(ryr_of(w, i), k, r, d);
    w = set_field(w, 8 + 4 * i, choose_dest(r, d, len, dt, y));
  }
  if (cl_leaves) w = set_field(w, 28, 3 - cl_of(w));
  lopen = lcc_open(w) ? R(1) : R(0);
  if (moved) nopen = ryr_open_masked(w);
  F.nsub++;
}

// ---- the FP64 substep -----------------------------------------------------------
template <>
struct Fru4<double> {
  FruClock<double> clk;
  CaAcc<double> jsr, ss;
  uint32_t w, nsub;
  int mti;
  bool lopen, small;
  double jcoef;  // JRyRmax x open RyRs of the cleft
  double dep[3], e2, a2j;
};
template <>
struct Sub4<double> {
  double cajsr, cass;
  float X, Y, Z, Rl, Rv, sat, sat2;  // FP32 estimates: LCC exit rates and total, VDI rate, RyR saturations
  uint32_t code;                     // the LCC state's row (LccRow64)
  bool ok;                           // the estimates hold (concentrations and potential in range)
  int regime, ne, pre, etot;
  uint32_t exmask;  // RyRs that draw an extra uniform (bit 0 of their nibbles)
  uint32_t any;     // 1: a CaSS of the FRU is above 1.5e-3; 2: not every cleft's estimates hold
  uint32_t exw[kRyR], bw[8];
};
template <typename R>
__device__ __forceinline__ void sub_begin(Sub4<R>& S) {
  S.etot = 0;
#pragma unroll
  for (int i = 0; i < kRyR; i++) S.exw[i] = 0u;
  S.p34 = R(0);
}
__device__ __forceinline__ void sub_begin(Sub4<double>& S) {
  S.etot = 0;
#pragma unroll
  for (int i = 0; i < kRyR; i++) S.exw[i] = 0u;
}

__device__ __forceinline__ double jryr_open(uint32_t w) {
  const int n = ryr_open_masked(w);
  double v = 0.0;
  v = (n == 1) ? JRyRmax * 1.0 : v;
  v = (n == 2) ? JRyRmax * 2.0 : v;
  v = (n == 3) ? JRyRmax * 3.0 : v;
  v = (n == 4) ? JRyRmax * 4.0 : v;
  v = (n == 5) ? JRyRmax * 5.0 : v;
  return v;
}

__device__ __forceinline__ void fru_begin(Fru4<double>& F, const LaneStage<double>& L) {
#pragma unroll
  for (int i = 0; i < 3; i++) F.dep[i] = L.dep0[i];
  F.lopen = lcc_open(F.w);
  F.jcoef = jryr_open(F.w);
  F.clk.begin(L);
  F.e2 = L.e2;
  F.a2j = L.a2j;
  F.small = L.small;
}

// LCC exit row of each state for the FP64 path: coefficients of the products
// X, Y, Z with bases (4 bits each from bit 0: 0 = 1, 1 = alpha, 2 = beta,
// 3 = gamma, 5 = beta'; alpha' = 2 alpha is in the coefficient, exactly), the
// total X + Y + Z in the reference's order (fru_rates_local.c:176-340), and
// from bit 12 the row's length and its destinations d1, d2, d3; bit 28 / 29:
// the row is (Y, X) / (X, Z, Y) instead of (X, Y, Z).
struct LccRow64 {
  double x, y, z;
  uint32_t code, pad;
};
constexpr uint32_t lcc_code(uint32_t basis, uint32_t len, uint32_t d1, uint32_t d2, uint32_t d3, uint32_t perm) {
  return basis | (len << 12) | (d1 << 16) | (d2 << 20) | (d3 << 24) | (perm << 28);
}
static __device__ const LccRow64 g_lcc_row64[13] = {
    {0.0, 0.0, 0.0, lcc_code(0x000, 1, 0, 0, 0, 0), 0},
    {4.0, 1.0, 0.0, lcc_code(0x031, 3, 2, 7, 0, 0), 0},                           // 1: 4a, g
    {1.0, 3.0, aL, lcc_code(0x312, 4, 1, 3, 8, 0), 0},                            // 2: b, 3a, aL g
    {2.0, 2.0, aL * aL, lcc_code(0x312, 4, 2, 4, 9, 0), 0},                       // 3
    {3.0, 1.0, aL * aL * aL, lcc_code(0x312, 4, 3, 5, 10, 0), 0},                 // 4
    {4.0, fL, aL * aL * aL * aL, lcc_code(0x302, 4, 4, 6, 11, 0), 0},             // 5
    {gL, 0.0, 0.0, lcc_code(0x000, 2, 5, 0, 0, 0), 0},                            // 6
    {4.0 * aL, CCa0_to_C0, 0.0, lcc_code(0x001, 3, 1, 8, 0, 1), 0},               // 7: 4a', omega
    {1.0, 3.0 * aL, CCa1_to_C1, lcc_code(0x015, 4, 7, 2, 9, 2), 0},               // 8: b', 3a', omega/bL
    {2.0, 2.0 * aL, CCa2_to_C2, lcc_code(0x015, 4, 8, 3, 10, 2), 0},              // 9
    {3.0, aL, CCa3_to_C3, lcc_code(0x015, 4, 9, 4, 11, 2), 0},                    // 10
    {4.0, CCa4_to_C4, fLprime, lcc_code(0x005, 4, 10, 5, 12, 0), 0},              // 11
    {gLprime, 0.0, 0.0, lcc_code(0x000, 2, 11, 0, 0, 0), 0},                      // 12
};

// The same coefficients in FP32.
struct __align__(16) LccRow32 {
  float x, y, z;
  uint32_t code;
};
#define GW_ROW32(x, y, z, code) {(float)(x), (float)(y), (float)(z), code}
static __device__ const LccRow32 g_lcc_row32[13] = {
    GW_ROW32(0.0, 0.0, 0.0, lcc_code(0x000, 1, 0, 0, 0, 0)),
    GW_ROW32(4.0, 1.0, 0.0, lcc_code(0x031, 3, 2, 7, 0, 0)),
    GW_ROW32(1.0, 3.0, aL, lcc_code(0x312, 4, 1, 3, 8, 0)),
    GW_ROW32(2.0, 2.0, aL * aL, lcc_code(0x312, 4, 2, 4, 9, 0)),
    GW_ROW32(3.0, 1.0, aL * aL * aL, lcc_code(0x312, 4, 3, 5, 10, 0)),
    GW_ROW32(4.0, fL, aL * aL * aL * aL, lcc_code(0x302, 4, 4, 6, 11, 0)),
    GW_ROW32(gL, 0.0, 0.0, lcc_code(0x000, 2, 5, 0, 0, 0)),
    GW_ROW32(4.0 * aL, CCa0_to_C0, 0.0, lcc_code(0x001, 3, 1, 8, 0, 1)),
    GW_ROW32(1.0, 3.0 * aL, CCa1_to_C1, lcc_code(0x015, 4, 7, 2, 9, 2)),
    GW_ROW32(2.0, 2.0 * aL, CCa2_to_C2, lcc_code(0x015, 4, 8, 3, 10, 2)),
    GW_ROW32(3.0, aL, CCa3_to_C3, lcc_code(0x015, 4, 9, 4, 11, 2)),
    GW_ROW32(4.0, CCa4_to_C4, fLprime, lcc_code(0x005, 4, 10, 5, 12, 0)),
    GW_ROW32(gLprime, 0.0, 0.0, lcc_code(0x000, 2, 11, 0, 0, 0)),
};
#undef GW_ROW32

// ---- exact rates and transitions, for what the FP32 estimates leave open -------
// LCC exit products X, Y, Z of the reference's total X + Y + Z.
__device__ __forceinline__ void lcc_exact(uint32_t w, double alpha, double beta, double cass, double& X, double& Y,
                                          double& Z) {
  const LccRow64* row = &g_lcc_row64[lcc_of(w)];
  const double2 xy = __ldg(reinterpret_cast<const double2*>(row));
  const double z = __ldg(&row->z);
  const uint32_t code = __ldg(&row->code);
  const int bx = code & 15u, by = (code >> 4) & 15u, bz = (code >> 8) & 15u;
  const double gam = gammacf * cass;
  double v = (bx == 1) ? alpha : 1.0;
  v = (bx == 2) ? beta : v;
  v = (bx == 5) ? const_div(beta, kDivBL) : v;  // / (bL * kappa)
  X = xy.x * v;
  v = (by == 1) ? alpha : 1.0;
  v = (by == 3) ? gam : v;
  Y = xy.y * v;
  v = (bz == 3) ? gam : 1.0;
  Z = z * v;
}
static __device__ __noinline__ double vdi_rate_exact(uint32_t w, double V) {
  const double yinf = 0.4 / (1.0 + fexp(const_div(V + 12.5, kDiv5))) + (1.0 - 0.4);
  const double tau = 60.0 + 340.0 / (1.0 + fexp(const_div(V + 30.0, kDiv12)));
  return ((vdi_of(w) == 2) ? 1.0 - yinf : yinf) / tau;
}
__device__ __forceinline__ double sat_exact(double cass) { return imin(threshMAX, const_div(cass * cass, kDivKrate)); }
// Exit total of RyR state s and the first two rates of its row, its length
// and destinations (fru_rates_local.c:374-736).
static __device__ __noinline__ double ryr_total_exact(int s, double cass, int regime, double& r1, double& r2, int& len,
                                               uint32_t& d) {
  const uint32_t to5 = (regime == 0) ? 5u : 8u, to7 = (regime == 2) ? 7u : 3u;
  const double sat = sat_exact(cass);
  r1 = r2 = 0.0;
  len = 2;
  switch (s) {
    case 1: d = 2u; return k12cf * imin(threshMAX, const_div(cass * cass, kDivKrate2));
    case 2: r1 = k21; r2 = k23cf * sat; len = 4; d = 1u | (to7 << 4) | (to5 << 8); return k21 + r2 + k25cf * sat;
    case 3: r1 = k32; len = 3; d = 0x42u; return k32 + k34cf * sat;
    case 4: r1 = k43; len = 3; d = 3u | (to5 << 4); return k43 + k45;
    case 5: r1 = k52; r2 = k54cf * sat; len = 4; d = 0x642u; return k52 + r2 + k56cf * sat;
    case 6: d = 5u; return k65;
    case 7: {
      const double k34 = k34cf * sat, a1 = fast_div(k34, k34 + k43);
      r1 = (1.0 - a1) * k32; len = 3; d = 0x82u; return r1 + a1 * k45;
    }
    default: {
      const double a1 = fast_div(k65, k56cf * sat + k65);
      r1 = a1 * k52; len = 3; d = (regime == 2) ? 0x72u : 0x42u; return r1 + a1 * (k54cf * sat);
    }
  }
}
// Destination of a channel that leaves its state (simfru_local.c:215-253):
// the cumulative walk from P = 1 - dt*total over the row r1, r2, (r3), the
// draw compared with each sum in the integer domain.  d holds d1, d2, d3 in
// its nibbles, len = 1 + destinations.
__device__ __forceinline__ uint32_t walk(uint32_t y, double P, double dt, double r1, double r2, int len, uint32_t d) {
  if (len > 2) {
    const double acc1 = P + dt * r1;
    if (u_above(y, acc1)) {
      d >>= 4;
      if (len > 3 && u_above(y, acc1 + dt * r2)) d >>= 4;
    }
  }
  return d & 15u;
}
// The transitions of one cleft's 8 channels (simfru_local.c:215-276): every
// rate and probability in FP64, the draws compared in the integer domain.
static __device__ __noinline__ uint32_t transitions_exact(uint32_t w, double V, double cass, double dt, int regime, uint4 ya,
                                                   uint4 yb) {
  const uint32_t y[8] = {ya.x, ya.y, ya.z, ya.w, yb.x, yb.y, yb.z, yb.w};
  {
    const double alpha = alphacf * fexp(0.012 * (V - 35.0)), beta = betacf * fexp(-0.05 * (V - 35.0));
    double X, Y, Z;
    lcc_exact(w, alpha, beta, cass, X, Y, Z);
    const double P = 1.0 - dt * (X + Y + Z);
    if (u_above(y[0], P)) {
      const uint32_t code = g_lcc_row64[lcc_of(w)].code, perm = code >> 28;
      const double r1 = (perm == 1) ? Y : X, r2 = (perm == 2) ? Z : (perm == 1) ? X : Y;
      w = set_field(w, 0, (int)walk(y[0], P, dt, r1, r2, (int)((code >> 12) & 15u), code >> 16));
    }
  }
  if (u_reaches(y[1], 1.0 - dt * vdi_rate_exact(w, V))) w = set_field(w, 4, 3 - vdi_of(w));
#pragma unroll
  for (int i = 0; i < kRyR; i++) {
    double r1, r2;
    int len;
    uint32_t d;
    const double P = 1.0 - dt * ryr_total_exact(ryr_of(w, i), cass, regime, r1, r2, len, d);
    if (u_above(y[2 + i], P)) w = set_field(w, 8 + 4 * i, (int)walk(y[2 + i], P, dt, r1, r2, len, d));
  }
  if (u_reaches(y[7], 1.0 - dt * ((cl_of(w) == 1) ? kfIto2 * cass : kbIto2))) w = set_field(w, 28, 3 - cl_of(w));
  return w;
}

// x truncated to FP32, for 0 or 2^-126 <= |x| < 2^127, without an FP64 instruction
__device__ __forceinline__ float trunc32(double x) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const uint32_t ah = max(hi & 0x7fffffffu, 0x38000000u) - 0x38000000u;
  return __uint_as_float(__funnelshift_l(lo, ah, 3) | (hi & 0x80000000u));
}

// Buffer factors of the local ODE: 1/(1 + a1 + a2) of the subspace and
// 1/(1 + a1) of the JSR (fcn_fru.c:103-131).  Concentrations of [0, 16) mM
// keep every divisor in the fast forms' range.
__device__ __forceinline__ bool conc_ok(double c) { return (uint32_t)__double2hiint(c) < 0x40300000u; }
__device__ __forceinline__ void buffer_factors(double cajsr, double cass, double& bSS, double& bJSR) {
  const double xr = cass + KBSR, xl = cass + KBSL, xj = cajsr + KmCSQN;
  const double dr = xr * xr, dl = xl * xl, dj = xj * xj;
  if (conc_ok(cass) && conc_ok(cajsr)) {
    const double a1 = fast_div(BSRtot * KBSR, dr), a2 = fast_div(BSLtot * KBSL, dl);
    const double aj = fast_div(CSQNtot * KmCSQN, dj);
    bSS = fast_rcp(1.0 + a1 + a2);
    bJSR = fast_rcp(1.0 + aj);
  } else {
    const double a1 = BSRtot * KBSR / dr, a2 = BSLtot * KBSL / dl;
    const double aj = CSQNtot * KmCSQN / dj;
    bSS = 1.0 / (1.0 + a1 + a2);
    bJSR = 1.0 / (1.0 + aj);
  }
}

// Local Ca ODE of one cleft (fcn_fru.c:23-137), FP64; see fcn_fru4 above.
__device__ __forceinline__ void fcn_fru4(const Group& g, double cajsr, double cass, const double dep[3], double e2,
                                         double a2j, bool small, bool lopen, double jcoef, double pca2, double& dJSR,
                                         double& dSS) {
  constexpr double JDHconstant = 1.0 / (2.0 * VSS * Faraday * 1000.0);
  const double Cai = dep[1], CaNSR = dep[2];
  double bSS, bJSR;
  buffer_factors(cajsr, cass, bSS, bJSR);
  const double JRyR = jcoef * (cajsr - cass);
  const double j0 = from(g, JRyR, 0), j1 = from(g, JRyR, 1), j2 = from(g, JRyR, 2), j3 = from(g, JRyR, 3);
  const double JRyRtot = j0 + j1 + j2 + j3;
  const double cnext = from(g, cass, (g.c + 1) & 3);
  const double Jss = const_div(cass - cnext, kDivTauss2ss);
  const double Jss_prev = from(g, Jss, (g.c + 3) & 3);
  const double Jxfer = const_div(cass - Cai, kDivTauxfer);
  double JDH = 0.0;
  if (lopen) {
    if (small) JDH = pca2 * (cass - Cao * 0.341) * JDHconstant;
    else JDH = -(cass * e2 - Cao * 0.341) * a2j;
  }
  dSS = bSS * (JDH + JRyR - Jxfer - Jss + Jss_prev);
  const double Jtr = const_div(CaNSR - cajsr, kDivTautr);
  dJSR = bJSR * (Jtr - (VSS / VJSR) * JRyRtot);
}

// The same on sixteen lanes: the copies of a cleft's lane take a quotient each
// (a1 and a2 of the subspace, a1 of the JSR), then a difference times a
// constant (JRyR, Jss, Jtr, Jxfer), then one sum (dCaSS on copy 0, dCaJSR on
// copy 2), every lane with operands of its own in one stream: 18 FP64
// instructions instead of 44.  x * 1 + y, x * y + 0 and x * (-1) + y round
// as the sum, the product and the difference alone.
__device__ __forceinline__ void fcn_fru4(const WideGroup& g, double cajsr, double cass, const double dep[3], double e2,
                                         double a2j, bool small, bool lopen, double jcoef, double pca2, double& dJSR,
                                         double& dSS) {
  constexpr double JDHconstant = 1.0 / (2.0 * VSS * Faraday * 1000.0);
  const int q = g.q;
  auto copy = [&](double v, int k, int c) { return __shfl_sync(g.mask, v, g.base + 4 * k + c); };
  double b;  // bSS, on copy 2 bJSR
  {
    const double x = (q == 2 ? cajsr : cass) + (q == 0 ? KBSR : q == 2 ? KmCSQN : KBSL);
    const double den = x * x, num = q == 0 ? BSRtot * KBSR : q == 2 ? CSQNtot * KmCSQN : BSLtot * KBSL;
    const bool ok = conc_ok(cass) && conc_ok(cajsr);  // alike on the copies of a cleft
    const double a = ok ? fast_div(num, den) : num / den;
    const double a1 = copy(a, 0, g.c), a2 = copy(a, 1, g.c), aj = copy(a, 2, g.c);
    const double t = (1.0 + (q == 2 ? aj : a1)) + (q == 2 ? 0.0 : a2);
    b = ok ? fast_rcp(t) : 1.0 / t;
  }
  const double cnext = from(g, cass, (g.c + 1) & 3);
  double lin;  // JRyR, Jss, Jtr, Jxfer
  {
    const double x = (q == 0 ? cajsr : q == 2 ? dep[2] : cass) - (q == 0 ? cass : q == 1 ? cnext : q == 2 ? cajsr : dep[1]);
    const double hi = q == 0 ? jcoef : q == 1 ? kDivTauss2ss.rhi : q == 2 ? kDivTautr.rhi : kDivTauxfer.rhi;
    const double lo = q == 0 ? 0.0 : q == 1 ? kDivTauss2ss.rlo : q == 2 ? kDivTautr.rlo : kDivTauxfer.rlo;
    lin = fma(x, hi, x * lo);
  }
  const double j0 = copy(lin, 0, 0), j1 = copy(lin, 0, 1), j2 = copy(lin, 0, 2), j3 = copy(lin, 0, 3);
  const double JRyR = copy(lin, 0, g.c), Jss = copy(lin, 1, g.c), Jss_prev = copy(lin, 1, (g.c + 3) & 3);
  const double Jxfer = copy(lin, 3, g.c);
  double JDH = 0.0;
  if (lopen) {
    if (small) JDH = pca2 * (cass - Cao * 0.341) * JDHconstant;
    else JDH = -(cass * e2 - Cao * 0.341) * a2j;
  }
  const bool jsr = q == 2;
  double s = (jsr ? j0 : JDH) + (jsr ? j1 : JRyR);
  s = s + (jsr ? j2 : -Jxfer);
  s = s + (jsr ? j3 : -Jss);
  s = fma(s, jsr ? VSS / VJSR : 1.0, jsr ? 0.0 : Jss_prev);
  s = fma(s, jsr ? -1.0 : 1.0, jsr ? lin : 0.0);  // copy 2: Jtr less it
  const double d = b * s;
  dSS = copy(d, 0, g.c);
  dJSR = copy(d, 2, 0);
}

// The rates of a substep decide two things: its size dt = min(0.1 / the
// largest rate, a cap), and, against the draws, which channels change state.
// Both are settled by FP32 estimates of the rates wherever the comparison is
// clear by kRateTol; the rates that could be the largest, and all of a cleft
// with a draw too close to its threshold (about one substep in 10^4), are formed
// in FP64 as the reference does.  Rates in FP64 throughout took about 60 of a
// substep's 190 FP64 instructions.
// The estimates' relative error is below 2^-15 (truncated inputs, a few
// roundings, exponentials of arguments below 10; the most in RyR state 7's
// total, where 1 - p7 cancels) but for the VDI gate: the exponentials of yinf
// and tau have arguments up to 33, and 1 - yinf, the rate of an open gate,
// cancels, to nothing at negative potentials.  Its error is small against the
// thresholds instead: over |V| < 150 mV and the longest substep, with the error
// bounds documented for the approximate functions, below 0.2 of the 2^32 values
// of a draw, which the 2 in a threshold's tolerance covers; and at most 1/60 per
// ms it is never the largest rate of a substep below the cap.
constexpr float kRateTol = 0x1p-13f;

// First half of one FP64 substep (simfru_local.c:83-146 up to the draws):
// the layout of the extra draws and the words that precede word 624 first
// (their loads overlap the rest), then the estimates of the voltage terms and
// exit totals.
__device__ __forceinline__ void substep_a(Fru4<double>& F, Sub4<double>& S, const LaneStage<double>& L, const Group& g,
                                          const StageCtx& sc) {
  const uint32_t w = F.w;
  const double cass = F.ss.v, V = F.dep[0];
  S.cajsr = F.jsr.v;
  S.cass = cass;
  {
    const double cc = imin(cass, threshMAXCa);
    S.regime = ilt(cc, threshCa56to8) ? 0 : (ilt(cc, threshCa34to7) ? 1 : 2);
  }
  S.ok = fits(cass) && conc_ok(cass) && abs_lt(V, 150.0);
  draw_layout(g, w, S.regime, (ilt(1.5e-3, cass) ? 1u : 0u) | (S.ok ? 0u : 2u), S.exmask, S.ne, S.pre, S.etot, S.any);
  fetch_old(sc, g, F.mti, S.pre, S.ne, S.etot, S.exw, S.bw);
  // ---- voltage terms at the substep start, one exponential per lane ----
  const float c = trunc32(cass);
  const float ev = __expf((trunc32(V) + L.cA) * L.cR);
  const float vterm = L.isdiv ? __fdividef(L.cK, 1.0f + ev) + L.cM : L.cCF * ev;
  const float alpha = from(g, vterm, 0), beta = from(g, vterm, 1);
  const float yinf = from(g, vterm, 2), tau = from(g, vterm, 3);
  const float bp = beta * (float)(1.0 / (bL * kappa)), gam = (float)gammacf * c;
  {
    const float4 row = __ldg(reinterpret_cast<const float4*>(&g_lcc_row32[lcc_of(w)]));
    const uint32_t code = __float_as_uint(row.w);
    const int bx = code & 15u, by = (code >> 4) & 15u, bz = (code >> 8) & 15u;
    S.code = code;
    S.X = row.x * ((bx == 1) ? alpha : (bx == 2) ? beta : (bx == 5) ? bp : 1.0f);
    S.Y = row.y * ((by == 1) ? alpha : (by == 3) ? gam : 1.0f);
    S.Z = row.z * ((bz == 3) ? gam : 1.0f);
    S.Rl = S.X + S.Y + S.Z;
  }
  S.Rv = __fdividef((vdi_of(w) == 2) ? 1.0f - yinf : yinf, tau);
  const float c2 = c * c;
  S.sat = fminf((float)threshMAX, c2 * (float)(1.0 / k_rate));
  S.sat2 = fminf((float)threshMAX, c2 * (float)(1.0 / k_rate2));
}

// Second half: the remaining words, the RyR pseudo-states, the substep size,
// the Heun step of the local Ca ODE and the transitions (:135-277).
template <typename G>
__device__ __forceinline__ void substep_b64(Fru4<double>& F, Sub4<double>& S, const LaneStage<double>& L, const G& g,
                                            StageCtx& sc) {
  uint32_t w = F.w;
  const double cajsr = S.cajsr, cass = S.cass, V = F.dep[0];
  const int regime = S.regime;
  uint32_t* bw = S.bw;
  fetch_new(sc, g, F.mti, S.pre, S.ne, S.etot, S.exw, bw);
  if (S.ne) {
    const double sat = sat_exact(cass), k34 = k34cf * sat, k56 = k56cf * sat;
    uint32_t ex = S.exmask;
    while (ex) {
      const int b = __ffs(ex) - 1;  // the RyR's nibble
      ex &= ex - 1u;
      const uint32_t y = S.exw[0];  // in RyR order, from a shifting window
      S.exw[0] = S.exw[1];
      S.exw[1] = S.exw[2];
      S.exw[2] = S.exw[3];
      S.exw[3] = S.exw[4];
      uint32_t s;
      if (((w >> (8 + b)) & 15u) == 7u) s = u_below(y, fast_div(k34, k34 + k43)) ? 4u : 3u;
      else s = u_below(y, fast_div(k56, k56 + k65)) ? 6u : 5u;
      w = set_field(w, 8 + b, (int)s);
    }
  }
  w = merge_ryr(w, regime);
  // ---- exit totals of the RyR states (estimates) ----
  const float k34 = (float)k34cf * S.sat, k56 = (float)k56cf * S.sat, k54 = (float)k54cf * S.sat,
              k23 = (float)k23cf * S.sat, k25 = (float)k25cf * S.sat;
  const float p7 = __fdividef(k34, k34 + (float)k43), p8 = __fdividef((float)k65, k56 + (float)k65);
  const float t7 = (1.0f - p7) * (float)k32, t8 = p8 * (float)k52;
  const float T1 = (float)k12cf * S.sat2, T2 = (float)k21 + k23 + k25, T3 = (float)k32 + k34, T4 = (float)(k43 + k45),
              T5 = (float)k52 + k54 + k56, T6 = (float)k65, T7 = t7 + p7 * (float)k45, T8 = t8 + p8 * k54;
  const float Rc = (cl_of(w) == 1) ? (float)kfIto2 * trunc32(cass) : (float)kbIto2;
  float r[kRyR];
#pragma unroll
  for (int i = 0; i < kRyR; i++) {
    const bool b0 = (w >> (8 + 4 * i)) & 1u, b1 = (w >> (9 + 4 * i)) & 1u, b2 = (w >> (10 + 4 * i)) & 1u;
    const float lo = b1 ? (b0 ? T3 : T2) : (b0 ? T1 : T8), hi = b1 ? (b0 ? T7 : T6) : (b0 ? T5 : T4);
    r[i] = b2 ? hi : lo;
  }
  // ---- substep size (simfru_local.c:135-146) ----
  const bool ok = !(S.any & 2u), fast_ca = S.any & 1u;
  double dtr = fast_ca ? 5.001e-3 : 10.001e-3;
  float mx = fmaxf(fmaxf(fmaxf(S.Rl, S.Rv), Rc), fmaxf(fmaxf(fmaxf(r[0], r[1]), fmaxf(r[2], r[3])), r[4]));
  mx = fmaxf(mx, __shfl_xor_sync(g.mask, mx, 1));
  mx = fmaxf(mx, __shfl_xor_sync(g.mask, mx, 2));
  // 0.1 / cap = 19.996 or 9.999: below these the cap is the smaller
  if (!ok || !(mx < (fast_ca ? 19.99f : 9.998f))) {
    const float near = ok ? mx * (1.0f - kRateTol) : -1.0f;  // -1: every rate
    double m = 0.0;
    const bool lcc = !(S.Rl < near);
    uint32_t need = lcc ? 1u : 0u;
    need |= __shfl_xor_sync(g.mask, need, 1);
    need |= __shfl_xor_sync(g.mask, need, 2);
    if (need) {
      // alpha on the even lanes, beta on the odd ones
      const bool odd = g.c & 1;
      const double t = (odd ? betacf : alphacf) * fexp((odd ? -0.05 : 0.012) * (V - 35.0));
      const double alpha = from(g, t, 0), beta = from(g, t, 1);
      double X, Y, Z;
      lcc_exact(w, alpha, beta, cass, X, Y, Z);
      if (lcc) m = imax(m, X + Y + Z);
    }
    if (!(S.Rv < near)) m = imax(m, vdi_rate_exact(w, V));
    if (!(Rc < near)) m = imax(m, (cl_of(w) == 1) ? kfIto2 * cass : kbIto2);
    const RyrMasks q = ryr_masks(w);
    if (q.s3 && !(T3 < near)) m = imax(m, k32 + k34cf * sat_exact(cass));
    if (q.s4 && !(T4 < near)) m = imax(m, k43 + k45);
    if (q.s6 && !(T6 < near)) m = imax(m, k65);
    const uint32_t rest = q.s1 | q.s2 | q.s5 | q.s7 | q.s8;
    if (rest) {
#pragma unroll 1
      for (int k = 0; k < 5; k++) {
        const int s = (k < 2) ? k + 1 : (k == 2) ? 5 : k + 4;  // 1, 2, 5, 7, 8
        const uint32_t there = (k == 0) ? q.s1 : (k == 1) ? q.s2 : (k == 2) ? q.s5 : (k == 3) ? q.s7 : q.s8;
        const float T = (k == 0) ? T1 : (k == 1) ? T2 : (k == 2) ? T5 : (k == 3) ? T7 : T8;
        if (there && !(T < near)) {
          double r1, r2;
          int len;
          uint32_t d;
          m = imax(m, ryr_total_exact(s, cass, regime, r1, r2, len, d));
        }
      }
    }
    m = gmax(g, m);
    dtr = imin(fits(m) ? fast_div(0.1, m) : 0.1 / m, dtr);
  }
  const double dt = F.clk.advance(dtr, L);
  // ---- Heun step (simfru_local.c:149-173) ----
  double dJ, dS;
  fcn_fru4(g, cajsr, cass, F.dep, F.e2, F.a2j, F.small, F.lopen, F.jcoef, L.pca2, dJ, dS);
  const double k1J = dt * dJ, k1S = dt * dS;
  const double y1J = cajsr + k1J, y1S = cass + k1S;
  {
    const double mine = L.mydep0 + F.clk.frac(L) * L.myspan;
    F.dep[0] = from(g, mine, 0);
    F.dep[1] = from(g, mine, 1);
    F.dep[2] = from(g, mine, 2);
  }
  ghk_terms(F.dep[0], L.pca4, F.e2, F.a2j, F.small, F.dep[1]);
  fcn_fru4(g, y1J, y1S, F.dep, F.e2, F.a2j, F.small, F.lopen, F.jcoef, L.pca2, dJ, dS);
  F.jsr.v = fma(k1J + dt * dJ, 0.5, cajsr);
  F.ss.v = fma(k1S + dt * dS, 0.5, cass);
  // ---- transitions of this cleft's 8 channels (:215-276) ----
  // A channel leaves when c = 2^32 - y is below about dt*R*2^32; `open` is set
  // where c is within the tolerance of a threshold: kRateTol of it, and 2 for
  // the roundings of the exact one (below 1) and the VDI gate's estimate (0.2).
  // The RyRs that leave take one
  // pass each: the lanes of a warp share the pass.  Each RyR's row depends
  // only on its own state and its cleft's constants, so the order of the
  // passes does not matter.
  const float dts = trunc32(dt) * 4294967296.0f;
  bool open = !S.ok;
  auto below = [&](float c, float t, float tol) {
    open = open || fabsf(c - t) <= tol;
    return c < t;
  };
  auto leaves = [&](uint32_t y, float R) {
    const float t = dts * R;
    return below(comp_u32(y), t, __fmaf_rn(t, kRateTol, 2.0f));
  };
  uint32_t n = w;
  if (leaves(bw[0], S.Rl)) {
    const uint32_t perm = S.code >> 28, len = (S.code >> 12) & 15u;
    uint32_t d = S.code >> 16;
    const float r1 = (perm == 1) ? S.Y : S.X, r2 = (perm == 2) ? S.Z : (perm == 1) ? S.X : S.Y;
    const float cc = comp_u32(bw[0]), tol = __fmaf_rn(dts * S.Rl, kRateTol, 2.0f);
    if (len > 2u && below(cc, dts * (S.Rl - r1), tol)) {
      d >>= 4;
      if (len > 3u && below(cc, dts * (S.Rl - r1 - r2), tol)) d >>= 4;
    }
    n = set_field(n, 0, (int)(d & 15u));
  }
  if (leaves(bw[1], S.Rv)) n = set_field(n, 4, 3 - vdi_of(w));
  uint32_t pend = 0u;
#pragma unroll
  for (int i = 0; i < kRyR; i++) pend |= leaves(bw[2 + i], r[i]) ? (1u << i) : 0u;
  while (pend) {
    const int i = __ffs(pend) - 1;
    pend &= pend - 1u;
    uint32_t y = bw[2];  // the RyR's uniform, by selection (no dynamic register indexing)
    y = (i == 1) ? bw[3] : y;
    y = (i == 2) ? bw[4] : y;
    y = (i == 3) ? bw[5] : y;
    y = (i == 4) ? bw[6] : y;
    const int s = ryr_of(w, i);
    // the total less the first one and the first two rates, row length and
    // destinations (fru_rates_local.c:374-736)
    const uint32_t to5 = (regime == 0) ? 5u : 8u, to7 = (regime == 2) ? 7u : 3u;
    float T = T1, u1 = 0.0f, u2 = 0.0f;
    int len = 2;
    uint32_t d = 2u;  // 1 -> 2
    if (s == 2) { T = T2; u1 = k23 + k25; u2 = k25; len = 4; d = 1u | (to7 << 4) | (to5 << 8); }
    if (s == 3) { T = T3; u1 = k34; len = 3; d = 0x42u; }
    if (s == 4) { T = T4; u1 = (float)k45; len = 3; d = 3u | (to5 << 4); }
    if (s == 5) { T = T5; u1 = k54 + k56; u2 = k56; len = 4; d = 0x642u; }
    if (s == 6) { T = T6; d = 5u; }
    if (s == 7) { T = T7; u1 = T7 - t7; len = 3; d = 0x82u; }
    if (s == 8) { T = T8; u1 = T8 - t8; len = 3; d = (regime == 2) ? 0x72u : 0x42u; }
    const float cc = comp_u32(y), tol = __fmaf_rn(dts * T, kRateTol, 2.0f);
    if (len > 2 && below(cc, dts * u1, tol)) {
      d >>= 4;
      if (len > 3 && below(cc, dts * u2, tol)) d >>= 4;
    }
    n = set_field(n, 8 + 4 * i, (int)(d & 15u));
  }
  if (leaves(bw[7], Rc)) n = set_field(n, 28, 3 - cl_of(w));
  if (open)
    n = transitions_exact(w, V, cass, dt, regime, make_uint4(bw[0], bw[1], bw[2], bw[3]),
                          make_uint4(bw[4], bw[5], bw[6], bw[7]));
  F.lopen = lcc_open(n);
  if (n != w) F.jcoef = jryr_open(n);
  F.w = n;
  F.nsub++;
}

__device__ __forceinline__ void substep_b(Fru4<double>& F, Sub4<double>& S, const LaneStage<double>& L, const Group& g,
                                          StageCtx& sc) {
  substep_b64(F, S, L, g, sc);
}
__device__ __forceinline__ void substep_b(Fru4<double>& F, Sub4<double>& S, const LaneStage<double>& L,
                                          const WideGroup& g, StageCtx& sc) {
  substep_b64(F, S, L, g, sc);
}

// Regenerate, with the whole warp, the MT rows whose draws in this substep
// run past word 624 (`go`: this lane's FRU takes a substep now).
template <typename R>
__device__ __forceinline__ void regen_step(const StageCtx& sc, int lane, const Group& g, bool go, const Fru4<R>& F,
                                           const Sub4<R>& S) {
  const bool cross = go && (F.mti + S.etot + 32 > kMtN);
  const bool lead = cross && g.c == 0 && g.q == 0;
  const unsigned cross_mask = __ballot_sync(0xffffffffu, lead);
  const unsigned copy_mask = __ballot_sync(0xffffffffu, lead && *sc.my_hold_epoch != sc.p->epoch);
  if (cross_mask) regen_crossing(sc, lane, cross_mask, copy_mask);
}

// One FRU over [t0, tf] by its four lanes (simfru_local.c:83-277).  cajsr and
// cass are the FRU's FP64 state; arithmetic runs in R.  Every lane of the
// warp calls it together (live = false for a group without an FRU).
template <typename R, typename G>
__device__ __forceinline__ void advance4(StageCtx& sc, const G& g, bool live, double& cajsr64, double& cass64,
                                         uint32_t& w, int& mti, uint32_t& nsub, bool& overflow) {
  LaneStage<R> L;
  lane_stage(*sc.p, g, L);
  Fru4<R> F;
  F.jsr.set(cajsr64);
  F.ss.set(cass64);
  F.w = w;
  F.mti = mti;
  F.nsub = nsub;
  fru_begin(F, L);
  const int lane = threadIdx.x & 31;
  while (true) {
    // all 32 lanes stay in the loop until every FRU of the warp is done, so
    // the warp can regenerate MT rows together; a group whose FRU has
    // reached tf (or never had one) idles
    bool go = live && F.clk.running(L);
    if (go && F.nsub >= (1u << 22)) {
      overflow = true;
      go = false;
    }
    if (!__any_sync(0xffffffffu, go)) break;
    Sub4<R> S;
    sub_begin(S);
    if (go) substep_a(F, S, L, g, sc);
    regen_step(sc, lane, g, go, F, S);
    if (go) substep_b(F, S, L, g, sc);
  }
  cajsr64 = F.jsr.get();
  cass64 = F.ss.get();
  w = F.w;
  mti = F.mti;
  nsub = F.nsub;
}

// The stage of one cell, block bidx of the cell's blocks (blockDim.x / 32
// warps of 8 FRUs each): load, optional snapshot save/restore, advance,
// store, and the fused deterministic flux reduction
// (calc_fru_flux_local.c:28-77, mpi_master.c:447-468, mpi_slave.c:150-226);
// the cell's totals go to out[0..8] and its error flag to out[kOutError].
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Where a launch's cell totals go: the 5 flux numerators, the currents and,
// when the launch carried kFlagAvg, the 11 output-average sums, to the
// launch's out[] slots: host memory, or the device-resident integrator's.
// Whole warp, with the totals in lane 0
__device__ __forceinline__ void put_totals(const DevState& s, const StageParams& p, double* out, double tot[5], int lane) {
#pragma unroll
  for (int k = 0; k < 5; k++) tot[k] = __shfl_sync(0xffffffffu, tot[k], 0);
  const double cur = lane_current(s, p, tot, lane);
  double v = tot[0];
#pragma unroll
  for (int k = 1; k < 5; k++) v = (lane == 4 + k) ? tot[k] : v;
  if (lane < 4) out[5 + lane] = cur;
  else if (lane < 9) out[lane - 4] = v;
}
// after every total: tell the host that waits for this launch
__device__ __forceinline__ void put_seq(const StageParams& p, double* out, int lane) {
  __syncwarp();
  if (lane == 0) {
    __threadfence_system();
    *reinterpret_cast<volatile unsigned long long*>(out + kOutSeq) = p.seq;
  }
}

template <typename R, typename G = Group>
__device__ __forceinline__ void stage_body(const DevState& s, const StageParams& p, int bidx, double* out, int fpw = 8) {
  constexpr bool wide = is_wide<G>::value;  // sixteen lanes per FRU, at most two FRUs per warp
  const int lane = threadIdx.x & 31;
  const int first = (bidx * (int)(blockDim.x >> 5) + (int)(threadIdx.x >> 5)) * fpw;  // the warp's first FRU
  const int grp = first >> 3;  // their 8-FRU group
  if ((p.flags & kFlagQueueReset) && bidx == 0 && threadIdx.x == 0) {
    // after a packed launch: ready the queue for the next one (the heavy-FRU
    // threshold becomes 3x this launch's mean substeps per FRU, at least 8)
    const uint32_t n = (uint32_t)s.nfru;
    const uint32_t thr = 3u * (s.qctl[3] / (n ? n : 1u));
    s.qctl[4] = thr > 8u ? thr : 8u;
    s.qctl[3] = 0u;
    s.qctl[0] = 0u;
    s.qctl[1 + ((p.launch + 1u) & 1u)] = 0u;
  }
  if (first >= s.nfru) return;  // whole warps past the cell's last FRU
  // traced group: its first warp's begin and its last warp's end
  if (s.trace_ns && lane == 0) {
    if (fpw < 8) atomicMin(&s.trace_ns[2 * grp], global_ns());
    else s.trace_ns[2 * grp] = global_ns();
  }
  G g;
  g.c = lane & 3;
  g.q = wide ? (lane >> 2) & 3 : 0;
  g.base = wide ? lane & ~15 : lane & ~3;
  g.mask = (wide ? 0xffffu : 0xfu) << g.base;
  const int slot = wide ? lane >> 4 : lane >> 2;
  bool active = slot < fpw && first + slot < s.nfru;  // uniform over each 4-lane group
  const int f = active ? first + slot : first;
  uint32_t nsub = 0;
  bool overflow = false;
  const size_t nf = (size_t)s.stride;
  double cajsr = 0.0, cass = 0.0;
  uint32_t w = 0u;
  int mti = 0;
  uint32_t* gm = s.mt + (size_t)f * kMtStride;
  StageCtx sc;
  sc.p = &p;
  sc.m = gm;
  sc.hold_base = s.mt_hold;
  sc.hold_epoch_base = s.hold_epoch;
  sc.f = f;
  sc.my_hold_epoch = s.hold_epoch + f;
  bool restore = false;
  if (active) {
    if (p.flags & kFlagResume) {
      cajsr = s.frus_s[f];
      cass = s.frus_s[(g.c + 1) * nf + f];
      w = s.chan_s[g.c * nf + f];
      mti = s.mti_s[f];
      restore = (*sc.my_hold_epoch == p.epoch);
    } else {
      cajsr = s.frus[f];
      cass = s.frus[(g.c + 1) * nf + f];
      w = s.chan[g.c * nf + f];
      mti = s.mti[f];
    }
    if ((p.flags & kFlagSave) && g.q == 0) {
      if (g.c == 0) {
        s.frus_s[f] = cajsr;
        s.mti_s[f] = mti;
      }
      s.frus_s[(g.c + 1) * nf + f] = cass;
      s.chan_s[g.c * nf + f] = w;
    }
  }
  const uint32_t* hold = sc.hold_base + (size_t)f * kMtStride;
  if (p.flags & kFlagAdvance) {
    if (active) use_row(sc, gm, hold, restore, g);
    __syncwarp();
    advance4<R>(sc, g, active, cajsr, cass, w, mti, nsub, overflow);
    __syncwarp();
  } else if (active && restore) {
    copy_row16(gm, hold, g);
  }
  if (active && g.q == 0) {
    if (s.trace_sub && g.c == 0) s.trace_sub[f] = nsub;
    if (g.c == 0) {
      s.frus[f] = cajsr;
      s.mti[f] = mti;
    }
    s.frus[(g.c + 1) * nf + f] = cass;
    s.chan[g.c * nf + f] = w;
  }
  // before the barrier, so that lane 0's fences carry it and the host, which
  // waits for the sequence number only, finds it with this launch's totals
  if (overflow) out[kOutError] = 1.0;
  __syncwarp();
  if (fpw == 8 && s.trace_ns && lane == 0) s.trace_ns[2 * grp + 1] = global_ns();
  if (s.substeps) {
    unsigned c = __reduce_add_sync(0xffffffffu, (g.c == 0 && g.q == 0) ? nsub : 0u);
    if (lane == 0 && c) atomicAdd(s.substeps, (unsigned long long)c);
  }
  if (fpw < 8) {
    // several warps share the group: the one that completes it sums it, from
    // the FRUs as stored
    const unsigned mine = (unsigned)min(fpw, s.nfru - first), size = (unsigned)min(8, s.nfru - grp * 8);
    unsigned last = 0u;
    if (lane == 0) {
      __threadfence();
      last = (atomicAdd(&s.gcount[grp], mine) + mine == size) ? 1u : 0u;
      if (last) s.gcount[grp] = 0u;
      if (last && s.trace_ns) s.trace_ns[2 * grp + 1] = global_ns();
    }
    if (!__shfl_sync(0xffffffffu, last, 0)) return;
    __syncwarp();  // lane 0's count before every lane's reads (a shuffle orders no memory)
    __threadfence();
    const int ff = grp * 8 + (lane >> 2);
    active = ff < s.nfru;
    if (active) {
      cajsr = __ldcg(&s.frus[ff]);
      cass = __ldcg(&s.frus[(g.c + 1) * nf + ff]);
      w = __ldcg(&s.chan[g.c * nf + ff]);
    }
  }
  if (p.flags & kFlagAvg) {
    AvgSums v = {};
    if (active) avg_terms(g.c, cajsr, cass, w, v);
    store_group(s, grp, v, lane);
    if (finish_groups(s, v, 1u, lane)) {
      double tot[16];
      unpack_avg(v, tot);
      put_totals(s, p, out, tot, lane);
      if (lane == 0)
#pragma unroll
        for (int k = 0; k < 11; k++) out[16 + k] = tot[5 + k];
      put_seq(p, out, lane);
    }
    return;
  }
  FluxSums v = {};
  if (active) flux_terms(g.c, cajsr, cass, w, v);
  store_group(s, grp, v, lane);
  if (finish_groups(s, v, 1u, lane)) {
    double tot[5];
    unpack_flux(v, tot);
    put_totals(s, p, out, tot, lane);
    put_seq(p, out, lane);
  }
}

// ---- packed stage: a queue of FRUs per 4-lane group -----------------------------
// A warp's eight 4-lane groups each advance one FRU at a time and, when it
// reaches tf, store it and take the next from the cell's queue, so a warp's
// lanes stay busy until the queue is empty instead of idling behind the
// slowest of eight fixed FRUs.  The queue hands out first the FRUs that were
// heavy (many substeps) in the cell's previous packed launch, then the others
// in order.  The per-FRU arithmetic is advance4's, so every FRU ends in the
// same state as with the fixed layout; the flux sums come from a following
// non-advancing launch over the stored states, in the usual fixed order.
template <typename R>
__device__ __forceinline__ void stage_body_packed(const DevState& s, const StageParams& p, double* out) {
  const int lane = threadIdx.x & 31;
  Group g;
  g.c = lane & 3;
  g.base = lane & ~3;
  g.mask = 0xfu << g.base;
  const size_t nf = (size_t)s.stride;
  const int n = s.nfru;
  const uint32_t L = p.launch;
  const int* heavy_prev = s.heavy_list + (size_t)((L + 1u) & 1u) * nf;
  int* heavy_next = s.heavy_list + (size_t)(L & 1u) * nf;
  // tags by launch parity too: this launch re-tags the FRUs it finds heavy
  // without changing what its own queue skips
  const uint32_t* tag_prev = s.heavy_tag + (size_t)((L + 1u) & 1u) * nf;
  uint32_t* tag_next = s.heavy_tag + (size_t)(L & 1u) * nf;
  const unsigned H = s.qctl[1 + ((L + 1u) & 1u)];
  const unsigned thr = s.qctl[4];
  LaneStage<R> LS;
  lane_stage(p, g, LS);
  StageCtx sc;
  sc.p = &p;
  sc.m = s.mt;
  sc.hold_base = s.mt_hold;
  sc.hold_epoch_base = s.hold_epoch;
  sc.f = 0;
  sc.my_hold_epoch = s.hold_epoch;
  Fru4<R> F;
  F.clk = {};
  F.jsr.set(0.0);
  F.ss.set(0.0);
  F.w = 0u;
  F.nsub = 0u;
  F.mti = 0;
  int f = -1;
  bool overflow = false;
  // the next FRU of the queue (every lane of the group gets it; -1: none left)
  auto take = [&]() -> int {
    int got = -1;
    if (g.c == 0) {
      for (int tries = 0; tries <= n + (int)H; tries++) {
        const unsigned i = atomicAdd(s.qctl, 1u);
        if (i < H) {
          got = heavy_prev[i];
          break;
        }
        const unsigned j = i - H;
        if (j >= (unsigned)n) break;
        if (H == 0u || tag_prev[j] != L) {  // tag L: in the previous launch's heavy list
          got = (int)j;
          break;
        }
      }
    }
    return __shfl_sync(g.mask, got, g.base);
  };
  auto load = [&](int ff) {
    f = ff;
    sc.f = ff;
    sc.my_hold_epoch = s.hold_epoch + ff;
    bool restore = false;
    if (p.flags & kFlagResume) {
      F.jsr.set(s.frus_s[ff]);
      F.ss.set(s.frus_s[(g.c + 1) * nf + ff]);
      F.w = s.chan_s[g.c * nf + ff];
      F.mti = s.mti_s[ff];
      restore = (*sc.my_hold_epoch == p.epoch);
    } else {
      F.jsr.set(s.frus[ff]);
      F.ss.set(s.frus[(g.c + 1) * nf + ff]);
      F.w = s.chan[g.c * nf + ff];
      F.mti = s.mti[ff];
    }
    if (p.flags & kFlagSave) {
      if (g.c == 0) {
        s.frus_s[ff] = F.jsr.get();
        s.mti_s[ff] = F.mti;
      }
      s.frus_s[(g.c + 1) * nf + ff] = F.ss.get();
      s.chan_s[g.c * nf + ff] = F.w;
    }
    use_row(sc, s.mt + (size_t)ff * kMtStride, s.mt_hold + (size_t)ff * kMtStride, restore, g);
    F.nsub = 0u;
    fru_begin(F, LS);
  };
  auto finish = [&]() {
    if (g.c == 0) {
      s.frus[f] = F.jsr.get();
      s.mti[f] = F.mti;
      if (s.trace_sub) s.trace_sub[f] = F.nsub;
      atomicAdd(&s.qctl[3], F.nsub);
      if (s.substeps) atomicAdd(s.substeps, (unsigned long long)F.nsub);
      if (F.nsub >= thr && thr > 0u) {
        tag_next[f] = L + 1u;
        heavy_next[atomicAdd(&s.qctl[1 + (L & 1u)], 1u)] = f;
      }
    }
    s.frus[(g.c + 1) * nf + f] = F.ss.get();
    s.chan[g.c * nf + f] = F.w;
  };
  {
    const int ff = take();
    if (ff >= 0) load(ff);
  }
  __syncwarp();
  while (true) {
    const bool has = f >= 0;
    bool go = has && F.clk.running(LS);
    if (go && F.nsub >= (1u << 22)) {
      overflow = true;
      go = false;
    }
    if (!__any_sync(0xffffffffu, has)) break;
    Sub4<R> S;
    sub_begin(S);
    if (go) substep_a(F, S, LS, g, sc);
    regen_step(sc, lane, g, go, F, S);
    if (go) substep_b(F, S, LS, g, sc);
    // a group whose FRU reached tf stores it and takes the next one
    if (has && !(go && F.clk.running(LS))) {
      finish();
      f = -1;
      const int ff = take();
      if (ff >= 0) load(ff);
    }
    __syncwarp();
  }
  if (overflow) out[kOutError] = 1.0;
}

// ---- many cells in one launch ------------------------------------------------
// Cell i owns blocks block0[i] .. block0[i+1]-1 of the grid (8 FRUs per
// warp); its parameters are params[i] and its totals go to outs[i*32 ..].
template <typename R>
__device__ __forceinline__ void batch_body(const BatchArgs& a) {
  // the cell of this block: binary search of the block prefix sums
  int lo = 0, hi = a.ncells - 1;
  const int b = blockIdx.x;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(&a.block0[mid]) <= b) lo = mid;
    else hi = mid - 1;
  }
  // the cell's arrays and parameters are read where used (through L1)
  // rather than copied into registers
  const DevState& s = a.cells[lo];
  const StageParams& p = a.params[lo];
  if (p.flags < 0) return;  // the cell posted no operation this round
  stage_body<R>(s, p, b - a.block0[lo], a.outs + kBatchOutStride * lo);
}

}  // namespace cleft
}  // namespace gw
