// FP64 division, reciprocal and exponential of the FRU substep with few
// instructions on the FP64 pipe.
//
// GB300 issues one FP64 warp instruction per 64 cycles per SM sub-partition,
// so the FRU stage kernels last as long as the FP64 instructions they issue.
// A division spends about eight there and an exponential about seventeen, and
// a substep has sixteen divisions and two exponentials per lane.  Here the
// parts that need no 53-bit arithmetic (seeds, argument reduction's integer,
// exponents) run on the FP32 and integer pipes, which are otherwise idle:
//   quotient            3 FP64 instructions (Markstein's final correction)
//   reciprocal          2
//   quotient by a constant 2 (Brisebarre, Muller and Raina)
//   exponential         7 (Tang's table-driven method)
// With the rest of the substep as it is in gw_fru_cleft.cuh, the five stages
// of one integration step at the peak of release took, before and after (one
// GB300, fixed layout): 250 FRUs 6.23 -> 3.92 ms, 12,500 FRUs 14.94 -> 8.98
// ms; in diastole 12,497 FRUs 3.08 -> 2.04 ms.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace gw {

// 1/b to about 45 bits for a normal b whose reciprocal is normal (the
// callers check the range).  b = m 2^e with m = mf + bl: mf the leading 24
// bits and bl the rest, both FP32 built from b's bits.  y0 = 1/mf to an FP32
// ulp; the residual 1 - m y0 is formed in FP32 (its first term is exact),
// and y0 (e + e^2) is added to y0's double as a multiple of its last place
// on the integer pipe (a double's bits are linear in its mantissa).
__device__ __forceinline__ double rcp_seed(double b) {
  const uint32_t hi = (uint32_t)__double2hiint(b), lo = (uint32_t)__double2loint(b);
  const float mf = __uint_as_float((__funnelshift_l(lo, hi, 3) & 0x007fffffu) | 0x3f800000u);
  // (the 29 low bits >> 6) + 1/2, in units of 2^-46
  const float bl = (__uint_as_float(((lo >> 6) & 0x007fffffu) | 0x4b000000u) - 8388607.5f) * 0x1p-46f;
  float y0;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(mf));
  float e = __fmaf_rn(-mf, y0, 1.0f);
  e = __fmaf_rn(-bl, y0, e);
  const float e2 = __fmaf_rn(e, e, e);
  const int ci = __float2int_rn(__fmul_rn(__fmul_rn(y0, 0x1p51f), e2));  // |e| <= 2^-22: |ci| < 2^30
  const uint32_t yb = __float_as_uint(y0);
  const uint64_t base = ((uint64_t)yb << 29) + ((uint64_t)(0x38000000u + (0x3ff00000u - (hi & 0xfff00000u))) << 32);
  return __longlong_as_double((long long)(base + ((uint64_t)(int64_t)ci << 2)));
}

// a / b and 1 / b for operands in the ranges fits() accepts.  With y within
// 2^-45 of 1/b, q = a y is within 2^-45 of a/b, the remainder a - q b is
// computed to 2^-53 of itself, and the last operation rounds q + r/b, known
// to 2^-90: the correctly rounded quotient, except where a/b lies within
// 2^-37 of a last place of a midpoint between two doubles.
// (P. W. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990.)
__device__ __forceinline__ double fast_div(double a, double b) {
  const double y = rcp_seed(b);
  const double q = a * y;
  return fma(fma(-b, q, a), y, q);
}
__device__ __forceinline__ double fast_rcp(double b) {
  const double y = rcp_seed(b);
  return fma(fma(-b, y, 1.0), y, y);
}
// 0x1p-100 <= x < 0x1p100 (false for negative, infinite and NaN x): a
// quotient of two such values and every intermediate above is normal.
__device__ __forceinline__ bool fits(double x) {
  return (uint32_t)__double2hiint(x) - (uint32_t)((1023 - 100) << 20) < (uint32_t)(200 << 20);
}

// a / b for any operands: the hardware's division where one is out of range.
__device__ __forceinline__ double checked_div(double a, double b) {
  return fits(fabs(a)) && fits(fabs(b)) ? fast_div(a, b) : a / b;
}

// x / d for a constant d: rhi = 1/d rounded, rlo = 1/d - rhi rounded; the
// two-instruction form returns the correctly rounded quotient for every finite
// x whose products do not underflow (|x| > 2^-900, far below any difference of
// two concentrations, or 0) for the constants below (N. Brisebarre, J.-M. Muller and S. K. Raina,
// "Accelerating correctly rounded floating-point division when the divisor
// is known in advance", IEEE Trans. Comput. 53, 2004; the finitely many x
// whose quotient lies close enough to a midpoint to matter are checked one
// by one in tests/test_fp64_math.py).
struct ConstDiv {
  double rhi, rlo;
};
__device__ __forceinline__ double const_div(double x, ConstDiv k) { return fma(x, k.rhi, x * k.rlo); }
#define GW_CONST_DIV(name, hi, lo) constexpr ConstDiv name = {hi, lo};
GW_CONST_DIV(kDiv5, 0x1.999999999999ap-3, -0x1.999999999999ap-57)        // 5.0
GW_CONST_DIV(kDiv12, 0x1.5555555555555p-4, 0x1.5555555555555p-58)        // 12.0
GW_CONST_DIV(kDivBL, 0x1.08847868898c9p-1, 0x1.0639772ca450bp-57)        // 1.9356
GW_CONST_DIV(kDivKrate, 0x1.890910cb01471p+9, 0x1.d2ef7237b73afp-45)     // 0.00127215
GW_CONST_DIV(kDivKrate2, 0x1.2b8532596fcf9p-2, 0x1.dd51fb96e28eep-56)    // 3.4188
GW_CONST_DIV(kDivTauss2ss, 0x1.4p+4, -0x1.4p-50)                         // 10.0 * 0.005
GW_CONST_DIV(kDivTauxfer, 0x1.9p+7, -0x1.2cp-48)                         // 0.005
GW_CONST_DIV(kDivTautr, 0x1.5555555555555p-2, 0x1.5555555555555p-56)     // 3.0
GW_CONST_DIV(kDivRTF, 0x1.32b8f17bfc76cp-5, 0x1.0c561143472dap-61)       // 8.314 * 310.0 / 96.5
#undef GW_CONST_DIV

// 2^(j/4096) as a rounded double and the remainder, j = 0 .. 4095 (written
// by build.py).
static __device__ const double2 g_exp2_table[4096] = {
#include "gw_exp2_table.h"
};

// exp(x).  x = k ln2/4096 + r with |r| <= 1.1 ln2/8192, exp(x) =
// 2^(k>>12) T[k & 4095] exp(r): k from an FP32 product and the double of k
// from its bits, so that the FP64 pipe sees only the reduction (two
// instructions), the polynomial of degree 3 (three; |error| < 2^-59) and the
// reconstruction (two).  Where |x| >= 64 the FP32 estimate of k could be
// further off and k is formed in FP64; |x| >= 600 and NaN take the library's
// exp.  (P. T. P. Tang, "Table-driven implementation of the exponential
// function in IEEE floating-point arithmetic", ACM TOMS 15, 1989.)
__device__ __forceinline__ double fexp(double x) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const uint32_t ah = hi & 0x7fffffffu;
  if (ah >= 0x4082c000u) return exp(x);  // 600.0
  int k;
  double kd;
  if (ah < 0x40500000u) {  // 64.0
    // |x| truncated to FP32 (0 below 2^-126, where k = 0 anyway)
    const float ax = __uint_as_float(__funnelshift_l(lo, max(ah, 0x38000000u) - 0x38000000u, 3));
    const float t = __fmaf_rn(__uint_as_float(__float_as_uint(ax) | (hi & 0x80000000u)), 5909.2788f, 12582912.0f);
    k = __float_as_int(t) - 0x4b400000;
    // k as a double (|k| < 2^20: its FP32 mantissa fits the high word; k = 0:
    // a number too small to matter)
    const uint32_t kb = __float_as_uint(__fadd_rn(t, -12582912.0f));
    kd = __hiloint2double((int)((((kb & 0x7fffffffu) >> 3) + 0x38000000u) | (kb & 0x80000000u)), 0);
  } else {
    kd = rint(x * 0x1.71547652b82fep+12);
    k = (int)kd;
  }
  const double2 T = __ldg(&g_exp2_table[k & 4095]);
  double r = fma(kd, -0x1.62e42fefa39efp-13, x);
  r = fma(kd, -0x1.abc9e3b39803fp-68, r);
  const double p = fma(r, 0x1.5555555555555p-3, 0x1.00000001553d7p-1);
  const double s = fma(r * r, p, r);
  const double e = T.x + fma(T.x, s, T.y);
  return __hiloint2double(__double2hiint(e) + ((k >> 12) << 20), __double2loint(e));
}

}  // namespace gw
