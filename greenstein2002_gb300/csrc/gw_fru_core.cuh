// Device building blocks of the FRU stage: the substep loop of one FRU and
// the deterministic flux reduction.  Shared by the FRU stage kernels.
//
// Reference: simfru_local.c:32-278, calc_fru_flux_local.c:28-77,
// mpi_master.c:447-468.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "gw_fru_model.cuh"
#include "gw_kernels.h"

namespace gw {

// Deterministic block reduction of NV doubles: warp shuffles, then warps in
// index order.  Result valid in thread 0.
template <int NV>
__device__ __forceinline__ void block_reduce(double v[NV], double* smem /* [32][NV] */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int k = 0; k < NV; k++)
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; k++) smem[warp * NV + k] = v[k];
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; k++) {
      double s = smem[k];
      for (int w = 1; w < nwarp; w++) s += smem[w * NV + k];
      v[k] = s;
    }
  }
  __syncthreads();
}

// Last-block pass: sum the per-block partials in a fixed order, so the result
// does not depend on which block finished last.  Returns true in thread 0 of
// the last block, with the totals in tot[].
template <int NV>
__device__ __forceinline__ bool grid_finish(const double v[NV], double* partials, unsigned* ticket, double* smem,
                                            double tot[NV]) {
  __shared__ bool last;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < NV; k++) partials[blockIdx.x * NV + k] = v[k];
    __threadfence();
    last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  double s[NV];
#pragma unroll
  for (int k = 0; k < NV; k++) s[k] = 0.0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x)
#pragma unroll
    for (int k = 0; k < NV; k++) s[k] += __ldcg(&partials[b * NV + k]);
  block_reduce<NV>(s, smem);
  if (threadIdx.x == 0) {
    *ticket = 0u;
#pragma unroll
    for (int k = 0; k < NV; k++) tot[k] = s[k];
  }
  return threadIdx.x == 0;
}

// ---- sums over the FRUs of a cell, the same bits for every launch shape ---------
// ND double sums and NI words of two 32-bit counts each: the counts (open
// channels and the like) are integers and need no FP64 additions.
template <int ND, int NI>
struct Sums {
  double d[ND];
  unsigned long long n[NI];
};
using FluxSums = Sums<3, 1>;  // CaSS, CaJSR, CaSS of open LCCs; open LCCs, open Cl channels
using AvgSums = Sums<6, 3>;   // FluxSums, JRyR, buffered CaSS and CaJSR; open and ready RyRs; LCCs in mode normal, open VDIs

// This lane's cleft (c; the FRU-level terms on the cleft-0 lane):
// calc_fru_flux_local.c:45-70 and calc_fru_avg_local.c:27-105.
template <int ND, int NI>
__device__ __forceinline__ void flux_terms(int c, double jsr, double ss, uint32_t w, Sums<ND, NI>& v) {
  v.d[0] = ss;
  v.d[1] = (c == 0) ? jsr : 0.0;
  v.d[2] = lcc_open(w) ? ss : 0.0;
  v.n[0] = (unsigned long long)(lcc_open(w) ? 1u : 0u) | ((unsigned long long)((cl_of(w) == 2) ? 1u : 0u) << 32);
}
__device__ __forceinline__ void avg_terms(int c, double jsr, double ss, uint32_t w, AvgSums& v) {
  flux_terms(c, jsr, ss, w, v);
  unsigned no = 0, ready = 0;
#pragma unroll
  for (int i = 0; i < kRyR; i++) {
    const int r = ryr_of(w, i);
    no += ryr_open(r);
    ready += (r == 1 || r == 2);
  }
  v.d[3] = JRyRmax * ((double)no) * (jsr - ss);
  v.d[4] = ss * (1.0 + BSRtot / (KBSR + ss) + BSLtot / (KBSL + ss));
  v.d[5] = (c == 0) ? jsr * (1.0 + CSQNtot / (KmCSQN + jsr)) : 0.0;
  v.n[1] = (unsigned long long)no | ((unsigned long long)ready << 32);
  v.n[2] = (unsigned long long)((lcc_of(w) <= 6) ? 1u : 0u) | ((unsigned long long)((vdi_of(w) == 2) ? 1u : 0u) << 32);
}
// the 5 flux numerators, and the 11 output sums after them
template <int ND, int NI>
__device__ __forceinline__ void unpack_flux(const Sums<ND, NI>& v, double tot[5]) {
#pragma unroll
  for (int k = 0; k < 3; k++) tot[k] = v.d[k];
  tot[3] = (double)(uint32_t)v.n[0];
  tot[4] = (double)(uint32_t)(v.n[0] >> 32);
}
__device__ __forceinline__ void unpack_avg(const AvgSums& v, double tot[16]) {
  unpack_flux(v, tot);
  const double a[11] = {v.d[0], v.d[1], v.d[3], (double)(uint32_t)v.n[1], (double)(uint32_t)(v.n[1] >> 32), v.d[4], v.d[5],
                        (double)(uint32_t)v.n[2], (double)(uint32_t)(v.n[2] >> 32), tot[3], tot[4]};
#pragma unroll
  for (int k = 0; k < 11; k++) tot[5 + k] = a[k];
}

// Over the 32 lanes of a warp by one fixed shuffle tree; the total in lane 0.
template <int ND, int NI>
__device__ __forceinline__ void warp_sum(Sums<ND, NI>& v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int k = 0; k < ND; k++) v.d[k] += __shfl_down_sync(0xffffffffu, v.d[k], o);
#pragma unroll
    for (int k = 0; k < NI; k++) v.n[k] += __shfl_down_sync(0xffffffffu, v.n[k], o);
  }
}
// Partial sums of group i.
template <int ND, int NI>
__device__ __forceinline__ void put_partial(const DevState& s, int i, const Sums<ND, NI>& v) {
  double* q = s.partials + (size_t)i * (ND + NI);
#pragma unroll
  for (int k = 0; k < ND; k++) q[k] = v.d[k];
#pragma unroll
  for (int k = 0; k < NI; k++) q[ND + k] = __longlong_as_double((long long)v.n[k]);
}
template <int ND, int NI>
__device__ __forceinline__ void get_partial(const DevState& s, int i, Sums<ND, NI>& v) {
  const double* q = s.partials + (size_t)i * (ND + NI);
#pragma unroll
  for (int k = 0; k < ND; k++) v.d[k] = __ldcg(q + k);
#pragma unroll
  for (int k = 0; k < NI; k++) v.n[k] = (unsigned long long)__double_as_longlong(__ldcg(q + ND + k));
}
// The warp's lanes (8 FRUs x 4 clefts) into group grp's partial sums.
template <int ND, int NI>
__device__ __forceinline__ void store_group(const DevState& s, int grp, Sums<ND, NI>& v, int lane) {
  warp_sum(v);
  if (lane == 0) put_partial(s, grp, v);
}

// Cross-FRU sums of one cell, independent of the launch shape: the warp that
// stores the cell's last group adds the groups lane-strided (groups lane,
// lane + 32, ... one after another) and by one warp tree.  Three dependent
// FP64 additions per 32 groups: the counts are integers (as doubles they made
// it five).
// Called by a warp that has stored `count` groups; true (in every lane) when
// that completed the cell, with the totals in lane 0's v.  The ticket counts
// groups and is reset by the warp that completes the cell.
template <int ND, int NI>
__device__ __forceinline__ bool finish_groups(const DevState& s, Sums<ND, NI>& v, unsigned count, int lane) {
  const int ngroups = (s.nfru + 7) >> 3;
  unsigned last = 0u;
  if (lane == 0) {
    __threadfence();
    last = (atomicAdd(s.ticket, count) + count == (unsigned)ngroups) ? 1u : 0u;
  }
  if (!__shfl_sync(0xffffffffu, last, 0)) return false;
  __syncwarp();  // lane 0's count before every lane's reads (a shuffle orders no memory)
  __threadfence();
  v = {};
#pragma unroll 8
  for (int b = lane; b < ngroups; b += 32) {
    Sums<ND, NI> t;
    get_partial(s, b, t);
#pragma unroll
    for (int k = 0; k < ND; k++) v.d[k] += t.d[k];
#pragma unroll
    for (int k = 0; k < NI; k++) v.n[k] += t.n[k];
  }
  warp_sum(v);
  if (lane == 0) *s.ticket = 0u;
  return true;
}

// Flux numerators -> (Jxfer, Jtr, ICa, Ito2): mpi_master.c:447-468.
static __device__ inline void currents_from_sums(int nfru, double scale, const double dep[3], const double num[5], double out[4]) {
  const double V = dep[0], Cai = dep[1], CaNSR = dep[2];
  const double VFRT = V / RT_over_F, VFsqRT = (1000.0 * Faraday) * VFRT;
  const double e1 = exp(VFRT), e2 = e1 * e1;
  double ica, ito2;
  if (fabs(V) < 1.e-6) {
    const double icanum = num[2] - num[3] * Cao * 0.341;
    ica = PCa * 2.0 * 1000.0 * Faraday * icanum;
    ica = ica / Acap;
    ito2 = num[4] * PCl * 1000.0 * Faraday * (Clo - Cli);
    ito2 = ito2 / Acap;
  } else {
    const double icanum = num[2] * e2 - num[3] * Cao * 0.341;
    ica = PCa * 4.0 * VFsqRT * icanum / (e2 - 1.0);
    ica = ica / Acap;
    ito2 = num[4] * PCl * VFsqRT * (Cli - Clo * e1) / (1.0 - e1);
    ito2 = ito2 / Acap;
  }
  const double jtr = (((double)nfru) * CaNSR - num[1]) / tautr;
  const double jxfer = (num[0] - ((double)nfru * (double)kClefts) * Cai) / tauxfer;
  out[0] = scale * jxfer;
  out[1] = scale * jtr;
  out[2] = scale * ica;
  out[3] = scale * ito2;
}

// a / b for a divisor in the fast form's range; a zero, of a cell without
// open channels, keeps the sign of the product (the fast form's last sum makes
// it +0).  `plain` is set where a is out of range (infinite, NaN).
__device__ __forceinline__ double current_div(double a, double b, bool& plain) {
  const bool zero = (__double_as_longlong(a) << 1) == 0;
  plain = plain || !(zero || fits(fabs(a)));
  const double y = rcp_seed(b), q = a * y;
  const double f = fma(fma(-b, q, a), y, q);
  return zero ? q : f;
}

// The currents of a launch's totals, one per lane: on return lanes 0..3 hold
// Jxfer, Jtr, ICa, Ito2 in cur.  num: the flux numerators, the same in every
// lane.  One instruction stream for the four (36 FP64 instructions; on one
// lane one after another about 120, 4 us of every launch): a product and a
// difference, two quotients and the scale, the operands selected by lane.
// Potentials at 0 or beyond 500 mV and numerators out of the quotients' range
// take the plain expressions.
// GW_CONTRACT (the mixed-precision unit): products feeding a difference are
// fused, as the compiler fuses currents_from_sums there.
__device__ __forceinline__ double lane_current(const DevState& s, const StageParams& p, const double num[5], int lane) {
  const double V = p.depf[0];
  const long long av = __double_as_longlong(V) & 0x7fffffffffffffffLL;
  bool plain = av < __double_as_longlong(1.e-6) || av >= __double_as_longlong(500.0);
  if (!plain) {
    const double VFRT = const_div(V, kDivRTF), VFsqRT = (1000.0 * Faraday) * VFRT;
    const double e1 = exp(VFRT), e2 = e1 * e1;
    const double n = (double)s.nfru;
    const double c = num[3] * Cao;
    // x * y, subtracted from or less the other operand z (lane 2: z = (num3 Cao) 0.341)
    const double x = lane == 0 ? n * (double)kClefts : lane == 1 ? n : lane == 2 ? num[2] : Clo;
    const double y = lane == 0 ? p.depf[1] : lane == 1 ? p.depf[2] : lane == 2 ? e2 : e1;
    const double z = lane == 0 ? num[0] : lane == 1 ? num[1] : lane == 2 ? c * 0.341 : Cli;
    const bool minus = lane == 0 || lane == 3;  // z - x y, else x y - z
#ifdef GW_CONTRACT
    double b = fma(minus ? -x : x, y, minus ? z : -z);
#else
    const double xy = x * y;
    double b = (minus ? z : xy) - (minus ? xy : z);
#endif
    const double a = (lane == 2 ? PCa * 4.0 : num[4] * PCl) * VFsqRT;
    const double ab = a * b;
    b = lane >= 2 ? ab : b;
    const double em1 = (lane == 2 ? e2 : 1.0) - (lane == 2 ? 1.0 : e1);
    const double q = current_div(b, lane == 0 ? tauxfer : lane == 1 ? tautr : em1, plain);
    const double r = current_div(q, Acap, plain);
    const double cur = p.nfru_scale * (lane >= 2 ? r : q);
    if (!plain) return lane == 2 ? cur * p.pca_scale : cur;  // ICa is proportional to the LCC permeability
  }
  double cur[4];
  currents_from_sums(s.nfru, p.nfru_scale, p.depf, num, cur);
  return lane == 0 ? cur[0] : lane == 1 ? cur[1] : lane == 2 ? cur[2] * p.pca_scale : cur[3];
}

// Categorical selection of simfru_local.c:217-226 for a channel that has left
// its state (u > 1 - dt*total): walk the cumulative probabilities.
__device__ __forceinline__ int pick_dest(const double r[4], const int d[4], int len, double dt, double u) {
  double acc = 1.0 - dt * r[0];
  int n = 1;
  acc += dt * r[1];
  while (u > acc && n + 1 < len) {
    n++;
    acc += dt * r[n];
  }
  return d[n];
}

// Upper bound on substeps of one FRU in one stage.  Valid states need far
// fewer (dt >= 0.1 / max exit rate, and rates are bounded); corrupted input
// (NaN or huge concentrations) stops here with an error flag instead of
// looping without end.
constexpr uint32_t kMaxSubsteps = 1u << 22;

// One FRU over [t0, tf]: simfru_local.c:83-277.
__device__ __forceinline__ void advance_fru(const StageParams& p, double y[5], uint32_t w[kClefts], MtRef& rng,
                                            uint32_t& nsub, bool& overflow) {
  double dep[3], lopen[kClefts], R0[32];
  int nopen[kClefts];
#pragma unroll
  for (int i = 0; i < 3; i++) dep[i] = p.dep0[i];
#pragma unroll
  for (int c = 0; c < kClefts; c++) {
    lopen[c] = lcc_open(w[c]) ? 1.0 : 0.0;
    nopen[c] = ryr_open_count(w[c]);
  }
  const double interval = p.tf - p.t0;
  double t = p.t0;
  while (t < p.tf) {
    if (nsub >= kMaxSubsteps) {
      overflow = true;
      break;
    }
    // ---- exit rates at the substep start (fru_rates_local.c:126-777) ----
    const LccBasis lb = lcc_basis(dep[0]);
    const double nu = 1.0;
    const double yinf = nu * (0.4 / (1.0 + fexp((dep[0] + 12.5) / 5.0)) + (1.0 - 0.4));
    const double tau = 60.0 + 340.0 / (1.0 + fexp((dep[0] + 30.0) / 12.0));
    const double vdi_open_rate = (1.0 - yinf) / tau, vdi_closed_rate = yinf / tau;
    double cass0[kClefts];
#pragma unroll
    for (int c = 0; c < kClefts; c++) {
      cass0[c] = y[c + 1];
      R0[8 * c + 0] = lcc_total(lcc_of(w[c]), lb, gammacf * y[c + 1]);
      R0[8 * c + 1] = (vdi_of(w[c]) == 2) ? vdi_open_rate : vdi_closed_rate;
    }
#pragma unroll
    for (int c = 0; c < kClefts; c++) {
      const RyrK k = ryr_constants(y[c + 1]);
#pragma unroll
      for (int i = 0; i < kRyR; i++) {
        const int s = ryr_resolve(ryr_of(w[c], i), k, rng);
        w[c] = set_field(w[c], 8 + 4 * i, s);
        R0[8 * c + 2 + i] = ryr_total(s, k);
      }
      R0[8 * c + 7] = (cl_of(w[c]) == 1) ? kfIto2 * y[c + 1] : kbIto2;
    }
    double mx = 0.0;
#pragma unroll
    for (int c = 0; c < kClefts; c++) {
      mx = dmax(mx, R0[8 * c + 0]);
      mx = dmax(mx, R0[8 * c + 1]);
      mx = dmax(mx, R0[8 * c + 7]);
#pragma unroll
      for (int i = 0; i < kRyR; i++) mx = dmax(mx, R0[8 * c + 2 + i]);
    }
    // ---- substep size (simfru_local.c:135-146) ----
    double dt = dmin(0.1 / mx, 10.001e-3);
    double cmax = 0.e-3;
#pragma unroll
    for (int c = 0; c < kClefts; c++) cmax = dmax(cmax, y[c + 1]);
    if (cmax > 1.5e-3) dt = dmin(dt, 5.001e-3);
    dt = dmin(dt, p.tf - t);
    // ---- Heun step of the local Ca ODE with pre-transition flags (:149-173) ----
    double k1[5], y1[5], dF[5];
    fcn_fru(y, dep, lopen, nopen, dF);
#pragma unroll
    for (int i = 0; i < 5; i++) {
      k1[i] = dt * dF[i];
      y1[i] = y[i] + k1[i];
    }
    t = t + dt;
#pragma unroll
    for (int i = 0; i < 3; i++) dep[i] = p.dep0[i] + (t - p.t0) / interval * p.span[i];
    fcn_fru(y1, dep, lopen, nopen, dF);
#pragma unroll
    for (int i = 0; i < 5; i++) y[i] = y[i] + (k1[i] + dt * dF[i]) / 2.0;
    // ---- 32 uniforms and transitions (:211-276) ----
#pragma unroll
    for (int c = 0; c < kClefts; c++) {
      bool moved = false;
      // LCC
      {
        const double u = rng.next();
        if (u > 1.0 - dt * R0[8 * c]) {
          double r[4];
          int d[4];
          const int len = lcc_row(lcc_of(w[c]), lb, gammacf * cass0[c], r, d);
          w[c] = set_field(w[c], 0, pick_dest(r, d, len, dt, u));
        }
      }
      // voltage-dependent inactivation gate
      {
        const double u = rng.next();
        if (u >= 1.0 - dt * R0[8 * c + 1]) w[c] = set_field(w[c], 4, 3 - vdi_of(w[c]));
      }
      // RyRs
#pragma unroll
      for (int i = 0; i < kRyR; i++) {
        const double u = rng.next();
        if (u > 1.0 - dt * R0[8 * c + 2 + i]) {
          const RyrK k = ryr_constants(cass0[c]);
          double r[4];
          int d[4];
          const int len = ryr_row(ryr_of(w[c], i), k, r, d);
          w[c] = set_field(w[c], 8 + 4 * i, pick_dest(r, d, len, dt, u));
          moved = true;
        }
      }
      // Ca-activated Cl channel
      {
        const double u = rng.next();
        if (u >= 1.0 - dt * R0[8 * c + 7]) w[c] = set_field(w[c], 28, 3 - cl_of(w[c]));
      }
      lopen[c] = lcc_open(w[c]) ? 1.0 : 0.0;
      if (moved) nopen[c] = ryr_open_count(w[c]);
    }
    nsub++;
  }
}

}  // namespace gw
