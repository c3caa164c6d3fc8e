// Measured FP64 FMA peak of the device: independent DFMA chains on every SM.
// The FRU stage kernel is FP64-pipe bound and the pool's measured-peak file
// lists no FP64 figure, so the benchmark measures this denominator in-run.
#include <cuda_runtime.h>

#include <chrono>

#include "gw_cell_model.h"
#include "gw_dp_device.cuh"
#include "gw_fp64_math.cuh"
#include "gw_intdiv.h"
#include "gw_kernels.h"

namespace gw {

__global__ void fp64_fma_loop(double* out, int iters, double a, double b) {
  double x0 = threadIdx.x * 1e-9, x1 = x0 + 1e-3, x2 = x0 + 2e-3, x3 = x0 + 3e-3;
  double x4 = x0 + 4e-3, x5 = x0 + 5e-3, x6 = x0 + 6e-3, x7 = x0 + 7e-3;
  for (int i = 0; i < iters; i++) {
    x0 = fma(x0, a, b); x1 = fma(x1, a, b); x2 = fma(x2, a, b); x3 = fma(x3, a, b);
    x4 = fma(x4, a, b); x5 = fma(x5, a, b); x6 = fma(x6, a, b); x7 = fma(x7, a, b);
  }
  const double s = ((x0 + x1) + (x2 + x3)) + ((x4 + x5) + (x6 + x7));
  if (s == 123.456) out[blockIdx.x * blockDim.x + threadIdx.x] = s;  // keeps the chains live
}

cudaError_t probe_fp64(int sms, double* tflops) {
  const int threads = 256, blocks = sms * 8, iters = 4096;
  double* out = nullptr;
  cudaEvent_t e0, e1;
  cudaError_t e = cudaMalloc(&out, sizeof(double) * threads * blocks);
  if (e != cudaSuccess) return e;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  double best = 0.0;
  for (int rep = 0; rep < 4 && e == cudaSuccess; rep++) {
    cudaEventRecord(e0);
    fp64_fma_loop<<<blocks, threads>>>(out, iters, 0.999999, 1e-7);
    cudaEventRecord(e1);
    e = cudaEventSynchronize(e1);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
    const double flops = 2.0 * 8.0 * (double)iters * threads * blocks;
    if (e == cudaSuccess && rep > 0 && ms > 0.f) best = fmax(best, flops / (ms * 1e-3) / 1e12);
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  *tflops = best;
  return e;
}

// Cost of the global right-hand side (fcn.c:29-1072) on one GPU thread:
// `calls` dependent evaluations at the rest state.  Every derivative and
// current feeds the next call's V by a negligible amount, so no part of the
// evaluation can be skipped.
__host__ __device__ inline double fcn_feedback(const double* F, const double* cur) {
  double s = 0.0;
  for (int i = 0; i < GW_NSTATE; i++) s += F[i];
  for (int i = 0; i < GW_NCUR; i++) s += cur[i];
  return 1e-300 * s;
}

__global__ void fcn_chain(const gw_protocol* P, int calls, double* out) {
  double y[GW_NSTATE], F[GW_NSTATE], cur[GW_NCUR];
  gw_rest_state(y);
  for (int i = 0; i < calls; i++) {
    gw_fcn(10.5, y, F, cur, 1, 1e-6, 1e-6, -1e-3, 0.0, P);
    y[GW_V] = y[GW_V] + fcn_feedback(F, cur);
  }
  out[0] = y[GW_V];
}

cudaError_t probe_fcn(double* device_us, double* host_us) {
  const int calls = 200;
  gw_protocol hp;
  gw_protocol_defaults(&hp);
  gw_protocol* dp = nullptr;
  double* out = nullptr;
  cudaEvent_t e0, e1;
  cudaError_t e = cudaMalloc(&dp, sizeof hp);
  if (e == cudaSuccess) e = cudaMalloc(&out, sizeof(double));
  if (e == cudaSuccess) e = cudaMemcpy(dp, &hp, sizeof hp, cudaMemcpyHostToDevice);
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  float best = 1e30f;
  for (int rep = 0; rep < 3 && e == cudaSuccess; rep++) {
    cudaEventRecord(e0);
    fcn_chain<<<1, 1>>>(dp, calls, out);
    cudaEventRecord(e1);
    e = cudaEventSynchronize(e1);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
    if (e == cudaSuccess && rep > 0) best = ms < best ? ms : best;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(dp);
  cudaFree(out);
  *device_us = 1e3 * best / calls;
  // the same chain on the host
  double y[GW_NSTATE], F[GW_NSTATE], cur[GW_NCUR];
  gw_rest_state(y);
  const auto t0 = std::chrono::steady_clock::now();
  for (int i = 0; i < 20 * calls; i++) {
    gw_fcn(10.5, y, F, cur, 1, 1e-6, 1e-6, -1e-3, 0.0, &hp);
    y[GW_V] = y[GW_V] + fcn_feedback(F, cur);
  }
  const double us = std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t0).count();
  volatile double sink = y[GW_V];
  (void)sink;
  *host_us = us / (20 * calls);
  return e;
}

// exp as the FRU substep evaluates it (fexp), element-wise,
// next to the host libm's: the FRU path's only transcendental (rates
// fru_rates_local.c:131-132, :346-348; GHK fcn_fru.c:80; currents
// mpi_master.c:406), so the only arithmetic the device cannot share with
// the reference's host build bit for bit.
__global__ void exp_map(const double* x, double* y, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = fexp(x[i]);
}

cudaError_t probe_exp(const double* x, double* device_y, double* host_y, int n) {
  double *dx = nullptr, *dy = nullptr;
  cudaError_t e = cudaMalloc(&dx, sizeof(double) * n);
  if (e == cudaSuccess) e = cudaMalloc(&dy, sizeof(double) * n);
  if (e == cudaSuccess) e = cudaMemcpy(dx, x, sizeof(double) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    exp_map<<<(n + 255) / 256, 256>>>(dx, dy, n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(device_y, dy, sizeof(double) * n, cudaMemcpyDeviceToHost);
  cudaFree(dx);
  cudaFree(dy);
  for (int i = 0; i < n; i++) host_y[i] = exp(x[i]);
  return e;
}

// FP64 issue cost on one SM: clock64()-timed chains of 4096 dependent (or 8
// independent) operations -- DFMA with 32/16/4/1 active lanes and 1-16 warps,
// a DDIV+DADD chain, an exp() chain and an FP32 FFMA chain.  Each kernel runs
// one block; out[1] receives warp 0's cycles per operation.
__global__ void issue_dep_fma(double* out, int n, int active, double a, double b) {
  if ((int)(threadIdx.x & 31) >= active) return;
  double x = threadIdx.x * 1e-6;
  const long long t0 = clock64();
  for (int i = 0; i < n; i++) x = fma(x, a, b);
  const long long t1 = clock64();
  if (threadIdx.x == 0) {
    out[0] = x;
    out[1] = (double)(t1 - t0) / n;
  } else if (x == 1.2345) {
    out[2] = x;
  }
}
__global__ void issue_ind_fma(double* out, int n, double a, double b) {
  double x0 = threadIdx.x, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3, x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6, x7 = x0 + 7;
  const long long t0 = clock64();
  for (int i = 0; i < n; i++) {
    x0 = fma(x0, a, b); x1 = fma(x1, a, b); x2 = fma(x2, a, b); x3 = fma(x3, a, b);
    x4 = fma(x4, a, b); x5 = fma(x5, a, b); x6 = fma(x6, a, b); x7 = fma(x7, a, b);
  }
  const long long t1 = clock64();
  const double s = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
  if (threadIdx.x == 0) {
    out[0] = s;
    out[1] = (double)(t1 - t0) / (8.0 * n);
  } else if (s == 1.2345) {
    out[2] = s;
  }
}
__global__ void issue_dep_div(double* out, int n, int active) {
  if ((int)(threadIdx.x & 31) >= active) return;
  double x = 1.0 + threadIdx.x * 1e-6;
  const long long t0 = clock64();
  for (int i = 0; i < n; i++) x = 1.0000001 + 1.0 / x;
  const long long t1 = clock64();
  if (threadIdx.x == 0) {
    out[0] = x;
    out[1] = (double)(t1 - t0) / n;
  } else if (x == 1.2345) {
    out[2] = x;
  }
}
__global__ void issue_dep_exp(double* out, int n, int active) {
  if ((int)(threadIdx.x & 31) >= active) return;
  double x = 0.1 + threadIdx.x * 1e-6;
  const long long t0 = clock64();
  for (int i = 0; i < n; i++) x = exp(-x);
  const long long t1 = clock64();
  if (threadIdx.x == 0) {
    out[0] = x;
    out[1] = (double)(t1 - t0) / n;
  } else if (x == 1.2345) {
    out[2] = x;
  }
}
__global__ void issue_dep_ffma(double* out, int n, float a, float b) {
  float x = threadIdx.x * 1e-6f;
  const long long t0 = clock64();
  for (int i = 0; i < n; i++) x = fmaf(x, a, b);
  const long long t1 = clock64();
  if (threadIdx.x == 0) {
    out[0] = x;
    out[1] = (double)(t1 - t0) / n;
  } else if (x == 1.2345f) {
    out[2] = x;
  }
}

cudaError_t probe_fp64_issue(double* cycles) {
  double* d = nullptr;
  double h[3];
  const int n = 4096;
  cudaError_t e = cudaMalloc(&d, 3 * sizeof(double));
  int k = 0;
  auto take = [&]() {
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost);
    cycles[k++] = (e == cudaSuccess) ? h[1] : -1.0;
  };
  for (int act : {32, 16, 4, 1}) {
    if (e == cudaSuccess) issue_dep_fma<<<1, 32>>>(d, n, act, 0.999999, 1e-7);
    take();
  }
  for (int w : {1, 2, 4, 8}) {
    if (e == cudaSuccess) issue_dep_fma<<<1, 32 * w>>>(d, n, 32, 0.999999, 1e-7);
    take();
  }
  for (int w : {1, 4, 16}) {
    if (e == cudaSuccess) issue_ind_fma<<<1, 32 * w>>>(d, n, 0.999999, 1e-7);
    take();
  }
  for (int act : {32, 1}) {
    if (e == cudaSuccess) issue_dep_div<<<1, 32>>>(d, n, act);
    take();
  }
  for (int act : {32, 1}) {
    if (e == cudaSuccess) issue_dep_exp<<<1, 32>>>(d, n, act);
    take();
  }
  if (e == cudaSuccess) issue_dep_ffma<<<1, 32>>>(d, n, 0.999f, 1e-3f);
  take();
  cudaFree(d);
  return e;
}

// gw_div_rn (division on the integer pipe, which no kernel uses) against the
// hardware division on the device: every thread draws operand pairs from a
// splitmix64 stream -- arbitrary bit patterns, then normal operands of
// magnitude 1e-8 .. 1e4 (the FRU substep's range) -- and counts quotients
// whose bits differ.
__device__ __forceinline__ uint64_t div_probe_next(uint64_t& st) {
  uint64_t z = (st += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

__global__ void div_probe_kernel(uint64_t seed, long long per_thread, unsigned long long* bad) {
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  uint64_t st = seed ^ (tid * 0xd1342543de82ef95ull);
  unsigned long long nbad = 0;
  for (long long i = 0; i < per_thread; i++) {
    uint64_t a = div_probe_next(st), b = div_probe_next(st);
    if (i & 1) {
      const uint64_t ea = 1023 - 27 + div_probe_next(st) % 41, eb = 1023 - 27 + div_probe_next(st) % 41;
      a = (a & 0x800fffffffffffffull) | (ea << 52);
      b = (b & 0x800fffffffffffffull) | (eb << 52);
    }
    const double x = __longlong_as_double((long long)a), y = __longlong_as_double((long long)b);
    const double q = x / y, g = gw_div_rn(x, y);
    const bool same = __double_as_longlong(q) == __double_as_longlong(g) || (q != q && g != g);
    nbad += same ? 0ull : 1ull;
  }
  if (nbad) atomicAdd(bad, nbad);
}

cudaError_t probe_div(unsigned long long seed, long long n, unsigned long long* mismatches) {
  const int threads = 256, blocks = 152 * 8;
  const long long per = (n + (long long)threads * blocks - 1) / ((long long)threads * blocks);
  unsigned long long* d = nullptr;
  cudaError_t e = cudaMalloc(&d, sizeof *d);
  if (e == cudaSuccess) e = cudaMemset(d, 0, sizeof *d);
  if (e == cudaSuccess) {
    div_probe_kernel<<<blocks, threads>>>(seed, per, d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(mismatches, d, sizeof *d, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e;
}

// The FRU substep's quotients, reciprocals and quotients by its constants
// (gw_fp64_math.cuh) against the hardware division: operands of magnitude
// 1e-8 .. 1e4 drawn as above; bad[0..2] count results whose bits differ.
__global__ void fp64_math_probe_kernel(uint64_t seed, long long per_thread, unsigned long long* bad) {
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  uint64_t st = seed ^ (tid * 0xd1342543de82ef95ull);
  const ConstDiv k[9] = {kDiv5, kDiv12, kDivBL, kDivKrate, kDivKrate2, kDivTauss2ss, kDivTauxfer, kDivTautr, kDivRTF};
  const double d[9] = {5.0, 12.0, 1.9356 * 1.0, 0.00127215, 3.4188, 10.0 * 0.005, 0.005, 3.0, 8.314 * 310.0 / 96.5};
  unsigned nq = 0, nr = 0, nc = 0;
  for (long long i = 0; i < per_thread; i++) {
    uint64_t a = div_probe_next(st), b = div_probe_next(st);
    const uint64_t ea = 1023 - 27 + div_probe_next(st) % 41, eb = 1023 - 27 + div_probe_next(st) % 41;
    a = (a & 0x800fffffffffffffull) | (ea << 52);
    b = (b & 0x800fffffffffffffull) | (eb << 52);
    const double x = __longlong_as_double((long long)a), y = __longlong_as_double((long long)b);
    nq += __double_as_longlong(x / y) != __double_as_longlong(fast_div(x, y));
    nr += __double_as_longlong(1.0 / y) != __double_as_longlong(fast_rcp(y));
    const int c = (int)(i % 9);
    nc += __double_as_longlong(x / d[c]) != __double_as_longlong(const_div(x, k[c]));
  }
  if (nq) atomicAdd(bad, (unsigned long long)nq);
  if (nr) atomicAdd(bad + 1, (unsigned long long)nr);
  if (nc) atomicAdd(bad + 2, (unsigned long long)nc);
}

cudaError_t probe_fp64_math(unsigned long long seed, long long n, unsigned long long* mismatches) {
  const int threads = 256, blocks = 152 * 8;
  const long long per = (n + (long long)threads * blocks - 1) / ((long long)threads * blocks);
  unsigned long long* d = nullptr;
  cudaError_t e = cudaMalloc(&d, 3 * sizeof *d);
  if (e == cudaSuccess) e = cudaMemset(d, 0, 3 * sizeof *d);
  if (e == cudaSuccess) {
    fp64_math_probe_kernel<<<blocks, threads>>>(seed, per, d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(mismatches, d, 3 * sizeof *d, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e;
}

// fcn of n states at `time`: one thread (gw_fcn) against a whole warp
// (the transcendental terms one per lane, tx_fill_warp, then gw_fcn_tx on
// every lane); derivatives and currents of both, for a bit-for-bit check.
__global__ void fcn_compare_kernel(const double* states, int n, const gw_protocol* P, double time, double* Fs,
                                   double* Fw, double* Cs, double* Cw) {
  __shared__ gw_tx tx;
  const int i = blockIdx.x, lane = threadIdx.x;
  if (i >= n) return;
  double y[GW_NSTATE], F[GW_NSTATE], cur[GW_NCUR];
  for (int k = 0; k < GW_NSTATE; k++) y[k] = states[(size_t)i * GW_NSTATE + k];
  if (lane == 0) {
    double ys[GW_NSTATE];
    for (int k = 0; k < GW_NSTATE; k++) ys[k] = y[k];
    gw_fcn(time, ys, F, cur, 1, 2e-6, 1e-6, -2e-3, 1e-4, P);
    for (int k = 0; k < GW_NSTATE; k++) Fs[(size_t)i * GW_NSTATE + k] = F[k];
    for (int k = 0; k < GW_NCUR; k++) Cs[(size_t)i * GW_NCUR + k] = cur[k];
  }
  __syncwarp();
  tx_fill_warp(time, y, P, &tx, lane);
  gw_fcn_tx(time, y, F, cur, 1, 2e-6, 1e-6, -2e-3, 1e-4, P, &tx, lane);
  if (lane == 0) {
    for (int k = 0; k < GW_NSTATE; k++) Fw[(size_t)i * GW_NSTATE + k] = F[k];
    for (int k = 0; k < GW_NCUR; k++) Cw[(size_t)i * GW_NCUR + k] = cur[k];
  }
}

cudaError_t probe_fcn_compare(const double* states, int n, double time, int clamp, double* Fs, double* Fw,
                              double* Cs, double* Cw) {
  gw_protocol hp;
  gw_protocol_defaults(&hp);
  if (clamp) {
    hp.vclamp_flag = 1;
    hp.vclamp_hold = -100.0;
    hp.vclamp_set = 0.0;
    hp.vclamp_shift = 0.0;
    hp.vclamp_duration = 200.0;
  }
  gw_protocol* dp = nullptr;
  double* d = nullptr;
  const size_t ns = (size_t)n * GW_NSTATE, nc = (size_t)n * GW_NCUR;
  cudaError_t e = cudaMalloc(&dp, sizeof hp);
  if (e == cudaSuccess) e = cudaMalloc(&d, sizeof(double) * (3 * ns + 2 * nc));
  if (e == cudaSuccess) e = cudaMemcpy(dp, &hp, sizeof hp, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d, states, sizeof(double) * ns, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    fcn_compare_kernel<<<n, 32>>>(d, n, dp, time, d + ns, d + 2 * ns, d + 3 * ns, d + 3 * ns + nc);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(Fs, d + ns, sizeof(double) * ns, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(Fw, d + 2 * ns, sizeof(double) * ns, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(Cs, d + 3 * ns, sizeof(double) * nc, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(Cw, d + 3 * ns + nc, sizeof(double) * nc, cudaMemcpyDeviceToHost);
  cudaFree(dp);
  cudaFree(d);
  return e;
}

// Microseconds per fcn evaluation on one warp (the transcendental terms one
// per lane), `calls` dependent evaluations as fcn_chain.
__global__ void fcn_chain_warp(const gw_protocol* P, int calls, double* out) {
  __shared__ gw_tx tx;
  const int lane = threadIdx.x;
  double y[GW_NSTATE], F[GW_NSTATE], cur[GW_NCUR];
  gw_rest_state(y);
  for (int i = 0; i < calls; i++) {
    tx_fill_warp(10.5, y, P, &tx, lane);
    gw_fcn_tx(10.5, y, F, cur, 1, 1e-6, 1e-6, -1e-3, 0.0, P, &tx, lane);
    y[GW_V] = y[GW_V] + fcn_feedback(F, cur);
    __syncwarp();
  }
  if (lane == 0) out[0] = y[GW_V];
}

cudaError_t probe_fcn_warp(double* us) {
  const int calls = 200;
  gw_protocol hp;
  gw_protocol_defaults(&hp);
  gw_protocol* dp = nullptr;
  double* out = nullptr;
  cudaEvent_t e0, e1;
  cudaError_t e = cudaMalloc(&dp, sizeof hp);
  if (e == cudaSuccess) e = cudaMalloc(&out, sizeof(double));
  if (e == cudaSuccess) e = cudaMemcpy(dp, &hp, sizeof hp, cudaMemcpyHostToDevice);
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  float best = 1e30f;
  for (int rep = 0; rep < 3 && e == cudaSuccess; rep++) {
    cudaEventRecord(e0);
    fcn_chain_warp<<<1, 32>>>(dp, calls, out);
    cudaEventRecord(e1);
    e = cudaEventSynchronize(e1);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
    if (e == cudaSuccess && rep > 0) best = ms < best ? ms : best;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(dp);
  cudaFree(out);
  *us = 1e3 * best / calls;
  return e;
}

}  // namespace gw
