// End of a step: the last CTA of the projection to finish turns the CTAs'
// partial sums and maxima into the step's scalars, so that the step needs no
// launch of its own for them (B200, FP64: 64^3 step 62 -> 59 us, 32^3 NS call
// 72 -> 69 us).
#pragma once
#include <math.h>
#include "common.cuh"

namespace mhit {

// M1, C3, R2 and the CFL guard (multi/main.f90:906-946) by one CTA of NT
// threads: means = sum/nx/ny/nz, removed lazily (stored in ctrl->mean and
// subtracted by every reader of u, v, w); gumax = max(max(u)-um, max(v)-vm,
// max(w)-wm), which equals the reference's max of the mean-removed fields
// because rounding is monotonic; then gamma, CFL, AB2 switch and the sticky
// error status.  Partials hold STRIDE values per CTA: sums of u, v, w, maxima
// of u, v, w, and (STRIDE 7, FP32 refine form) the max |div u| of the FP64
// projection.  The order of the sums depends on nparts and NT only.  Not
// inlined: one CTA runs it, and the loop before it keeps its own registers.
template <int NT, int STRIDE>
__device__ __noinline__ void finalize_step(const double* partials, int nparts, Ctrl* ctrl, double nd, double dt,
                                           double dxi) {
  static_assert(NT % 32 == 0, "whole warps");
  double v[7] = {0, 0, 0, -INFINITY, -INFINITY, -INFINITY, 0};
  for (int b = threadIdx.x; b < nparts; b += NT) {
#pragma unroll
    for (int t = 0; t < STRIDE; ++t) {
      const double x = __ldcg(partials + (size_t)b * STRIDE + t);
      v[t] = t < 3 ? v[t] + x : fmax(v[t], x);
    }
  }
  __shared__ double red[NT / 32][7];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int t = 0; t < 7; ++t) {
      const double x = __shfl_xor_sync(0xffffffffu, v[t], o);
      v[t] = t < 3 ? v[t] + x : fmax(v[t], x);
    }
  }
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int t = 0; t < 7; ++t) red[threadIdx.x >> 5][t] = v[t];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < NT / 32; ++w) {
#pragma unroll
      for (int t = 0; t < 7; ++t) red[0][t] = t < 3 ? red[0][t] + red[w][t] : fmax(red[0][t], red[w][t]);
    }
    const double um = red[0][0] / nd / nd / nd;
    const double vm = red[0][1] / nd / nd / nd;
    const double wm = red[0][2] / nd / nd / nd;
    const double uc = red[0][3] - um, vc = red[0][4] - vm, wc = red[0][5] - wm;
    const double umax = fmax(wc, fmax(uc, vc));
    const double cou = umax * dt * dxi;
    ctrl->mean[0] = um;
    ctrl->mean[1] = vm;
    ctrl->mean[2] = wm;
    ctrl->last_mean[0] = um;
    ctrl->last_mean[1] = vm;
    ctrl->last_mean[2] = wm;
    ctrl->gumax = umax;
    ctrl->cfl = cou;
    ctrl->alpha = 1.5;
    ctrl->beta = 0.5;
    ctrl->nstep += 1;
    const double s = red[0][0] + red[0][1] + red[0][2];
    // the maximum drops a NaN, which the sums of the same velocities keep
    ctrl->max_div = (STRIDE > 6) ? (s != s ? s : red[0][6]) : -1.0;
    if (!isfinite(s) || !isfinite(umax)) ctrl->status = 5;  // MHIT_ERR_NONFINITE
    else if (cou > ctrl->cfl_limit) ctrl->status = 4;      // MHIT_ERR_CFL
  }
}

// Called by every CTA of the projection after its thread 0 has written the
// CTA's partials: counts the CTA in, and the last of nparts runs
// finalize_step.  The count wraps to 0, ready for the next step.
template <int NT, int STRIDE>
__device__ __forceinline__ void finish_step(const double* partials, int nparts, Ctrl* ctrl, const StepConst& c) {
  __shared__ bool last;
  if (threadIdx.x == 0) {
    __threadfence();  // the partials, before the count
    last = atomicInc(&ctrl->ticket, (unsigned)(nparts - 1)) == (unsigned)(nparts - 1);
    __threadfence();  // the count, before the other CTAs' partials
  }
  __syncthreads();
  if (last) finalize_step<NT, STRIDE>(partials, nparts, ctrl, (double)c.n, c.dt, c.dxi);
}

}  // namespace mhit
