// On-GPU FP64 diagnostics of the resident state.
//
// The reference has no in-solver energy or dissipation output; its
// dissipation comes from the serial post-processor post/compute_diss
// (main.f90:72-117): eps = 2 nu <S_ij S_ij> with centred differences and
// periodic wrap on the stored (staggered) fields, dx = 2 pi/(nx-1) where pi is
// the default-real literal 3.14159265358979 of post/compute_diss/module.f90:5
// (so rounded to float32).  This kernel computes the same sum on the GPU, plus
// the kinetic energy 0.5<u^2+v^2+w^2>, the max |div u| of the projection's
// forward-difference divergence, and the phi volume sum and bounds.
#include <cuda_runtime.h>
#include <math.h>
#include "common.cuh"
#include "internal.h"

namespace mhit {

constexpr int DTX = 32, DTY = 8, DNT = DTX * DTY;
constexpr int NSTAT = 8;  // sum(u^2+v^2+w^2), sum(SijSij), max|div|, sum phi, min phi, max phi, sum u, pad
// z planes per CTA: 32 where the grid still fills the GPU, fewer below.
static int stats_planes(int n) { return n >= 256 ? 32 : (n >= 128 ? 8 : 4); }

// A thread marches one column up: its own u, v, w of planes k-1, k, k+1 pass
// through registers, and a plane's x and y neighbours come through L1 (15
// velocity loads per point instead of 21).  Each plane's loads are issued
// before its arithmetic.  256^3 FP64 on B200: Solver.stats 0.34 -> 0.25 ms.
template <class T>
__global__ void __launch_bounds__(DNT, 3) stats_kernel(const T* __restrict__ u, const T* __restrict__ v,
                                                       const T* __restrict__ w, const T* __restrict__ phi,
                                                       const Ctrl* __restrict__ ctrl, int n, int kz, double dxi_c,
                                                       double dxi_d, double* __restrict__ partials) {
  const double mu = ctrl->mean[0], mv = ctrl->mean[1], mw = ctrl->mean[2];
  const int i = blockIdx.x * DTX + threadIdx.x % DTX, j = blockIdx.y * DTY + threadIdx.x / DTX;
  const int ip = (i + 1 == n) ? 0 : i + 1, im = i ? i - 1 : n - 1;
  const int jp = (j + 1 == n) ? 0 : j + 1, jm = j ? j - 1 : n - 1;
  const size_t nn = (size_t)n * n;
  const unsigned oc = i + (unsigned)n * j, oxp = ip + (unsigned)n * j, oxm = im + (unsigned)n * j,
                 oyp = i + (unsigned)n * jp, oym = i + (unsigned)n * jm;
  const int k0 = blockIdx.z * kz;
  const double h = 0.5 * dxi_d;
  double s[NSTAT] = {0, 0, 0, 0, INFINITY, -INFINITY, 0, 0};
  bool bad = false;  // a NaN was seen, which fmax drops
  const size_t zb = nn * (size_t)wrapi(k0 - 1, n), zc = nn * (size_t)k0;
  double um = (double)u[zb + oc] - mu, vm = (double)v[zb + oc] - mv, wm = (double)w[zb + oc] - mw;
  double uc = (double)u[zc + oc] - mu, vc = (double)v[zc + oc] - mv, wc = (double)w[zc + oc] - mw;
  for (int k = k0; k < k0 + kz; ++k) {
    const size_t z = nn * (size_t)k, zp = nn * (size_t)wrapi(k + 1, n);
    const T *up = u + z, *vp = v + z, *wp = w + z;
    const T lu[5] = {up[oxp], up[oxm], up[oyp], up[oym], u[zp + oc]};
    const T lv[5] = {vp[oxp], vp[oxm], vp[oyp], vp[oym], v[zp + oc]};
    const T lw[5] = {wp[oxp], wp[oxm], wp[oyp], wp[oym], w[zp + oc]};
    const T lf = phi ? phi[z + oc] : (T)0;
    const double uxp = (double)lu[0] - mu, uxm = (double)lu[1] - mu, uyp = (double)lu[2] - mu,
                 uym = (double)lu[3] - mu, uzp = (double)lu[4] - mu;
    const double vxp = (double)lv[0] - mv, vxm = (double)lv[1] - mv, vyp = (double)lv[2] - mv,
                 vym = (double)lv[3] - mv, vzp = (double)lv[4] - mv;
    const double wxp = (double)lw[0] - mw, wxm = (double)lw[1] - mw, wyp = (double)lw[2] - mw,
                 wym = (double)lw[3] - mw, wzp = (double)lw[4] - mw;
    s[0] += uc * uc + vc * vc + wc * wc;
    s[6] += uc;
    // compute_diss (post/compute_diss/main.f90:87-111)
    const double dudx = (uxp - uxm) * h, dudy = (uyp - uym) * h, dudz = (uzp - um) * h;
    const double dvdx = (vxp - vxm) * h, dvdy = (vyp - vym) * h, dvdz = (vzp - vm) * h;
    const double dwdx = (wxp - wxm) * h, dwdy = (wyp - wym) * h, dwdz = (wzp - wm) * h;
    const double S12 = 0.5 * (dudy + dvdx), S13 = 0.5 * (dudz + dwdx), S23 = 0.5 * (dvdz + dwdy);
    s[1] += dudx * dudx + dvdy * dvdy + dwdz * dwdz + 2.0 * (S12 * S12 + S13 * S13 + S23 * S23);
    // forward-difference divergence of the projection (multi/main.f90:723-725)
    const double div = ((uxp - uc) + (vyp - vc) + (wzp - wc)) * dxi_c;
    s[2] = fmax(s[2], fabs(div));
    bad |= div != div;
    if (phi) {
      const double f = (double)lf;
      s[3] += f;
      s[4] = fmin(s[4], f);
      s[5] = fmax(s[5], f);
    }
    um = uc; uc = uzp;
    vm = vc; vc = vzp;
    wm = wc; wc = wzp;
  }
  if (bad) s[2] = NAN;
  __shared__ double red[DNT / 32][NSTAT];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    for (int t = 0; t < NSTAT; ++t) {
      const double x = __shfl_xor_sync(0xffffffffu, s[t], o);
      if (t == 2) s[t] = max_nan(s[t], x);
      else if (t == 5) s[t] = fmax(s[t], x);
      else if (t == 4) s[t] = fmin(s[t], x);
      else s[t] += x;
    }
  }
  if ((threadIdx.x & 31) == 0)
    for (int t = 0; t < NSTAT; ++t) red[threadIdx.x >> 5][t] = s[t];
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int wdx = 1; wdx < DNT / 32; ++wdx)
      for (int t = 0; t < NSTAT; ++t) {
        const double x = red[wdx][t];
        if (t == 2) red[0][t] = max_nan(red[0][t], x);
        else if (t == 5) red[0][t] = fmax(red[0][t], x);
        else if (t == 4) red[0][t] = fmin(red[0][t], x);
        else red[0][t] += x;
      }
    const size_t b = (size_t)blockIdx.x + (size_t)gridDim.x * (blockIdx.y + (size_t)gridDim.y * blockIdx.z);
    for (int t = 0; t < NSTAT; ++t) partials[b * NSTAT + t] = red[0][t];
  }
}

__global__ void stats_final_kernel(const double* __restrict__ partials, int nparts, double* __restrict__ out) {
  __shared__ double red[256][NSTAT];
  double s[NSTAT] = {0, 0, 0, 0, INFINITY, -INFINITY, 0, 0};
  for (int b = threadIdx.x; b < nparts; b += 256)
    for (int t = 0; t < NSTAT; ++t) {
      const double x = partials[(size_t)b * NSTAT + t];
      if (t == 2) s[t] = max_nan(s[t], x);
      else if (t == 5) s[t] = fmax(s[t], x);
      else if (t == 4) s[t] = fmin(s[t], x);
      else s[t] += x;
    }
  for (int t = 0; t < NSTAT; ++t) red[threadIdx.x][t] = s[t];
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if ((int)threadIdx.x < st)
      for (int t = 0; t < NSTAT; ++t) {
        const double x = red[threadIdx.x + st][t];
        double& y = red[threadIdx.x][t];
        if (t == 2) y = max_nan(y, x);
        else if (t == 5) y = fmax(y, x);
        else if (t == 4) y = fmin(y, x);
        else y += x;
      }
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int t = 0; t < NSTAT; ++t) out[t] = red[0][t];
}

int stats_partials(int n) { return (n / DTX) * (n / DTY) * (n / stats_planes(n)); }

template <class T>
cudaError_t launch_stats(const T* u, const T* v, const T* w, const T* phi, const Ctrl* ctrl, int n, double dxi_c,
                         double dxi_d, double* partials, double* out, cudaStream_t st) {
  dim3 grid(n / DTX, n / DTY, n / stats_planes(n));
  stats_kernel<T><<<grid, DNT, 0, st>>>(u, v, w, phi, ctrl, n, stats_planes(n), dxi_c, dxi_d, partials);
  stats_final_kernel<<<1, 256, 0, st>>>(partials, stats_partials(n), out);
  return cudaGetLastError();
}

template cudaError_t launch_stats<double>(const double*, const double*, const double*, const double*, const Ctrl*,
                                          int, double, double, double*, double*, cudaStream_t);
template cudaError_t launch_stats<float>(const float*, const float*, const float*, const float*, const Ctrl*, int,
                                         double, double, double*, double*, cudaStream_t);

}  // namespace mhit
