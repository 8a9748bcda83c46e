// Stencil kernels of the MHIT36 step on one B200: the ACDI phase-field update,
// the momentum RHS + AB2 predictor, the unfused projections with the mean/max
// reductions (FP32: and a one-CTA finalize), and the FP32 form's divergence
// check.
//
// Fields are stored without halo cells, x fastest (n^3 values); periodic
// neighbours come from index wrap.  On one rank this is exactly what the
// reference's cuDecomp halo updates (periodic, multi/main.f90:418-429,
// 483-486, 630-641, 685-696, 817-818, 923-934) provide, so none of the 28 halo
// calls of a reference step has a counterpart here.
//
// Both stencil kernels march a TX x TY column tile through a chunk of KZ z
// planes ("2.5D" blocking): each z plane of every input is read from HBM once
// per tile (plus its x/y halo ring, mostly L2 hits), kept in a small ring of
// shared-memory planes, and every intermediate the reference materialises in
// HBM (psidi, normx/y/z, rhsphi, rhsu/v/w, chempot, gradphi*, f*st) lives
// only in shared memory or registers.
#include <cuda.h>
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>
#include "common.cuh"
#include "finish.cuh"
#include "internal.h"

namespace mhit {

constexpr int TX = 32, TY = 8, NT = TX * TY;

// Default number of z chunks of a stencil kernel with `tiles` column tiles and
// `slots` CTAs resident on the GPU.  Large grids: chunks of 32 planes, 64 from
// 512^3 up (2-3% faster than 32 there; a chunk recomputes a few planes to
// fill its rings).  A grid with less than two waves of such CTAs (up to 192^3,
// and the FP32 phase kernel at 256^3, 182 us in 9 chunks against 190 in 8) is
// split into the number of chunks, from n/32 up, with the least waves * (longest
// chunk + lead), lead being the planes a chunk recomputes.  Chunks need not
// divide n evenly.  The cost takes an iteration's time as the same however many
// CTAs share an SM, which holds roughly only (FP64 phase: 2.4 us with one CTA
// per SM at 32^3, 4.4 with three at 128^3).
// B200, FP64 step against chunks of 32 planes everywhere (with project_kz):
// 32^3 NS 108 -> 72 us a call, 64^3 182 -> 62 us a step, 128^3 277 -> 214,
// 192^3 664 -> 627; chunks of 2 or 4 planes cost 128^3 30% and 256^3 30-80%.
static int pick_chunks(int n, int tiles, int slots, int lead) {
  const int nz = n / (n >= 512 ? 64 : 32);
  if ((long long)tiles * nz >= 2LL * slots) return nz;
  int best = nz;
  long long cost = -1;
  for (int q = nz; q <= n / 2; ++q) {
    const long long waves = ((long long)tiles * q + slots - 1) / slots;
    const long long c = waves * ((n + q - 1) / q + lead);
    if (cost < 0 || c < cost) {
      cost = c;
      best = q;
    }
  }
  return best;
}
// SMs of the current device.
static int sm_count() {
  int dev = 0, v = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v < 1)
    return 148;
  return v;
}

// Momentum tile height.  Both tiles run 256 threads; the 16-row tile gives
// each thread two rows.  Measured on B200 at 512^3: FP64 8 rows 3.06 ms,
// 16 rows 4.18 ms (128 registers); FP32 8 rows 2.00 ms, 16 rows 1.87 ms.
int default_mty(int n, int fp32) { return (n >= 16 && fp32) ? 16 : 8; }

// ============================================================ psi arithmetic
// psi = eps*log(a/b) (A3) is the phase kernel's most expensive expression.
// FP64: a/b by Newton-Raphson from the PTX reciprocal approximation
// (rcp.approx.ftz.f64, two iterations and a remainder correction: the
// correctly rounded quotient for these operands, which are normal numbers
// in [1e-16, 1 + 1e-16]), and the logarithm by P. T. P. Tang's table-driven
// method ("Table-driven implementation of the logarithm function in IEEE
// floating-point arithmetic", ACM TOMS 16(4), 1990): x = 2^k m, m in
// [1, 2), F = 1 + j/128 nearest to m, r = (m - F)/F with |r| <= 2^-8, and
// log x = k ln2 + log F + log(1 + r), the last by its Taylor series to r^7
// (truncation below 2^-59 relative).  log F and ln2 are double-double
// values computed on the host in long double.  Both are branch-free, so the
// psi of a thread's elements overlap.  Measured against CUDA's log and
// division on B200 over 134M phase-field values: at most 2 ulp apart, and
// 1.45x faster.  FP32: the hardware approximations __fdividef and __logf
// (about 1 ulp of psi on these operands).
constexpr int LOGTAB = 3 * 129 + 2;  // 1/F, log F (hi), log F (lo), then ln2 (hi, lo)
__device__ double g_log_table[LOGTAB];

__device__ __forceinline__ double div_nr(double a, double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  double e = fma(-b, y, 1.0);
  y = fma(y, e, y);
  e = fma(-b, y, 1.0);
  y = fma(y, e, y);
  const double q = a * y;
  return fma(fma(-b, q, a), y, q);
}

// log x for positive normal x; tab = g_log_table (in shared memory).  The
// integers k and j become doubles by their bit patterns (2^52 + k, and F
// itself) instead of conversion instructions.
__device__ __forceinline__ double tang_log(double x, const double* __restrict__ tab) {
  const int hi = __double2hiint(x), lo = __double2loint(x);
  const int mant = hi & 0x000fffff;
  const int j = (mant + (1 << 12)) >> 13;  // nearest j/128, 0..128
  const double m = __hiloint2double(mant | 0x3ff00000, lo);
  const double F = __hiloint2double(0x3ff00000 + (j << 13), 0);
  const double kd = __hiloint2double(0x43300000, hi >> 20) - (4503599627370496.0 + 1023.0);
  const double r = (m - F) * tab[j];  // m - F is exact
  double p = fma(r, 1.0 / 7, -1.0 / 6);
  p = fma(p, r, 0.2);
  p = fma(p, r, -0.25);
  p = fma(p, r, 1.0 / 3);
  p = fma(p, r, -0.5);
  p = fma(p, r * r, r);
  return fma(kd, tab[3 * 129], tab[129 + j]) + (fma(kd, tab[3 * 129 + 1], tab[2 * 129 + j]) + p);
}

template <class T> struct PsiMath;
template <> struct PsiMath<double> {
  static constexpr int TAB = LOGTAB;  // table entries staged in shared memory
  static __device__ __forceinline__ double log_ratio(double a, double b, const double* tab) {
    return tang_log(div_nr(a, b), tab);
  }
};
template <> struct PsiMath<float> {
  static constexpr int TAB = 0;
  static __device__ __forceinline__ float log_ratio(float a, float b, const double*) { return __logf(__fdividef(a, b)); }
};

// The table of tang_log, once per device (before any graph capture).
static cudaError_t upload_log_table() {
  static bool done[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e) return e;
  if (dev >= 0 && dev < 64 && done[dev]) return cudaSuccess;
  double t[LOGTAB];
  for (int j = 0; j <= 128; ++j) {
    const long double F = 1.0L + (long double)j / 128.0L;
    const long double l = logl(F);
    t[j] = (double)(1.0L / F);
    t[129 + j] = (double)l;
    t[2 * 129 + j] = (double)(l - (long double)t[129 + j]);
  }
  const long double ln2 = logl(2.0L);
  t[3 * 129] = (double)ln2;
  t[3 * 129 + 1] = (double)(ln2 - (long double)t[3 * 129]);
  if ((e = cudaMemcpyToSymbol(g_log_table, t, sizeof(t)))) return e;
  if (dev >= 0 && dev < 64) done[dev] = true;
  return cudaSuccess;
}

// ============================================================ phase field
// ACDI step A1..A7 (multi/main.f90:341-480) fused into one kernel:
//   psi = eps*log((min(phi,1)+enum)/(1-min(phi,1)+enum))      (A3)
//   n   = grad(psi) / (|grad(psi)| + 1e-16f)                  (A4, A5)
//   F   = 0.25*(1 - tanh(psi/(2 eps))^2) * n                  (A6 flux)
//   rhs = -div(u phi_face) + gamma*eps*lap(phi) - gamma*div_c(F)   (A1, A2, A6)
//   phi_new = phi + dt*rhs                                    (A7)
// psi needs phi on a radius-2 neighbourhood; it is computed per plane on the
// tile plus a 2-cell ring, F on the tile plus a 1-cell ring.
// Tile 32 x 16 with two output rows per thread (rows ty and ty + 8, 256
// threads): the per-plane barriers, ring bookkeeping and copy issue are
// shared by two points, and the psi / F loops run three rounds per thread
// (B200, 512^3 FP64: 2.61 -> 2.36 ms against one row per thread).
constexpr int PTY = 16;            // phase tile height
constexpr int PPT = 2;             // output rows per thread (rows ty + h*PTY/PPT)
constexpr int PNT = TX * PTY / PPT;  // phase threads per CTA
// Resident CTAs per SM the phase kernel is built for: 3 in FP64 (80 registers),
// 4 in FP32 (64 registers; 512^3: 1.57 -> 1.37 ms against 2).
template <class T> __host__ __device__ constexpr int phase_min_blocks() { return sizeof(T) == 4 ? 4 : 3; }

// Momentum ring depth (planes per field): planes m-2 .. m+1, one in flight.
// (A 5-plane ring with two planes in flight measured 30% slower on B200 at
// 512^3: it leaves fewer CTAs per SM.)
__host__ __device__ constexpr int momentum_ring(int) { return 4; }
// Resident CTAs per SM the momentum kernel is built for: what its shared
// memory allows with ACDI (3 with 8-row tiles), 4 without; registers follow.
// FP32 16-row tiles: 3 (80 registers, no spill; 1.73 -> 1.62 ms at 512^3 on
// B200 against 2), FP64 16-row tiles 2 (128 registers).
template <class T> __host__ __device__ constexpr int momentum_min_blocks(bool pf, int mty) {
  return mty == 8 ? (pf ? 3 : 4) : (sizeof(T) == 4 ? 3 : 2);
}

// Staged-plane geometry of the momentum kernel.  A staged plane is a box of
// cells whose first column lies XS cells left of the tile, XS cells being 16
// bytes, so that a tensor-map box load starts on a 16-byte boundary: UX x UY
// cells for the velocities (the tile and its 1-cell ring), EX x EY for phi
// (2-cell ring), widths rounded up to 16 bytes.  Ring slots are 128-byte
// multiples; the slot barriers follow the force ring.
template <class T, int TYv> struct MomGeo {
  static constexpr int XS = 16 / (int)sizeof(T);
  static constexpr int AL = 128 / (int)sizeof(T);
  static constexpr int UX = (XS + TX + 1 + XS - 1) / XS * XS, UY = TYv + 2, UE = UX * UY;
  static constexpr int EX = (XS + TX + 2 + XS - 1) / XS * XS, EY = TYv + 4, PE = EX * EY;
  static constexpr int USL = (UE + AL - 1) / AL * AL, PSL = (PE + AL - 1) / AL * AL;
  static constexpr int QE = (TX + 1) * (TYv + 1);
  static __host__ __device__ constexpr size_t bar_offset(bool pf, int ns) {
    return ((sizeof(T) * (3 * ns * USL + (pf ? ns * PSL + 6 * QE : 0))) + 7) / 8 * 8;
  }
  static __host__ __device__ constexpr unsigned tx_bytes(bool pf) {
    return (unsigned)(sizeof(T) * (3 * UE + (pf ? PE : 0)));
  }
  // every box of the tile inside the n x n plane
  static __host__ __device__ bool interior(int x0, int y0, int n, bool pf) {
    const int bw = UX > EX ? UX : EX, r = pf ? 2 : 1;
    return x0 >= XS && x0 - XS + bw <= n && y0 >= r && y0 + TYv + r <= n;
  }
};
static_assert(MomGeo<double, 8>::UX == 36 && MomGeo<double, 8>::EX == 36, "FP64 staged box widths");
static_assert(MomGeo<float, 16>::UX == 40 && MomGeo<float, 16>::EX == 40, "FP32 staged box widths");

// Staged planes of the phase kernel: phi on the tile and its 2-cell ring in a
// box starting XS cells (16 bytes) left of the tile, row pitch EX, and u, v,
// w on the cells the face fluxes need (u one more to the right, v one more
// above).  Every staged array is a multiple of 128 bytes.
template <class T> struct PhaseGeo {
  static constexpr int XS = 16 / (int)sizeof(T);
  static constexpr int AL = 128 / (int)sizeof(T);
  static constexpr int EX = (XS + TX + 2 + XS - 1) / XS * XS, EY = PTY + 4;
  static constexpr int PSL = (EX * EY + AL - 1) / AL * AL;
  static constexpr int UW = (TX + 1 + XS - 1) / XS * XS;
  static constexpr int UE = UW * PTY, VE = TX * (PTY + 1), WE = TX * PTY;
  static constexpr int VOFF = (UE + AL - 1) / AL * AL, WOFF = VOFF + (VE + AL - 1) / AL * AL;
  static constexpr int VSL = WOFF + (WE + AL - 1) / AL * AL;
  static constexpr int FXE = PTY * (TX + 2), FYE = (PTY + 2) * TX;
  static __host__ __device__ constexpr unsigned phi_bytes() { return (unsigned)(sizeof(T) * EX * EY); }
  static __host__ __device__ constexpr unsigned vel_bytes() { return (unsigned)(sizeof(T) * (UE + VE + WE)); }
  static __host__ __device__ constexpr size_t smem(int tab) {
    return sizeof(T) * (size_t)(6 * PSL + FXE + FYE + 2 * VSL) + sizeof(double) * (tab + 3);
  }
  // the phi box of the tile inside the n x n plane
  static __host__ __device__ bool interior(int x0, int y0, int n) {
    return x0 >= XS && x0 - XS + EX <= n && y0 >= 2 && y0 + PTY + 2 <= n;
  }
};
static_assert(PhaseGeo<double>::EX == 36 && PhaseGeo<float>::EX == 40, "staged phi box widths");
static_assert(PhaseGeo<double>::FXE % 16 == 0 && PhaseGeo<double>::FYE % 16 == 0, "128-byte aligned stages");
static_assert(PhaseGeo<float>::FXE % 32 == 0 && PhaseGeo<float>::FYE % 32 == 0, "128-byte aligned stages");

// 1/(sqrt(s) + tiny) for s > 0, the normalisation of A5.  With r = rsqrt(s),
// 1/(sqrt(s) + tiny) = r/(1 + tiny*r) = r - tiny*r^2 + r*O((tiny*r)^2); the
// first-order form is used while tiny*r < 2^-30, where the dropped term is
// below 2^-60 r (far under an ulp), and the direct formula otherwise.
template <class T>
__device__ __forceinline__ T inv_norm_plus(T s, T tiny) {
  const T r = rsqrt(s);
  const T tr = tiny * r;
  if (tr < (T)9.3e-10) return fma(-tr, r, r);
  return (T)1 / (sqrt(s) + tiny);
}

// One tile and z chunk of the phase-field update.
//
// Schedule at iteration m (stage m has landed: phi plane m, u and v of plane
// m-1, w of plane m): psi(m) | barrier | F(m-1) | barrier | phi_new(m-2) and
// the x, y part of plane m-1.  A thread owns its column (tx, ty + 8h): the z
// neighbours of phi, F_z and w pass from plane to plane in registers, and
// only F_x and F_y of the current plane go through shared memory.
// The rings are 3 phi and 3 psi planes, one plane of F_x and F_y and two
// velocity stages, 72 KB in FP64 with 78 registers: three CTAs per SM, where
// the kernel was bound by latency at two (93 KB with 5 + 3 + 9 planes, 114
// registers with the velocities prefetched into them).
//
// u, v and w arrive by tensor-map box loads on every tile; where the face
// right of or above the tile wraps, its few values are read directly.  phi
// arrives by a box load on the tiles whose box lies inside the grid
// (tma_phi); on the others each thread copies the ring cells it computes psi
// for with cp.async and periodic wrap.  Both fill the same shared cells.
//
// FP32 runs the loop over planes unrolled over the three ring slots, whose
// addresses are then constants.  FP64 does not: its psi and F are four times
// the instructions, and three copies of them stalled on instruction fetch
// (5.2 of 12 cycles per issue).
//
// B200 against the kernel before (two CTAs per SM, velocities in registers, F
// in nine shared planes): FP64 192^3 167 -> 147 us, 256^3 339 -> 307, 384^3 882
// -> 755, 512^3 2260 -> 1920; FP32 512^3 1346 -> 1149; 96^3 and below unchanged.
template <class T, bool SLOT>
__device__ __forceinline__ void phase_body(const StencilArgs<T>& a, const T* __restrict__ phi_in,
                                           T* __restrict__ phi_out, int nz, int bx, int by, int bz,
                                           const PhaseMaps* __restrict__ maps) {
  constexpr int TY = PTY, NT = PNT;
  typedef PhaseGeo<T> G;
  constexpr int LX = TX + 4, PE = LX * G::EY, EX = G::EX, OFF = G::XS - 2, SL = G::PSL;
  constexpr int FXP = TX + 2;  // row pitch of F_x (x = -1 .. TX)
  extern __shared__ __align__(128) unsigned char smem_raw[];
  T* const s_phi = reinterpret_cast<T*>(smem_raw);
  T* const s_psi = s_phi + 3 * SL;
  T* const s_fx = s_psi + 3 * SL;
  T* const s_fy = s_fx + G::FXE;
  T* const s_vel = s_fy + G::FYE;  // two stages of u, v, w
  double* const s_tab = reinterpret_cast<double*>(s_vel + 2 * G::VSL);
  unsigned long long* const s_bar = reinterpret_cast<unsigned long long*>(s_tab + PsiMath<T>::TAB);
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int n = a.c.n;
  // z chunk bz of nz
  const int x0 = bx * TX, y0 = by * TY, k0 = bz * n / nz, KZ = (bz + 1) * n / nz - k0;
  const bool tma_phi = G::interior(x0, y0, n);
  for (int q = tid; q < PsiMath<T>::TAB; q += NT) s_tab[q] = g_log_table[q];
  if (tid == 0) {
#pragma unroll
    for (int q = 0; q < 3; ++q) mbar_init(s_bar + q, 1);
    mbar_init_fence();
    if (SLOT) {  // maps in the ensemble's slot table
      tensormap_acquire(&maps->phi);
      tensormap_acquire(&maps->u);
      tensormap_acquire(&maps->v);
      tensormap_acquire(&maps->w);
    }
  }
  if (stopped(a.ctrl)) return;  // also publishes the barriers and the table
  const T eps = (T)a.c.eps, enumv = (T)a.c.enumv, tiny = (T)a.c.tiny;
  const T dt = (T)a.c.dt, hdxi = (T)(0.5 * a.c.dxi);
  const double gamma = 1.0 * a.ctrl->gumax;  // multi/main.f90:362
  const T gh = (T)(gamma * (0.5 * a.c.dxi)), ge = (T)(gamma * (a.c.eps * a.c.ddxi));
  const T mu = (T)a.ctrl->mean[0], mv = (T)a.ctrl->mean[1], mw = (T)a.ctrl->mean[2];
  const bool floored = a.c.phi_floor;
  const T floor0 = floored ? (T)0 : (T)-INFINITY;
  const T inv12e = (T)1 / ((T)1 + (T)2 * enumv);
  // psi where min(phi,1) is exactly 1 (drop interiors) or so small that both
  // val + enum == enum and 1 - val + enum == 1 - 0 + enum in floating point
  // (far field; the first implies the second, since it needs |val| below
  // half an ulp of enum, far under 2^-54): there the reference's expression
  // evaluates to psi1 / psi0 exactly, so those constants are computed once
  // and the log is skipped -- bitwise the same values.  With the floor every
  // negative phi is of the second kind.  Without it a phi at or below -enum has
  // the logarithm of 0 (-inf) or of a negative number (NaN), which tang_log, for
  // positive numbers only, does not give (FP32's __logf does).
  const T psi0 = eps * PsiMath<T>::log_ratio((T)0 + enumv, (T)1 - (T)0 + enumv, s_tab);
  const T psi1 = eps * PsiMath<T>::log_ratio((T)1 + enumv, (T)1 - (T)1 + enumv, s_tab);
  const size_t nn = (size_t)n * n;
  // Each thread owns ring elements tid + r*NT of every plane (copy and psi);
  // pidx(r) is the stored index (row pitch EX, first column OFF).
  constexpr int NPE = (PE + NT - 1) / NT;
  const auto pidx = [&](int r) {
    const int e = tid + r * NT;
    if constexpr (EX == LX && OFF == 0) return e;
    else return (e % LX + OFF) + (e / LX) * EX;
  };
  // Ring cells of F: F_x left and right of the tile, F_y below and above it,
  // one each for threads 0 .. NRING-1.
  constexpr int NRING = 2 * TY + 2 * TX;
  const bool rx = tid < 2 * TY;
  int rpe, rfe;  // plane index and F_x / F_y index of the thread's ring cell
  {
    const int q = rx ? tid : tid - 2 * TY;
    const int ex = rx ? (q < TY ? -1 : TX) : q % TX, ey = rx ? q % TY : (q < TX ? -1 : TY);
    rpe = (ex + 2 + OFF) + (ey + 2) * EX;
    rfe = rx ? (ex + 1) + ey * FXP : ex + (ey + 1) * TX;
  }
  constexpr int RY = TY / PPT;
  const int pe0 = (tx + 2 + OFF) + (ty + 2) * EX;  // own cell, row h: + h*RY*EX
  const int fx0 = (tx + 1) + ty * FXP, fy0 = tx + (ty + 1) * TX;
  const unsigned ij = (unsigned)(x0 + tx) + (unsigned)n * (unsigned)(y0 + ty);
  const bool wrap_x = x0 + tx + 1 == n;

  // Stage j (m = k0 - 2 + j) into ring slot S: phi plane m; for 2 <= j <= KZ+2
  // also u, v of plane m-1 and w of plane m into velocity stage j & 1.
  auto issue = [&](int S, int j) {
    const int m0 = wrapi(k0 - 2 + j, n), m1 = wrapi(k0 - 3 + j, n);
    T* const dp = s_phi + S * SL;
    const bool vel = j >= 2 && j <= KZ + 2;
    if (tid == 0 && (tma_phi || vel)) {
      unsigned long long* const bar = s_bar + S;
      mbar_arrive_expect_tx(bar, (tma_phi ? G::phi_bytes() : 0u) + (vel ? G::vel_bytes() : 0u));
      if (tma_phi) tma_load_2d(dp, &maps->phi, x0 - G::XS, m0 * n + y0 - 2, bar);
      if (vel) {
        T* const dv = s_vel + (j & 1) * G::VSL;
        tma_load_2d(dv, &maps->u, x0, m1 * n + y0, bar);
        tma_load_2d(dv + G::VOFF, &maps->v, x0, m1 * n + y0, bar);
        tma_load_2d(dv + G::WOFF, &maps->w, x0, m0 * n + y0, bar);
      }
    }
    if (!tma_phi) {
      const T* const src = phi_in + nn * m0;
#pragma unroll
      for (int r = 0; r < NPE; ++r) {
        const int e = tid + r * NT;
        if (r < NPE - 1 || e < PE)
          cp_async_elem(dp + pidx(r), src + (unsigned)(wrapi(x0 - 2 + e % LX, n) + n * wrapi(y0 - 2 + e / LX, n)));
      }
      cp_async_commit();
    }
  };
  // carried per own row: phi, F_z and w of the previous plane, and the part
  // of the update that does not need F_z of the plane above
  T c_[PPT], fz_[PPT], wc_[PPT], s_[PPT];
#pragma unroll
  for (int h = 0; h < PPT; ++h) c_[h] = fz_[h] = wc_[h] = s_[h] = (T)0;
  unsigned bar_phase = 0;  // bit s: parity of the next phase of slot s's barrier

  auto iter = [&](const int S, const int j) __attribute__((always_inline)) {
    const int Sm1 = S == 0 ? 2 : S - 1, Sm2 = S == 2 ? 0 : S + 1;  // slots of planes m-1, m-2
    // plane m has landed: the slot's barrier phase for the box loads (a wait
    // that gives up records a timeout and carries on, so that no thread is
    // left at a barrier), or this thread's cp.async copies
    if (tma_phi || (j >= 2 && j <= KZ + 2)) {
      if (!mbar_wait(s_bar + S, (bar_phase >> S) & 1u, kWaitCycles)) atomicCAS(&a.ctrl->status, 0, kStatusTimeout);
      bar_phase ^= 1u << S;
    }
    if (!tma_phi) cp_async_wait<0>();
    const T *const Ph0 = s_phi + S * SL, *const Phm1 = s_phi + Sm1 * SL;
    T* const Ps0 = s_psi + S * SL;
    const T *const Psm1 = s_psi + Sm1 * SL, *const Psm2 = s_psi + Sm2 * SL;
    // (1) psi of plane m on the elements this thread copied
#pragma unroll
    for (int r = 0; r < NPE; ++r) {
      if (r < NPE - 1 || tid + r * NT < PE) {
        const int ep = pidx(r);
        const T val = fmin(Ph0[ep], (T)1), sum = val + enumv;
        T psi;
        if (sum <= enumv && (floored || sum == enumv)) {
          psi = psi0;
        } else if (val < (T)1) {
          psi = eps * PsiMath<T>::log_ratio(sum, (T)1 - val + enumv, s_tab);
          if (sizeof(T) == 8 && !floored && sum <= (T)0) psi = sum < (T)0 ? (T)NAN : -(T)INFINITY;
        } else {
          psi = psi1;
        }
        Ps0[ep] = psi;
      }
    }
    // psi(m) is visible and every thread is done with iteration m-1, so the
    // phi slot of plane m-2 and the velocity stage that stage j+1 refills are free
    __syncthreads();
    if (j < KZ + 3) issue(Sm2, j + 1);
    // (2) F on plane m-1: own cells (F_z stays in registers), then one ring cell
    T fzc[PPT];
#pragma unroll
    for (int h = 0; h < PPT; ++h) fzc[h] = (T)0;
    if (j >= 2) {
#pragma unroll
      for (int r = 0; r <= PPT; ++r) {
        if (r == PPT && tid >= NRING) break;
        const int pe = r < PPT ? pe0 + r * RY * EX : rpe;
        const T gxv = Psm1[pe + 1] - Psm1[pe - 1];
        const T gyv = Psm1[pe + EX] - Psm1[pe - EX];
        const T gzv = Ps0[pe] - Psm2[pe];
        T fx = (T)0, fy = (T)0, fz = (T)0;
        if (gxv != (T)0 || gyv != (T)0 || gzv != (T)0) {  // uniform psi: n = 0 and F = 0 exactly
          const T normod = inv_norm_plus(fma(gzv, gzv, fma(gyv, gyv, gxv * gxv)), tiny);
          T t;
          if (a.c.tanh_identity) {
            // tanh(0.5*log(a/b)) = (a-b)/(a+b) with a = val+enum, b = 1-val+enum
            const T val = fmax(fmin(Phm1[pe], (T)1), floor0);
            t = ((T)2 * val - (T)1) * inv12e;
          } else {
            t = tanh((T)0.5 * Psm1[pe] * (T)a.c.epsi);
          }
          const T g = (T)0.25 * ((T)1 - t * t);
          fx = g * (gxv * normod);
          fy = g * (gyv * normod);
          fz = g * (gzv * normod);
        }
        if (r < PPT) {
          s_fx[fx0 + r * RY * FXP] = fx;
          s_fy[fy0 + r * RY * TX] = fy;
          fzc[r < PPT ? r : 0] = fz;
        } else if (rx) {
          s_fx[rfe] = fx;
        } else {
          s_fy[rfe] = fy;
        }
      }
    }
    __syncthreads();
    if (j >= 2) {
      // (3) phi_new of plane m-2, then the x, y part of plane m-1
      const T* const V = s_vel + (j & 1) * G::VSL;
      const int k = k0 - 3 + j;  // plane m-1
      if (j >= 4) {
        T* const out = phi_out + nn * (k - 1);
#pragma unroll
        for (int h = 0; h < PPT; ++h) out[ij + (unsigned)(h * RY * n)] = fma(dt, fma(-gh, fzc[h], s_[h]), c_[h]);
      }
#pragma unroll
      for (int h = 0; h < PPT; ++h) {
        const int pe = pe0 + h * RY * EX, row = ty + h * RY;
        const T c = Phm1[pe];
        if (j <= KZ + 2) {
          const T wzp = V[G::WOFF + tx + row * TX] - mw;
          if (j >= 3) {
            T uxp = V[tx + 1 + row * G::UW], vyp = V[G::VOFF + tx + (row + 1) * TX];
            if (wrap_x) uxp = a.u[nn * k + (unsigned)n * (unsigned)(y0 + row)];
            if (y0 + row + 1 == n) vyp = a.v[nn * k + (unsigned)(x0 + tx)];
            uxp -= mu;
            vyp -= mv;
            const T uc = V[tx + row * G::UW] - mu, vc = V[G::VOFF + tx + row * TX] - mv;
            const T pxp = Phm1[pe + 1], pxm = Phm1[pe - 1], pyp = Phm1[pe + EX], pym = Phm1[pe - EX];
            const T pzp = Ph0[pe], pzm = c_[h];
            const int fx = fx0 + h * RY * FXP, fy = fy0 + h * RY * TX;
            // The factors 0.5 of the face averages and central differences
            // are folded into hdxi = 0.5*dxi and gh = gamma*hdxi.  The fused
            // multiply-adds are written out, so that every instantiation (a
            // slot of the ensemble among them) rounds alike.
            T conv = uxp * (pxp + c);
            conv = fma(-uc, c + pxm, conv);
            conv = fma(vyp, pyp + c, conv);
            conv = fma(-vc, c + pym, conv);
            conv = fma(wzp, pzp + c, conv);
            conv = fma(-wc_[h], c + pzm, conv);
            const T lap = (pxp - (T)2 * c + pxm) + (pyp - (T)2 * c + pym) + (pzp - (T)2 * c + pzm);
            const T div = (s_fx[fx + 1] - s_fx[fx - 1]) + (s_fy[fy + TX] - s_fy[fy - TX]) - fz_[h];
            s_[h] = fma(-gh, div, fma(-hdxi, conv, ge * lap));
          }
          wc_[h] = wzp;
        }
        c_[h] = c;
        fz_[h] = fzc[h];
      }
    }
  };
  issue(0, 0);
  if constexpr (sizeof(T) == 4) {
#pragma unroll 1
    for (int j = 0; j <= KZ + 3; j += 3) {
      iter(0, j);
      if (j + 1 > KZ + 3) break;
      iter(1, j + 1);
      if (j + 2 > KZ + 3) break;
      iter(2, j + 2);
    }
  } else {
    int S = 0;
#pragma unroll 1
    for (int j = 0; j <= KZ + 3; ++j) {
      iter(S, j);
      S = S == 2 ? 0 : S + 1;
    }
  }
}

// ============================================================ momentum
// B1..B7 (multi/main.f90:513-682) fused: conservative convection, viscous
// term, ABC forcing, optional linear forcing A*u, surface tension
// f = 6 sigma chempot grad(phi) at cell centres interpolated to the faces,
// and the AB2 (Euler on the first step) predictor.  Writes ustar and the new
// rhs_o; reads the NEW phi (the reference computes B4 after A7).
// momentum tile height: 8 or 16 rows (a tuning choice per grid size)
template <class T, bool PF, int MTYv, bool TMA>
__device__ __forceinline__ void momentum_body(const StencilArgs<T>& a, int nz, int bx, int by, int bz,
                                              const PlaneMaps* __restrict__ maps, bool gmaps) {
  // MPT output rows per thread (rows ty + 8h): 256 threads for either tile
  constexpr int TY = MTYv, MPT = MTYv / 8, NT = TX * 8;
  typedef MomGeo<T, MTYv> G;
  constexpr int XS = G::XS, UX = G::UX, UE = G::UE, EX = G::EX, PE = G::PE;
  constexpr int QX = TX + 1, QY = TY + 1, QE = QX * QY;  // force over [-1,TX) x [-1,TY)
  // Ring of NS planes per field: planes m-2 .. m+PD at iteration m, the
  // last PD of them in flight.
  constexpr int NS = momentum_ring(MTYv), PD = NS - 3;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  T* s_u = reinterpret_cast<T*>(smem_raw);
  T* s_v = s_u + NS * G::USL;
  T* s_w = s_v + NS * G::USL;
  T* s_phi = s_w + NS * G::USL;  // PF only
  T* s_f = s_phi + NS * G::PSL;  // ring of 2 planes x 3 components (PF only)
  unsigned long long* s_bar = reinterpret_cast<unsigned long long*>(smem_raw + G::bar_offset(PF, NS));
  const int n = a.c.n;
  // The kernel is bound by issue, so each term's constant factors are multiplied
  // once and a product that two terms share is formed once (B200: FP32 512^3
  // 1608 -> 1557 us, 384^3 700 -> 677, 256^3 238 -> 234; FP64 512^3 2690 -> 2679,
  // 64^3 18 -> 17).  Differences of products are still formed before they are
  // summed, and the update of u still rounds once at the size of u: errors
  // against FP64 and the oracle are those of the term-by-term form.  The
  // factors: 0.25*dxi (convection), mu*rhoi*ddxi (viscous), eps*ddxi and
  // 6 sigma * 0.5*dxi * 0.5*rhoi (force: central difference and face average),
  // dt*alpha and dt*beta (AB2).
  const T cq = (T)(0.25 * a.c.dxi), cv = (T)(a.c.mu * a.c.rhoi * a.c.ddxi);
  const T epsi = (T)a.c.epsi, ed = (T)(a.c.eps * a.c.ddxi);
  const T cf = (T)(6.0 * a.c.sigma * (0.5 * a.c.dxi) * (0.5 * a.c.rhoi)), lin = (T)a.c.lin_force;
  const T f1 = (T)a.c.f1, f2 = (T)a.c.f2, f3 = (T)a.c.f3;
  const T dta = (T)(a.c.dt * a.ctrl->alpha), dtb = (T)(a.c.dt * a.ctrl->beta);
  const T mu = (T)a.ctrl->mean[0], mv = (T)a.ctrl->mean[1], mw = (T)a.ctrl->mean[2];
  // z chunk bz of nz
  const int x0 = bx * TX, y0 = by * TY, k0 = bz * n / nz, KZ = (bz + 1) * n / nz - k0;
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int i = x0 + tx;
  const size_t nn = (size_t)n * n;
  // Tiles whose staged boxes lie inside the grid (no periodic wrap) load
  // each plane with four tensor-map box loads issued by one thread; the
  // edge tiles copy the same boxes element-wise with cp.async and wrap.
  const bool tma = TMA && G::interior(x0, y0, n, PF);
  // Each thread owns elements tid + r*NT of the velocity, phi and force
  // planes; their in-plane offsets are the same on every plane.
  constexpr int NUE = (UE + NT - 1) / NT, NPE = (PE + NT - 1) / NT, NQE = (QE + NT - 1) / NT;
  int uoff[NUE], poff[NPE], qpe[NQE];
#pragma unroll
  for (int r = 0; r < NUE; ++r) {
    const int e = min(tid + r * NT, UE - 1);
    uoff[r] = wrapi(x0 - XS + e % UX, n) + n * wrapi(y0 - 1 + e / UX, n);
  }
#pragma unroll
  for (int r = 0; r < NPE; ++r) {
    const int e = min(tid + r * NT, PE - 1);
    poff[r] = PF ? wrapi(x0 - XS + e % EX, n) + n * wrapi(y0 - 2 + e / EX, n) : 0;
  }
#pragma unroll
  for (int r = 0; r < NQE; ++r) {
    const int e = min(tid + r * NT, QE - 1);
    qpe[r] = (e % QX + 1) + (e / QX + 1) * EX;
  }
  // sl[q] is the ring slot of plane m-2+q at iteration m; the roles rotate
  // once per plane.
  int sl[NS];
#pragma unroll
  for (int q2 = 0; q2 < NS; ++q2) sl[q2] = q2;
  unsigned bar_phase = 0;  // bit s: parity of the next phase of slot s's barrier
  if (tma && tid == 0) {
#pragma unroll
    for (int q2 = 0; q2 < NS; ++q2) mbar_init(s_bar + q2, 1);
    mbar_init_fence();
    if (gmaps) {  // maps in the ensemble's slot table
      tensormap_acquire(&maps->u);
      tensormap_acquire(&maps->v);
      tensormap_acquire(&maps->w);
      if (PF) tensormap_acquire(&maps->phi);
    }
  }
  if (stopped(a.ctrl)) return;  // also publishes the barriers

  // Plane m of u, v, w (1-cell ring) and phi (2-cell ring) is copied into a
  // ring slot PD iterations ahead of its use, so the HBM latency of the
  // planes in flight overlaps the arithmetic of plane m-1.
  auto issue = [&](int slot, int m) {
    if (tma) {
      if (tid == 0) {
        const int yr = wrapi(m, n) * n;
        mbar_arrive_expect_tx(s_bar + slot, G::tx_bytes(PF));
        tma_load_2d(s_u + slot * G::USL, &maps->u, x0 - XS, yr + y0 - 1, s_bar + slot);
        tma_load_2d(s_v + slot * G::USL, &maps->v, x0 - XS, yr + y0 - 1, s_bar + slot);
        tma_load_2d(s_w + slot * G::USL, &maps->w, x0 - XS, yr + y0 - 1, s_bar + slot);
        if (PF) tma_load_2d(s_phi + slot * G::PSL, &maps->phi, x0 - XS, yr + y0 - 2, s_bar + slot);
      }
      return;
    }
    const size_t zoff = (size_t)wrapi(m, n) * nn;
    const T* su = a.u + zoff;
    const T* sv = a.v + zoff;
    const T* sw = a.w + zoff;
#pragma unroll
    for (int r = 0; r < NUE; ++r) {
      const int e = tid + r * NT;
      if (r < NUE - 1 || e < UE) {
        cp_async_elem(s_u + slot * G::USL + e, su + uoff[r]);
        cp_async_elem(s_v + slot * G::USL + e, sv + uoff[r]);
        cp_async_elem(s_w + slot * G::USL + e, sw + uoff[r]);
      }
    }
    if (PF) {
      const T* sp = a.phi_in + zoff;
#pragma unroll
      for (int r = 0; r < NPE; ++r) {
        const int e = tid + r * NT;
        if (r < NPE - 1 || e < PE) cp_async_elem(s_phi + slot * G::PSL + e, sp + poff[r]);
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int q2 = 0; q2 < PD; ++q2) issue(sl[2 + q2], k0 - 2 + q2);
  // registers carried from one output plane to the next (see below)
  T r_uc[MPT], r_uzp[MPT], r_uxp[MPT], r_vc[MPT], r_vzp[MPT], r_vyp[MPT], r_wc[MPT], r_wzp[MPT], r_wxmzp[MPT],
      r_wymzp[MPT];
  bool have_prev = false;
  for (int m = k0 - 2; m <= k0 + KZ; ++m) {
    // plane m has landed: this thread's cp.async copies, or the slot's
    // barrier phase for the box loads (a wait that gives up records a
    // timeout and carries on, so that no thread is left at a barrier)
    if (tma) {
      const int s = sl[2];
      if (!mbar_wait(s_bar + s, (bar_phase >> s) & 1u, kWaitCycles)) atomicCAS(&a.ctrl->status, 0, kStatusTimeout);
      bar_phase ^= 1u << s;
    } else {
      cp_async_wait<0>();
    }
    // rhs_o of the output plane k = m-1, loaded now so that its latency hides
    // behind the force computation below
    T ruo[MPT], rvo[MPT], rwo[MPT];
    if (m >= k0 + 1) {
#pragma unroll
      for (int hh = 0; hh < MPT; ++hh) {
        const size_t g = (size_t)i + (size_t)n * (y0 + ty + 8 * hh) + nn * wrapi(m - 1, n);
        ruo[hh] = a.ru[g];
        rvo[hh] = a.rv[g];
        rwo[hh] = a.rw[g];
      }
    }
    // plane m is visible, and every thread is done with iteration m-1, so the
    // slot plane m+PD reuses (plane m-3) is free: one barrier per plane fewer
    // than issuing the copy first (512^3: FP64 3.04 -> 2.98 ms, FP32 1.86 ->
    // 1.75 ms)
    __syncthreads();
    if (m + PD <= k0 + KZ) issue(sl[NS - 1], m + PD);
    else cp_async_commit();
    if (PF && m >= k0) {
      // B4: chempot, grad(phi), f at plane m-1 (multi/main.f90:617-623)
      const int fm = m - 1;
      // staged phi boxes start XS - 2 cells left of the ring
      const T* P0 = s_phi + sl[1] * G::PSL + (XS - 2);
      const T* Pm = s_phi + sl[0] * G::PSL + (XS - 2);
      const T* Pp = s_phi + sl[2] * G::PSL + (XS - 2);
      T* F = s_f + ((fm + 8) & 1) * 3 * QE;
#pragma unroll
      for (int r = 0; r < NQE; ++r) {
        const int e = tid + r * NT;
        if (r == NQE - 1 && e >= QE) break;
        const int pe = qpe[r];
        const T c = P0[pe], pxp = P0[pe + 1], pxm = P0[pe - 1], pyp = P0[pe + EX], pym = P0[pe - EX];
        const T pzp = Pp[pe], pzm = Pm[pe];
        const T ch = cf * fma(c * ((T)1 - c) * ((T)1 - (T)2 * c), epsi,
                              -(ed * fma((T)-6, c, pxp + pxm + pyp + pym + pzp + pzm)));
        F[e] = ch * (pxp - pxm);
        F[QE + e] = ch * (pyp - pym);
        F[2 * QE + e] = ch * (pzp - pzm);
      }
    }
    if (PF) __syncthreads();
    if (m >= k0 + 1) {
      const int k = m - 1;
      // staged velocity boxes start XS - 1 cells left of the ring
      const T* U0 = s_u + sl[1] * G::USL + (XS - 1);
      const T* Um = s_u + sl[0] * G::USL + (XS - 1);
      const T* Up = s_u + sl[2] * G::USL + (XS - 1);
      const T* V0 = s_v + sl[1] * G::USL + (XS - 1);
      const T* Vm = s_v + sl[0] * G::USL + (XS - 1);
      const T* Vp = s_v + sl[2] * G::USL + (XS - 1);
      const T* W0 = s_w + sl[1] * G::USL + (XS - 1);
      const T* Wm = s_w + sl[0] * G::USL + (XS - 1);
      const T* Wp = s_w + sl[2] * G::USL + (XS - 1);
#pragma unroll
      for (int hh = 0; hh < MPT; ++hh) {
        const int j = y0 + ty + 8 * hh;
        const int e = (tx + 1) + (ty + 8 * hh + 1) * UX;
        // The pending mean removal is applied as values enter registers.  Values
        // of this thread's column at planes k-1 and k, and the x/y neighbours
        // the previous plane already loaded, come from the previous output
        // plane's registers (z-marching register blocking): 17 shared loads
        // per point instead of 27.
        T uc, uzm, uxpzm, vc, vzm, vypzm, wc, wzm, wxm, wym;
        if (have_prev) {
          uzm = r_uc[hh]; uc = r_uzp[hh]; uxpzm = r_uxp[hh];
          vzm = r_vc[hh]; vc = r_vzp[hh]; vypzm = r_vyp[hh];
          wzm = r_wc[hh]; wc = r_wzp[hh]; wxm = r_wxmzp[hh]; wym = r_wymzp[hh];
        } else {
          uc = U0[e] - mu; uzm = Um[e] - mu; uxpzm = Um[e + 1] - mu;
          vc = V0[e] - mv; vzm = Vm[e] - mv; vypzm = Vm[e + UX] - mv;
          wc = W0[e] - mw; wzm = Wm[e] - mw; wxm = W0[e - 1] - mw; wym = W0[e - UX] - mw;
        }
        const T uxp = U0[e + 1] - mu, uxm = U0[e - 1] - mu, uyp = U0[e + UX] - mu, uym = U0[e - UX] - mu;
        const T uzp = Up[e] - mu, uxpym = U0[e + 1 - UX] - mu;
        const T vxp = V0[e + 1] - mv, vxm = V0[e - 1] - mv, vyp = V0[e + UX] - mv, vym = V0[e - UX] - mv;
        const T vzp = Vp[e] - mv, vxmyp = V0[e - 1 + UX] - mv;
        const T wxp = W0[e + 1] - mw, wyp = W0[e + UX] - mw;
        const T wzp = Wp[e] - mw, wxmzp = Wp[e - 1] - mw, wymzp = Wp[e - UX] - mw;
        r_uc[hh] = uc; r_uzp[hh] = uzp; r_uxp[hh] = uxp;
        r_vc[hh] = vc; r_vzp[hh] = vzp; r_vyp[hh] = vyp;
        r_wc[hh] = wc; r_wzp[hh] = wzp; r_wxmzp[hh] = wxmzp; r_wymzp[hh] = wymzp;
        // B1 (multi/main.f90:527-549); the fused multiply-adds are written out,
        // so that every instantiation (a slot of the ensemble among them)
        // rounds alike
        const T uyv = (uc + uym) * (vc + vxm), uzw = (uc + uzm) * (wc + wxm), vzw = (vc + vzm) * (wc + wym);
        const T cu = fma(uxp + uc, uxp + uc, -((uc + uxm) * (uc + uxm))) + fma(uyp + uc, vyp + vxmyp, -uyv) +
                     fma(uzp + uc, wzp + wxmzp, -uzw);
        const T cvv = fma(uxp + uxpym, vxp + vc, -uyv) + fma(vyp + vc, vyp + vc, -((vc + vym) * (vc + vym))) +
                      fma(wzp + wymzp, vzp + vc, -vzw);
        const T cw = fma(wxp + wc, uxp + uxpzm, -uzw) + fma(vyp + vypzm, wyp + wc, -vzw) +
                     fma(wzp + wc, wzp + wc, -((wc + wzm) * (wc + wzm)));
        // B2 (multi/main.f90:567-578)
        const T lu = (uxp - (T)2 * uc + uxm) + (uyp - (T)2 * uc + uym) + (uzp - (T)2 * uc + uzm);
        const T lv = (vxp - (T)2 * vc + vxm) + (vyp - (T)2 * vc + vym) + (vzp - (T)2 * vc + vzm);
        const T lw = (wxp - (T)2 * wc + wxm) + (wyp - (T)2 * wc + wym) + (wzp - (T)2 * wc + wzm);
        T ru = fma(cv, lu, -(cq * cu));
        T rv = fma(cv, lv, -(cq * cvv));
        T rw = fma(cv, lw, -(cq * cw));
        const int kz = wrapi(k, n);
        // B3 ABC forcing (multi/main.f90:591-593), global interior coordinates
        if (a.c.abc) {
          ru = fma(f2, (T)a.fcos[j], fma(f3, (T)a.fsin[kz], ru));
          rv = fma(f3, (T)a.fcos[kz], fma(f1, (T)a.fsin[i], rv));
          rw = fma(f1, (T)a.fcos[i], fma(f2, (T)a.fsin[j], rw));
        }
        if (lin != (T)0) {  // linear forcing (extension)
          ru = fma(lin, uc, ru);
          rv = fma(lin, vc, rv);
          rw = fma(lin, wc, rw);
        }
        if (PF) {  // B5 (multi/main.f90:652-654)
          const T* F0 = s_f + ((k + 8) & 1) * 3 * QE;
          const T* Fm = s_f + ((k + 7) & 1) * 3 * QE;
          const int qe = (tx + 1) + (ty + 8 * hh + 1) * QX;
          ru = ru + (F0[qe - 1] + F0[qe]);
          rv = rv + (F0[QE + qe - QX] + F0[QE + qe]);
          rw = rw + (Fm[2 * QE + qe] + F0[2 * QE + qe]);
        }
        // B6, B7 (multi/main.f90:666-681)
        const size_t g = (size_t)i + (size_t)n * j + nn * kz;
        a.us[g] = uc + fma(dta, ru, -(dtb * ruo[hh]));
        a.vs[g] = vc + fma(dta, rv, -(dtb * rvo[hh]));
        a.ws[g] = wc + fma(dta, rw, -(dtb * rwo[hh]));
        a.ru[g] = ru;
        a.rv[g] = rv;
        a.rw[g] = rw;
      }
      have_prev = true;
    }
    // rotate: the slot of plane m-2 takes plane m+PD+1 at the next iteration
    const int t = sl[0];
#pragma unroll
    for (int q2 = 0; q2 < NS - 1; ++q2) sl[q2] = sl[q2 + 1];
    sl[NS - 1] = t;
  }
}

// ============================================================ projection
// C2 + R1 (multi/main.f90:873-903): u = ustar - dt/rho*(p - p_m)*dxi, with the
// sums and maxima of the projected u, v, w reduced per CTA in FP64.
// z planes per projection CTA: 64 where n allows (512^3: FP64 projection plus
// finalize 1.47 -> 1.41 ms against 16 planes, with a quarter of the partials
// to reduce; FP32 projection 1.85 -> 1.49 ms); fewer on small grids, so that
// they too fill the GPU (FP64: 32^3 21 -> 8 us, 64^3 42 -> 9 us, 96^3 25 -> 14
// us, 128^3 68 -> 30 us, 192^3 92 -> 86 us).  The FP64 loop takes it as a
// compile-time trip count (a run-time one measured 1.79 ms at 512^3); the FP32
// refinement's loop, with a run-time one, depends on how the compiler unrolls it
// (384^3: 614 us as it stands, 644 not unrolled, 734 by 4 on request).
__host__ __device__ constexpr int project_kz(int n) {
  return n <= 96 ? 4 : (n <= 128 ? 8 : (n <= 192 ? 16 : (n % 64 == 0 ? 64 : 32)));
}

template <int PKZ>
__device__ __forceinline__ void project_body(const StencilArgs<double>& a, int bx, int by, int bz, int gx, int gy) {
  if (a.ctrl->status) return;
  const int n = a.c.n;
  const double dtr = a.c.dtr, dxi = a.c.dxi;
  const int i = bx * TX + threadIdx.x % TX, j = by * TY + threadIdx.x / TX;
  const int k0 = bz * PKZ;
  const int im = i ? i - 1 : n - 1, jm = j ? j - 1 : n - 1;
  const size_t nn = (size_t)n * n;
  double su = 0, sv = 0, sw = 0;
  double xu = -INFINITY, xv = -INFINITY, xw = -INFINITY;
  double pprev = a.p[(size_t)i + (size_t)n * j + nn * wrapi(k0 - 1, n)];
#pragma unroll 4
  for (int k = k0; k < k0 + PKZ; ++k) {
    const size_t g = (size_t)i + (size_t)n * j + nn * k;
    const double pc = a.p[g];
    const double uo = a.us[g] - dtr * (pc - a.p[g - i + im]) * dxi;
    const double vo = a.vs[g] - dtr * (pc - a.p[g + (size_t)n * jm - (size_t)n * j]) * dxi;
    const double wo = a.ws[g] - dtr * (pc - pprev) * dxi;
    pprev = pc;
    a.uo[g] = uo;
    a.vo[g] = vo;
    a.wo[g] = wo;
    su += uo;
    sv += vo;
    sw += wo;
    xu = fmax(xu, uo);
    xv = fmax(xv, vo);
    xw = fmax(xw, wo);
    // NaN must not vanish in fmax: fold it into the sums too
    if (uo != uo || vo != vo || wo != wo) su = NAN;
  }
  // deterministic block reduction: xor-shuffle in warps, then warps in order
  double vals[6] = {su, sv, sw, xu, xv, xw};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int t = 0; t < 3; ++t) vals[t] += __shfl_xor_sync(0xffffffffu, vals[t], o);
#pragma unroll
    for (int t = 3; t < 6; ++t) vals[t] = fmax(vals[t], __shfl_xor_sync(0xffffffffu, vals[t], o));
  }
  __shared__ double red[NT / 32][6];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
#pragma unroll
    for (int t = 0; t < 6; ++t) red[wid][t] = vals[t];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double r[6];
#pragma unroll
    for (int t = 0; t < 6; ++t) r[t] = red[0][t];
    for (int w = 1; w < NT / 32; ++w) {
      for (int t = 0; t < 3; ++t) r[t] += red[w][t];
      for (int t = 3; t < 6; ++t) r[t] = fmax(r[t], red[w][t]);
    }
    const size_t b = (size_t)bx + (size_t)gx * (by + (size_t)gy * bz);
    for (int t = 0; t < 6; ++t) a.partials[b * 6 + t] = r[t];
  }
  finish_step<NT, 6>(a.partials, gx * gy * (n / PKZ), a.ctrl, a.c);
}

// ============================================================ projection (FP32 refine)
// FP32 refinement form of C2 + R1: the pressure is p = p0 + dp (first FP32
// solve plus the FP32 correction solve of the FP64 residual), the projection
// u = ustar - dt/rho*(p - p_m)*dxi is evaluated in FP64 and rounded to FP32
// only when stored, and the forward-difference divergence of the FP64
// projected field is reduced (max |div u|) before that rounding.
__device__ __forceinline__ void project_refine_body(const StencilArgs<float>& a, const float* __restrict__ dp, int bx,
                                                    int by, int bz, int gx, int gy) {
  if (a.ctrl->status) return;
  const int n = a.c.n;
  const double dtr = a.c.dtr, dxi = a.c.dxi;
  const int i = bx * TX + threadIdx.x % TX, j = by * TY + threadIdx.x / TX;
  const int pkz = project_kz(n), k0 = bz * pkz;
  const int im = i ? i - 1 : n - 1, jm = j ? j - 1 : n - 1;
  const int ip = (i + 1 == n) ? 0 : i + 1, jp = (j + 1 == n) ? 0 : j + 1;
  const size_t nn = (size_t)n * n;
  const float* p0 = a.p;
  auto P = [&](size_t g) { return (double)p0[g] + (double)dp[g]; };
  double su = 0, sv = 0, sw = 0, mdiv = 0;
  double xu = -INFINITY, xv = -INFINITY, xw = -INFINITY;
  const size_t col = (size_t)i + (size_t)n * j;
  double pm = P(col + nn * wrapi(k0 - 1, n));
  double pc = P(col + nn * k0);
  double wsc = (double)a.ws[col + nn * k0];
  for (int k = k0; k < k0 + pkz; ++k) {
    const size_t g = col + nn * k;
    const int kp = (k + 1 == n) ? 0 : k + 1;
    const size_t gzp = col + nn * kp;
    const double pn = P(gzp);
    const double wsn = (double)a.ws[gzp];
    const size_t gxm = g - i + im, gxp = g - i + ip;
    const size_t gym = g - (size_t)n * j + (size_t)n * jm, gyp = g - (size_t)n * j + (size_t)n * jp;
    const double uo = (double)a.us[g] - dtr * (pc - P(gxm)) * dxi;
    const double vo = (double)a.vs[g] - dtr * (pc - P(gym)) * dxi;
    const double wo = wsc - dtr * (pc - pm) * dxi;
    const double u1 = (double)a.us[gxp] - dtr * (P(gxp) - pc) * dxi;
    const double v1 = (double)a.vs[gyp] - dtr * (P(gyp) - pc) * dxi;
    const double w1 = wsn - dtr * (pn - pc) * dxi;
    const double div = ((u1 - uo) + (v1 - vo) + (w1 - wo)) * dxi;
    mdiv = fmax(mdiv, fabs(div));
    if (div != div) mdiv = NAN;
    a.uo[g] = (float)uo;
    a.vo[g] = (float)vo;
    a.wo[g] = (float)wo;
    su += uo;
    sv += vo;
    sw += wo;
    xu = fmax(xu, uo);
    xv = fmax(xv, vo);
    xw = fmax(xw, wo);
    if (uo != uo || vo != vo || wo != wo) su = NAN;
    pm = pc;
    pc = pn;
    wsc = wsn;
  }
  double vals[7] = {su, sv, sw, xu, xv, xw, mdiv};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int t = 0; t < 3; ++t) vals[t] += __shfl_xor_sync(0xffffffffu, vals[t], o);
#pragma unroll
    for (int t = 3; t < 7; ++t) vals[t] = fmax(vals[t], __shfl_xor_sync(0xffffffffu, vals[t], o));
  }
  __shared__ double red[NT / 32][7];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0)
    for (int t = 0; t < 7; ++t) red[wid][t] = vals[t];
  __syncthreads();
  if (threadIdx.x == 0) {
    double r[7];
    for (int t = 0; t < 7; ++t) r[t] = red[0][t];
    for (int w = 1; w < NT / 32; ++w) {
      for (int t = 0; t < 3; ++t) r[t] += red[w][t];
      for (int t = 3; t < 7; ++t) r[t] = fmax(r[t], red[w][t]);
    }
    const size_t b = (size_t)bx + (size_t)gx * (by + (size_t)gy * bz);
    for (int t = 0; t < 7; ++t) a.partials[b * 7 + t] = r[t];
  }
}

// ============================================================ divergence check (FP32 refine)
// On request, the max |div u| of the FP32 refinement form's FP64 projection
// u = ustar - dt/rho*(p - p_m)*dxi with p = p0 + dp, from the stored ustar,
// p0 and dp: the arithmetic of project_refine_body's divergence, so it
// measures the field the step projected before rounding it to FP32.  Maxima
// are order-independent: CTAs combine theirs with an integer atomicMax on the
// bit patterns of the (non-negative, or NaN) values.
//
// A plane's p on the tile and its 1-cell ring is formed in FP64 once and shared
// through shared memory (two planes in turn, one barrier per plane), and a
// thread's own column passes through registers: 8 loads and conversions to
// FP64 per point instead of 17 (B200, 512^3: a call of two steps, which measures
// the divergence once, 16.31 -> 16.08 ms).
__global__ void __launch_bounds__(NT) refine_div_kernel(StencilArgs<float> a, const float* __restrict__ dp,
                                                        unsigned long long* __restrict__ out) {
  constexpr int PX = TX + 2, PY = TY + 2, NRING = 2 * TX + 2 * TY;
  __shared__ double sp[2][PX * PY];
  const int n = a.c.n, tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const double dtr = a.c.dtr, dxi = a.c.dxi;
  const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY;
  const int i = x0 + tx, j = y0 + ty;
  const int pkz = project_kz(n), k0 = blockIdx.z * pkz;
  const int ip = (i + 1 == n) ? 0 : i + 1, jp = (j + 1 == n) ? 0 : j + 1;
  const size_t nn = (size_t)n * n;
  const float* __restrict__ p0 = a.p;
  const float *__restrict__ us = a.us, *__restrict__ vs = a.vs, *__restrict__ ws = a.ws;
  auto P = [&](size_t g) { return (double)p0[g] + (double)dp[g]; };
  // the thread's ring cell (threads 0 .. NRING-1): bottom, top, left, right
  int rcell = 0;
  unsigned rcol = 0;
  {
    const int q = tid < 2 * TX ? tid : tid - 2 * TX;
    const int ex = tid < 2 * TX ? q % TX : (q < TY ? -1 : TX);
    const int ey = tid < 2 * TX ? (q < TX ? -1 : TY) : q % TY;
    rcell = (ex + 1) + (ey + 1) * PX;
    rcol = (unsigned)wrapi(x0 + ex, n) + (unsigned)n * (unsigned)wrapi(y0 + ey, n);
  }
  const int cell = (tx + 1) + (ty + 1) * PX;
  const unsigned col = (unsigned)i + (unsigned)n * j, colx = (unsigned)ip + (unsigned)n * j,
                 coly = (unsigned)i + (unsigned)n * jp;
  double mdiv = 0;
  double pm = P(nn * wrapi(k0 - 1, n) + col);
  double pc = P(nn * k0 + col);
  double wsc = (double)ws[nn * k0 + col];
  for (int k = k0; k < k0 + pkz; ++k) {
    const size_t z = nn * k, zp = nn * wrapi(k + 1, n);
    double* const s = sp[k & 1];
    s[cell] = pc;
    if (tid < NRING) s[rcell] = P(z + rcol);
    const double pn = P(zp + col), wsn = (double)ws[zp + col];
    const double usc = (double)us[z + col], usx = (double)us[z + colx];
    const double vsc = (double)vs[z + col], vsy = (double)vs[z + coly];
    __syncthreads();  // the other buffer is written next, after every thread has passed here
    const double uo = usc - dtr * (pc - s[cell - 1]) * dxi;
    const double vo = vsc - dtr * (pc - s[cell - PX]) * dxi;
    const double wo = wsc - dtr * (pc - pm) * dxi;
    const double u1 = usx - dtr * (s[cell + 1] - pc) * dxi;
    const double v1 = vsy - dtr * (s[cell + PX] - pc) * dxi;
    const double w1 = wsn - dtr * (pn - pc) * dxi;
    const double div = ((u1 - uo) + (v1 - vo) + (w1 - wo)) * dxi;
    mdiv = max_nan(mdiv, fabs(div));
    pm = pc;
    pc = pn;
    wsc = wsn;
  }
  for (int o = 16; o > 0; o >>= 1) mdiv = max_nan(mdiv, __shfl_xor_sync(0xffffffffu, mdiv, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, (unsigned long long)__double_as_longlong(fabs(mdiv)));
}

cudaError_t launch_refine_divergence(const StencilArgs<float>& a, const float* dp, double* out, cudaStream_t st) {
  const int n = a.c.n;
  cudaError_t e = cudaMemsetAsync(out, 0, sizeof(double), st);
  if (e) return e;
  dim3 grid(n / TX, n / TY, n / project_kz(n));
  refine_div_kernel<<<grid, NT, 0, st>>>(a, dp, reinterpret_cast<unsigned long long*>(out));
  return cudaGetLastError();
}

constexpr int FNT = 1024;  // threads of the FP32 refinement form's finalize

// ============================================================ entry points
// Single simulation: block coordinates are the grid's.
template <class T>
__global__ void __launch_bounds__(PNT, phase_min_blocks<T>())
    phase_kernel(const __grid_constant__ StencilArgs<T> a, const __grid_constant__ PhaseMaps maps) {
  phase_body<T, false>(a, a.phi_in, a.phi_out, gridDim.z, blockIdx.x, blockIdx.y, blockIdx.z, &maps);
}
template <class T, bool PF, int MTYv>
__global__ void __launch_bounds__(TX * 8, momentum_min_blocks<T>(PF, MTYv))
    momentum_kernel(const __grid_constant__ StencilArgs<T> a, const __grid_constant__ PlaneMaps maps) {
  momentum_body<T, PF, MTYv, true>(a, gridDim.z, blockIdx.x, blockIdx.y, blockIdx.z, &maps, false);
}
template <int PKZ> __global__ void __launch_bounds__(NT, 4) project_kernel(StencilArgs<double> a) {
  project_body<PKZ>(a, blockIdx.x, blockIdx.y, blockIdx.z, gridDim.x, gridDim.y);
}
__global__ void __launch_bounds__(NT) project_refine_kernel(StencilArgs<float> a, const float* __restrict__ dp) {
  project_refine_body(a, dp, blockIdx.x, blockIdx.y, blockIdx.z, gridDim.x, gridDim.y);
}

// The FP32 refinement form's projection is followed by a launch of its own for
// the step's scalars: with finish_step in it, it kept fewer loads in flight
// (384^3 on B200: 632 us with this launch, 786 us without).
__global__ void __launch_bounds__(FNT) finalize_refine_kernel(const double* __restrict__ partials, int nparts,
                                                              Ctrl* ctrl, StepConst c) {
  if (ctrl->status) return;
  finalize_step<FNT, 7>(partials, nparts, ctrl, (double)c.n, c.dt, c.dxi);
}

// Batched over the slots of a served ensemble: grid z (x for the finalize)
// covers the slots; each slot runs exactly the arithmetic of a single
// simulation, so a result is the same alone and in any mix.
template <class T>
__global__ void __launch_bounds__(PNT, phase_min_blocks<T>()) phase_kernel_b(const SlotArgs<T>* __restrict__ slots, int zch) {
  const int sl = blockIdx.z / zch;
  if (!slots[sl].active) return;
  const StencilArgs<T>& a = shared_args<PNT>(slots[sl].st);
  const int par = (int)(a.ctrl->nstep & 1);
  phase_body<T, true>(a, slots[sl].phi[par], slots[sl].phi[par ^ 1], zch, blockIdx.x, blockIdx.y,
                      blockIdx.z - sl * zch, &slots[sl].maps.phase[par]);
}
template <class T, bool PF, int MTYv>
__global__ void __launch_bounds__(TX * 8, momentum_min_blocks<T>(PF, MTYv)) momentum_kernel_b(const SlotArgs<T>* __restrict__ slots, int zch) {
  const int sl = blockIdx.z / zch;
  if (!slots[sl].active) return;
  StencilArgs<T> a = slots[sl].st;
  const int par = (int)((a.ctrl->nstep + 1) & 1);
  if (PF) a.phi_in = slots[sl].phi[par];  // the updated phi
  momentum_body<T, PF, MTYv, true>(a, zch, blockIdx.x, blockIdx.y, blockIdx.z - sl * zch,
                                   &slots[sl].maps.mom[MTYv == 16 ? 1 : 0][par], true);
}
template <int PKZ>
__global__ void __launch_bounds__(NT, 4) project_kernel_b(const SlotArgs<double>* __restrict__ slots, int zch) {
  const int sl = blockIdx.z / zch;
  if (!slots[sl].active) return;
  project_body<PKZ>(slots[sl].st, blockIdx.x, blockIdx.y, blockIdx.z - sl * zch, gridDim.x, gridDim.y);
}
__global__ void __launch_bounds__(NT) project_refine_kernel_b(const SlotArgs<float>* __restrict__ slots, int zch) {
  const int sl = blockIdx.z / zch;
  if (!slots[sl].active) return;
  project_refine_body(slots[sl].st, slots[sl].dp, blockIdx.x, blockIdx.y, blockIdx.z - sl * zch, gridDim.x,
                      gridDim.y);
}
__global__ void __launch_bounds__(FNT) finalize_refine_kernel_b(const SlotArgs<float>* __restrict__ slots, int nparts) {
  const int sl = blockIdx.x;
  if (!slots[sl].active || slots[sl].st.ctrl->status) return;
  const StepConst& c = slots[sl].st.c;
  finalize_step<FNT, 7>(slots[sl].st.partials, nparts, slots[sl].st.ctrl, (double)c.n, c.dt, c.dxi);
}

// Self-check of the bounded slot-barrier wait the staged-plane kernels use:
// one warp arms a barrier; if `arrive`, a thread arrives on it, otherwise
// nothing does and the wait gives up after `limit` cycles.  Writes 0 or the
// timeout status; the kernel returns either way.
__global__ void wait_check_kernel(int arrive, long long limit, int* out) {
  __shared__ unsigned long long bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_init_fence();
  }
  __syncthreads();
  if (arrive && threadIdx.x == 0) mbar_arrive(&bar);
  const bool ok = mbar_wait(&bar, 0, limit);
  __syncwarp();
  if (threadIdx.x == 0) *out = ok ? 0 : kStatusTimeout;
}

// u -= mean in place, then mean = 0 (materialises the lazy mean removal).  The
// last CTA clears the mean, which every CTA has read by then.
template <class T>
__global__ void materialize_kernel(T* u, T* v, T* w, size_t count, Ctrl* ctrl) {
  const T mu = (T)ctrl->mean[0], mv = (T)ctrl->mean[1], mw = (T)ctrl->mean[2];
  for (size_t g = blockIdx.x * (size_t)blockDim.x + threadIdx.x; g < count; g += (size_t)gridDim.x * blockDim.x) {
    u[g] = u[g] - mu;
    v[g] = v[g] - mv;
    w[g] = w[g] - mw;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicInc(&ctrl->ticket, gridDim.x - 1) == gridDim.x - 1) ctrl->mean[0] = ctrl->mean[1] = ctrl->mean[2] = 0;
  }
}

// ============================================================ launchers
template <class T> static size_t phase_smem() { return PhaseGeo<T>::smem(PsiMath<T>::TAB); }
template <class T> static size_t momentum_smem(bool pf, int mty) {
  const int ns = momentum_ring(mty);
  const size_t b = mty == 8 ? MomGeo<T, 8>::bar_offset(pf, ns) : MomGeo<T, 16>::bar_offset(pf, ns);
  return b + sizeof(unsigned long long) * ns;
}

// cuTensorMapEncodeTiled from the driver, resolved once through the runtime
// (no link-time dependency on the driver library).
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

cudaError_t encode_tensor_map(CUtensorMap* m, int rank, const void* base, const uint64_t* dims,
                              const uint64_t* strides, const uint32_t* box, int elem_bytes) {
  EncodeTiledFn fn = encode_tiled();
  if (!fn) return cudaErrorNotSupported;
  if (rank < 1 || rank > 3) return cudaErrorInvalidValue;
  cuuint64_t d[3], sb[2];
  cuuint32_t bx[3], estr[3] = {1, 1, 1};
  for (int i = 0; i < rank; ++i) {
    d[i] = dims[i];
    bx[i] = box[i];
    if (i + 1 < rank) sb[i] = strides[i];
  }
  const CUresult r = fn(m, elem_bytes == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64, (cuuint32_t)rank, const_cast<void*>(base), d, sb, bx, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// 2D map of an n^3 field as n columns by n*n rows, box bw x bh.
template <class T> static cudaError_t plane_map(CUtensorMap* m, const T* base, int n, int bw, int bh) {
  EncodeTiledFn fn = encode_tiled();
  if (!fn) return cudaErrorNotSupported;
  const cuuint64_t dims[2] = {(cuuint64_t)n, (cuuint64_t)n * n};
  const cuuint64_t strides[1] = {(cuuint64_t)n * sizeof(T)};
  const cuuint32_t box[2] = {(cuuint32_t)bw, (cuuint32_t)bh};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(m, sizeof(T) == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2,
                        const_cast<T*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <class T, int TYv> static cudaError_t momentum_maps(PlaneMaps* pm, const StencilArgs<T>& a, bool pf) {
  typedef MomGeo<T, TYv> G;
  const int n = a.c.n;
  cudaError_t e;
  if ((e = plane_map(&pm->u, a.u, n, G::UX, G::UY))) return e;
  if ((e = plane_map(&pm->v, a.v, n, G::UX, G::UY))) return e;
  if ((e = plane_map(&pm->w, a.w, n, G::UX, G::UY))) return e;
  if (pf && (e = plane_map(&pm->phi, a.phi_in, n, G::EX, G::EY))) return e;
  return cudaSuccess;
}

template <class T> static cudaError_t phase_maps(PhaseMaps* pm, const StencilArgs<T>& a) {
  typedef PhaseGeo<T> G;
  const int n = a.c.n;
  cudaError_t e;
  if ((e = plane_map(&pm->phi, a.phi_in, n, G::EX, G::EY))) return e;
  if ((e = plane_map(&pm->u, a.u, n, G::UW, PTY))) return e;
  if ((e = plane_map(&pm->v, a.v, n, TX, PTY + 1))) return e;
  return plane_map(&pm->w, a.w, n, TX, PTY);
}

// A served-ensemble slot's tensor maps: the momentum boxes for both tile
// heights and both phi parities, the phase kernel's boxes per parity, and
// the column passes' spectrum views.
template <class T> cudaError_t encode_slot_maps(SlotArgs<T>* s, int n, bool pf) {
  cudaError_t e;
  StencilArgs<T> a = s->st;
  a.c.n = n;
  for (int par = 0; par < 2; ++par) {
    a.phi_in = pf ? s->phi[par] : nullptr;
    if ((e = momentum_maps<T, 8>(&s->maps.mom[0][par], a, pf))) return e;
    if ((e = momentum_maps<T, 16>(&s->maps.mom[1][par], a, pf))) return e;
    if (pf && (e = phase_maps(&s->maps.phase[par], a))) return e;
  }
  return encode_column_maps<T>(&s->maps.col_y, &s->maps.col_z, s->po.spec, n);
}
template cudaError_t encode_slot_maps<double>(SlotArgs<double>*, int, bool);
template cudaError_t encode_slot_maps<float>(SlotArgs<float>*, int, bool);

int stencil_size_ok(int n) {
  return n >= 32 && n % TX == 0 && n % TY == 0 && n % PTY == 0 && n % project_kz(n) == 0;
}

int project_partials(int n) { return (n / TX) * (n / TY) * (n / project_kz(n)); }

template <class T> static cudaError_t prep_t() {
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(phase_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)phase_smem<T>())))
    return e;
  const void* mk[8] = {(const void*)momentum_kernel<T, true, 8>, (const void*)momentum_kernel<T, false, 8>,
                       (const void*)momentum_kernel<T, true, 16>, (const void*)momentum_kernel<T, false, 16>,
                       (const void*)momentum_kernel_b<T, true, 8>, (const void*)momentum_kernel_b<T, false, 8>,
                       (const void*)momentum_kernel_b<T, true, 16>, (const void*)momentum_kernel_b<T, false, 16>};
  for (int q = 0; q < 8; ++q) {
    const bool pf = (q % 2) == 0;
    const int mty = ((q / 2) % 2) ? 16 : 8;
    if ((e = cudaFuncSetAttribute(mk[q], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)momentum_smem<T>(pf, mty))))
      return e;
  }
  if ((e = cudaFuncSetAttribute(phase_kernel_b<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)phase_smem<T>())))
    return e;
  return cudaSuccess;
}

cudaError_t prepare_stencils() {
  cudaError_t e = upload_log_table();
  if (e) return e;
  e = prep_t<double>();
  if (e) return e;
  return prep_t<float>();
}

template <class T> cudaError_t launch_phase(const StencilArgs<T>& a, cudaStream_t st, int kz) {
  const int n = a.c.n;
  const int tiles = (n / TX) * (n / PTY);
  dim3 grid(n / TX, n / PTY, kz > 0 ? n / kz : pick_chunks(n, tiles, phase_min_blocks<T>() * sm_count(), 4));
  PhaseMaps pm;
  cudaError_t e = phase_maps(&pm, a);
  if (e) return e;
  phase_kernel<T><<<grid, PNT, phase_smem<T>(), st>>>(a, pm);
  return cudaGetLastError();
}

template <class T> cudaError_t launch_momentum(const StencilArgs<T>& a, bool pf, cudaStream_t st, int kz, int mty) {
  const int n = a.c.n;
  if (mty != 8) mty = 16;
  const int tiles = (n / TX) * (n / mty);
  dim3 grid(n / TX, n / mty, kz > 0 ? n / kz : pick_chunks(n, tiles, momentum_min_blocks<T>(pf, mty) * sm_count(), 3));
  const size_t sm = momentum_smem<T>(pf, mty);
  PlaneMaps pm;
  memset(&pm, 0, sizeof(pm));
  cudaError_t e = mty == 8 ? momentum_maps<T, 8>(&pm, a, pf) : momentum_maps<T, 16>(&pm, a, pf);
  if (e) return e;
  if (mty == 8) {
    if (pf) momentum_kernel<T, true, 8><<<grid, TX * 8, sm, st>>>(a, pm);
    else momentum_kernel<T, false, 8><<<grid, TX * 8, sm, st>>>(a, pm);
  } else {
    if (pf) momentum_kernel<T, true, 16><<<grid, TX * 8, sm, st>>>(a, pm);
    else momentum_kernel<T, false, 16><<<grid, TX * 8, sm, st>>>(a, pm);
  }
  return cudaGetLastError();
}

cudaError_t launch_project(const StencilArgs<double>& a, cudaStream_t st) {
  const int n = a.c.n;
  dim3 grid(n / TX, n / TY, n / project_kz(n));
  switch (project_kz(n)) {
    case 64: project_kernel<64><<<grid, NT, 0, st>>>(a); break;
    case 16: project_kernel<16><<<grid, NT, 0, st>>>(a); break;
    case 8: project_kernel<8><<<grid, NT, 0, st>>>(a); break;
    default: project_kernel<4><<<grid, NT, 0, st>>>(a); break;
  }
  return cudaGetLastError();
}

cudaError_t launch_project_refine(const StencilArgs<float>& a, const float* dp, cudaStream_t st) {
  const int n = a.c.n;
  dim3 grid(n / TX, n / TY, n / project_kz(n));
  project_refine_kernel<<<grid, NT, 0, st>>>(a, dp);
  return cudaGetLastError();
}

cudaError_t launch_finalize_refine(const StencilArgs<float>& a, cudaStream_t st) {
  finalize_refine_kernel<<<1, FNT, 0, st>>>(a.partials, project_partials(a.c.n), a.ctrl, a.c);
  return cudaGetLastError();
}
cudaError_t launch_finalize_refine_batched(const SlotArgs<float>* slots, int nslots, int n, cudaStream_t st) {
  finalize_refine_kernel_b<<<nslots, FNT, 0, st>>>(slots, project_partials(n));
  return cudaGetLastError();
}

template <class T> cudaError_t launch_materialize(T* u, T* v, T* w, int n, Ctrl* ctrl, cudaStream_t st) {
  const size_t count = (size_t)n * n * n;
  const int grid = (int)(count / 256 < 1184 ? count / 256 : 1184);
  materialize_kernel<T><<<grid, 256, 0, st>>>(u, v, w, count, ctrl);
  return cudaGetLastError();
}

int stencil_kz_ok(int n, int kz) { return kz >= 2 && kz <= n && n % kz == 0; }

cudaError_t launch_wait_check(int arrive, long long limit_cycles, int* out_dev, cudaStream_t st) {
  wait_check_kernel<<<1, 32, 0, st>>>(arrive, limit_cycles, out_dev);
  return cudaGetLastError();
}

template <class T>
cudaError_t launch_phase_batched(const SlotArgs<T>* slots, int nslots, int n, int kz, cudaStream_t st) {
  dim3 grid(n / TX, n / PTY, (n / kz) * nslots);
  phase_kernel_b<T><<<grid, PNT, phase_smem<T>(), st>>>(slots, n / kz);
  return cudaGetLastError();
}
template <class T>
cudaError_t launch_momentum_batched(const SlotArgs<T>* slots, int nslots, int n, int kz, bool pf, cudaStream_t st,
                                   int mty) {
  if (mty != 8) mty = 16;
  dim3 grid(n / TX, n / mty, (n / kz) * nslots);
  const size_t sm = momentum_smem<T>(pf, mty);
  if (mty == 8) {
    if (pf) momentum_kernel_b<T, true, 8><<<grid, TX * 8, sm, st>>>(slots, n / kz);
    else momentum_kernel_b<T, false, 8><<<grid, TX * 8, sm, st>>>(slots, n / kz);
  } else {
    if (pf) momentum_kernel_b<T, true, 16><<<grid, TX * 8, sm, st>>>(slots, n / kz);
    else momentum_kernel_b<T, false, 16><<<grid, TX * 8, sm, st>>>(slots, n / kz);
  }
  return cudaGetLastError();
}
template <class T>
cudaError_t launch_project_batched(const SlotArgs<T>* slots, int nslots, int n, cudaStream_t st) {
  dim3 grid(n / TX, n / TY, (n / project_kz(n)) * nslots);
  if constexpr (sizeof(T) == 8) {
    switch (project_kz(n)) {
      case 64: project_kernel_b<64><<<grid, NT, 0, st>>>(slots, n / project_kz(n)); break;
      case 16: project_kernel_b<16><<<grid, NT, 0, st>>>(slots, n / project_kz(n)); break;
      case 8: project_kernel_b<8><<<grid, NT, 0, st>>>(slots, n / project_kz(n)); break;
      default: project_kernel_b<4><<<grid, NT, 0, st>>>(slots, n / project_kz(n)); break;
    }
  } else
    project_refine_kernel_b<<<grid, NT, 0, st>>>(slots, n / project_kz(n));
  return cudaGetLastError();
}
template cudaError_t launch_project_batched<double>(const SlotArgs<double>*, int, int, cudaStream_t);
template cudaError_t launch_project_batched<float>(const SlotArgs<float>*, int, int, cudaStream_t);
template cudaError_t launch_phase_batched<double>(const SlotArgs<double>*, int, int, int, cudaStream_t);
template cudaError_t launch_phase_batched<float>(const SlotArgs<float>*, int, int, int, cudaStream_t);
template cudaError_t launch_momentum_batched<double>(const SlotArgs<double>*, int, int, int, bool, cudaStream_t, int);
template cudaError_t launch_momentum_batched<float>(const SlotArgs<float>*, int, int, int, bool, cudaStream_t, int);

template cudaError_t launch_phase<double>(const StencilArgs<double>&, cudaStream_t, int);
template cudaError_t launch_phase<float>(const StencilArgs<float>&, cudaStream_t, int);
template cudaError_t launch_momentum<double>(const StencilArgs<double>&, bool, cudaStream_t, int, int);
template cudaError_t launch_momentum<float>(const StencilArgs<float>&, bool, cudaStream_t, int, int);
template cudaError_t launch_materialize<double>(double*, double*, double*, int, Ctrl*, cudaStream_t);
template cudaError_t launch_materialize<float>(float*, float*, float*, int, Ctrl*, cudaStream_t);

}  // namespace mhit
