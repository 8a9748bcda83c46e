// Drop count and size distribution of the phase field on the GPU.
//
// Restates the serial post-processor post/DropCountSize: binarise phi >= 0.5
// (get_interface.f90:12-22), find 26-connected components with periodic wrap
// (the recursive flood fill of flood_fill.f90:1-127, which overflows the stack
// for large drops), number the drops in the order the Fortran scan meets
// their first cell (get_interface.f90:28-47), and give each drop's equivalent
// diameter deq = dx*(6 V/pi)^(1/3) with V its cell count (calculate_deq.f90:29-33).
//
// GPU algorithm: cells are packed into one bit each, 32 to a word along x, and
// the nodes of a lock-free union-find are the runs of set bits within a word,
// named by their first cell's linear index.  A word's runs are united with
// the runs they touch in the next word of the row and in the four forward
// rows (the other half of the 26 neighbours is seen from the other side).
// Roots only ever decrease (atomicMin), so each component's root ends as its
// smallest linear index -- the cell the reference's scan reaches first -- and
// sorting the roots reproduces the reference's order.  What bounds it is the
// one read of phi: the passes after it read a bit per cell and touch labels
// only where a run starts (a label per cell, written, read and united cell by
// cell, moved 16 bytes per cell more and queued every cell of a drop on one
// counter).  256^3 with 8 drops on B200: Solver.drops 0.79 -> 0.16 ms.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <vector>

#include "internal.h"

namespace mhit {

constexpr int WPT = 4;  // words a warp packs at a time (loads in flight per thread)

// bits[w] = (phi >= 0.5) of cells 32w .. 32w+31; a run's first cell starts as
// its own root with count 0.
template <class T>
__global__ void __launch_bounds__(256) ccl_pack_kernel(const T* __restrict__ phi, unsigned* __restrict__ bits,
                                                       int* __restrict__ lab, int* __restrict__ cnt, int nwords) {
  const int lane = threadIdx.x & 31;
  const int warps = (int)(gridDim.x * (blockDim.x >> 5));
  for (int w = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * WPT; w < nwords; w += warps * WPT) {
    T v[WPT];
#pragma unroll
    for (int q = 0; q < WPT; ++q) v[q] = phi[(size_t)(w + q) * 32 + lane];
#pragma unroll
    for (int q = 0; q < WPT; ++q) {
      const unsigned b = __ballot_sync(0xffffffffu, v[q] >= (T)0.5);
      if (lane == q) bits[w + q] = b;
      if (((b & ~(b << 1)) >> lane) & 1u) {
        const int g = (w + q) * 32 + lane;
        lab[g] = g;
        cnt[g] = 0;
      }
    }
  }
}

// Root of x.  Labels only decrease and L[x] <= x, so the chain strictly
// decreases and ends within x steps; the loop bound only makes that explicit.
__device__ __forceinline__ int ccl_find(const int* L, int x) {
  int p = L[x];
  for (int it = 0; p != x && it < (1 << 30); ++it) {
    x = p;
    p = L[x];
  }
  return x;
}

__device__ __forceinline__ void ccl_unite(int* L, int a, int b, int* err) {
  for (int it = 0; it < (1 << 24); ++it) {
    a = ccl_find(L, a);
    b = ccl_find(L, b);
    if (a == b) return;
    if (a > b) {
      const int t = a;
      a = b;
      b = t;
    }
    const int old = atomicMin(&L[b], a);
    if (old == b) return;
    b = old;
  }
  atomicExch(err, 1);  // bounded retry loop gave up (never expected)
}

// The lowest run of m (m != 0), and the first bit of the run of b that holds bit p.
__device__ __forceinline__ unsigned low_run(unsigned m) { return m & ~(m + (m & (0u - m))); }
__device__ __forceinline__ int run_start(unsigned b, int p) {
  const unsigned z = ~b & ((1u << p) - 1u);  // zeros below p
  return z ? 32 - __clz(z) : 0;
}

__global__ void __launch_bounds__(256) ccl_merge_kernel(const unsigned* __restrict__ bits, int* L, int n, int nwords,
                                                        int* err) {
  const int W = n / 32;  // words per row
  for (int w = (int)(blockIdx.x * blockDim.x + threadIdx.x); w < nwords; w += (int)(gridDim.x * blockDim.x)) {
    const unsigned b = bits[w];
    if (!b) continue;
    const int row = w / W, wx = w % W, j = row % n, k = row / n;
    const int xl = wx ? wx - 1 : W - 1, xr = (wx + 1 == W) ? 0 : wx + 1;
    if (b >> 31) {
      const int wr = row * W + xr;
      if (bits[wr] & 1u) ccl_unite(L, w * 32 + run_start(b, 31), wr * 32, err);
    }
    // forward rows (dj, dk): (1, 0), (-1, 1), (0, 1), (1, 1)
    for (int q = 0; q < 4; ++q) {
      const int row2 = wrapi(j + (q == 0 ? 1 : q - 2), n) + n * wrapi(k + (q == 0 ? 0 : 1), n);
      const int w2 = row2 * W + wx;
      const unsigned nb = bits[w2];
      const unsigned nl = (b & 1u) ? bits[row2 * W + xl] >> 31 : 0u, nr = (b >> 31) ? bits[row2 * W + xr] & 1u : 0u;
      if (!(nb | nl | nr)) continue;
      for (unsigned m = b; m;) {
        const unsigned run = low_run(m);
        m &= ~run;
        const int g = w * 32 + __ffs(run) - 1;
        for (unsigned touch = (run | (run << 1) | (run >> 1)) & nb; touch;) {
          const int s = run_start(nb, __ffs(touch) - 1);
          touch &= ~low_run(nb & ~((1u << s) - 1u));
          ccl_unite(L, g, w2 * 32 + s, err);
        }
        if ((run & 1u) && nl) ccl_unite(L, g, (row2 * W + xl) * 32 + run_start(bits[row2 * W + xl], 31), err);
        if ((run >> 31) && nr) ccl_unite(L, g, (row2 * W + xr) * 32, err);
      }
    }
  }
}

__global__ void __launch_bounds__(256) ccl_count_kernel(const unsigned* __restrict__ bits, const int* __restrict__ L,
                                                        int* __restrict__ cnt, int nwords) {
  for (int w = (int)(blockIdx.x * blockDim.x + threadIdx.x); w < nwords; w += (int)(gridDim.x * blockDim.x)) {
    for (unsigned m = bits[w]; m;) {
      const unsigned run = low_run(m);
      m &= ~run;
      atomicAdd(&cnt[ccl_find(L, w * 32 + __ffs(run) - 1)], __popc(run));
    }
  }
}

__global__ void __launch_bounds__(256) ccl_roots_kernel(const unsigned* __restrict__ bits, const int* __restrict__ L,
                                                        const int* __restrict__ cnt, int nwords,
                                                        int2* __restrict__ out, int cap, int* __restrict__ nout) {
  for (int w = (int)(blockIdx.x * blockDim.x + threadIdx.x); w < nwords; w += (int)(gridDim.x * blockDim.x)) {
    for (unsigned m = bits[w]; m;) {
      const unsigned run = low_run(m);
      m &= ~run;
      const int g = w * 32 + __ffs(run) - 1;
      if (L[g] == g) {
        const int slot = atomicAdd(nout, 1);
        if (slot < cap) out[slot] = make_int2(g, cnt[g]);
      }
    }
  }
}

// n is a multiple of 32 (every built size), so a row is a whole number of
// words and the words a multiple of WPT.
template <class T>
cudaError_t launch_dropcount(const T* phi, int n, unsigned* bits, int* lab, int* cnt, int2* roots, int cap,
                             int* d_counter, cudaStream_t st) {
  if (n % 32) return cudaErrorInvalidValue;
  const int nwords = (int)((size_t)n * n * n / 32);
  const int block = 256, grid = std::min(148 * 8, (nwords + block - 1) / block);
  const int pgrid = std::min(148 * 8, (nwords / WPT + 7) / 8);
  cudaError_t e = cudaMemsetAsync(d_counter, 0, 2 * sizeof(int), st);  // [0] roots, [1] error flag
  if (e) return e;
  ccl_pack_kernel<T><<<pgrid, block, 0, st>>>(phi, bits, lab, cnt, nwords);
  ccl_merge_kernel<<<grid, block, 0, st>>>(bits, lab, n, nwords, d_counter + 1);
  ccl_count_kernel<<<grid, block, 0, st>>>(bits, lab, cnt, nwords);
  ccl_roots_kernel<<<grid, block, 0, st>>>(bits, lab, cnt, nwords, roots, cap, d_counter);
  return cudaGetLastError();
}

template cudaError_t launch_dropcount<double>(const double*, int, unsigned*, int*, int*, int2*, int, int*,
                                              cudaStream_t);
template cudaError_t launch_dropcount<float>(const float*, int, unsigned*, int*, int*, int2*, int, int*,
                                             cudaStream_t);

}  // namespace mhit
