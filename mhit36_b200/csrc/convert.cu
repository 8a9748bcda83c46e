// FP32 fields at the FP64 boundary: rounding to FP32 and widening to FP64 on
// the GPU, between the host copy's staging buffer and the resident field.  A
// pass moves 12 bytes per value (16 with a second operand) through HBM, about
// 2 us per million values, where a host loop into a fresh array took 1.3 ms
// (192^3 on B200: set_fields 37 -> 21 ms, get_fields 82 -> 52 ms).
#include <cuda_runtime.h>
#include "internal.h"

namespace mhit {

__global__ void __launch_bounds__(256) narrow_kernel(const double* __restrict__ src, float* __restrict__ dst,
                                                     size_t count) {
  for (size_t g = blockIdx.x * (size_t)blockDim.x + threadIdx.x; g < count; g += (size_t)gridDim.x * blockDim.x)
    dst[g] = (float)src[g];
}

// dst = a (+ b), in FP64
__global__ void __launch_bounds__(256) widen_kernel(const float* __restrict__ a, const float* __restrict__ b,
                                                    double* __restrict__ dst, size_t count) {
  for (size_t g = blockIdx.x * (size_t)blockDim.x + threadIdx.x; g < count; g += (size_t)gridDim.x * blockDim.x)
    dst[g] = b ? (double)a[g] + (double)b[g] : (double)a[g];
}

static int convert_grid(size_t count) {
  const size_t g = (count + 255) / 256;
  return (int)(g < 148 * 16 ? g : 148 * 16);
}

cudaError_t launch_narrow(const double* src, float* dst, size_t count, cudaStream_t st) {
  narrow_kernel<<<convert_grid(count), 256, 0, st>>>(src, dst, count);
  return cudaGetLastError();
}

cudaError_t launch_widen(const float* a, const float* b, double* dst, size_t count, cudaStream_t st) {
  widen_kernel<<<convert_grid(count), 256, 0, st>>>(a, b, dst, count);
  return cudaGetLastError();
}

}  // namespace mhit
