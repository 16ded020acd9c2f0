// The kernels' own elementary functions, one value per thread, for the accuracy
// tests (not part of the C ABI's header).
#include "atb_physics.cuh"

namespace atb {
// 0: logarithmic mean of x and y (log_mean_parts)
__global__ void math_kernel(int fn, const double* x, const double* y, double* out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double r = 0.0;
  if (fn == 0) {
    double num, den;
    log_mean_parts(x[i], y[i], num, den);
    r = num * rcp_cheb(den);
  }
  out[i] = r;
}
}  // namespace atb

// x, y, out: device arrays of n values; returns the launch's CUDA status
extern "C" int atb_detail_math(int fn, const double* x, const double* y, double* out, int n, void* stream) {
  if (n <= 0) return 0;
  atb::math_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(fn, x, y, out, n);
  return (int)cudaGetLastError();
}
