// The kernels' own elementary functions, one value per thread, for the accuracy
// tests (not part of the C ABI's header).
#include "atb_fd.cuh"

namespace atb {
// 0: logarithmic mean of x and y (log_mean_parts); of x: 1 rcp_cheb, 2 sqrt_house,
// 3 mean_F, 4 mean_Gh, 5 mean_F_wide; 6: x / y in FP32 (div32)
__global__ void math_kernel(int fn, const double* x, const double* y, double* out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double r = 0.0;
  if (fn == 0) {
    double num, den;
    log_mean_parts(x[i], y[i], num, den);
    r = num * rcp_cheb(den);
  } else if (fn == 6) {
    r = (double)div32((float)x[i], (float)y[i], rcp32((float)y[i]));
  } else {
    const double v = x[i];
    r = fn == 1 ? rcp_cheb(v) : fn == 2 ? sqrt_house(v) : fn == 3 ? mean_F(v) : fn == 4 ? mean_Gh(v) : mean_F_wide(v);
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
