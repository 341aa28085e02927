// Test-only: the device side of amcafe_gb300/csrc/cafe_intmath.h beside the
// floating-point functions, as intmath_check.cpp does for the host side. Built by
// tests/test_gpu_intmath.py.
#include <cuda_runtime.h>

#include "../../amcafe_gb300/csrc/cafe_intmath.h"

template <int FN>
__global__ void k_eval(long n, const double *x, const double *y, double *got, double *want) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const double a = x[i], b = y[i];
    if (FN == 0) got[i] = crm_exp_int(a), want[i] = crm_exp(a);
    if (FN == 1) got[i] = crm_div_int(a, b), want[i] = a / b;
    if (FN == 2) got[i] = crm_quotient(a, crm_reciprocal(b), b, 1), want[i] = a / (2 * b);
    if (FN == 3) got[i] = crm_sqrt_int(a), want[i] = sqrt(a);
    if (FN == 4) got[i] = crm_atan2_int(a, b), want[i] = crm_atan2(a, b);
    if (FN == 5) got[i] = crm_cos_int(a), want[i] = crm_cos(a);
    if (FN == 6) got[i] = crm_sin_int(a), want[i] = crm_sin(a);
  }
}

// 0, or the CUDA error.
extern "C" int ic_gpu(int fn, long n, const double *x, const double *y, double *got, double *want) {
  double *d = nullptr;
  const size_t b = (size_t)n * sizeof(double);
  cudaError_t e = cudaMalloc((void **)&d, 4 * b);
  if (e) return (int)e;
  cudaMemcpy(d, x, b, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, y, b, cudaMemcpyHostToDevice);
  void (*const k[])(long, const double *, const double *, double *, double *) = {
      k_eval<0>, k_eval<1>, k_eval<2>, k_eval<3>, k_eval<4>, k_eval<5>, k_eval<6>};
  k[fn]<<<608, 256>>>(n, d, d + n, d + 2 * n, d + 3 * n);
  cudaMemcpy(got, d + 2 * n, b, cudaMemcpyDeviceToHost);
  cudaMemcpy(want, d + 3 * n, b, cudaMemcpyDeviceToHost);
  e = cudaGetLastError();
  cudaFree(d);
  return (int)e;
}
