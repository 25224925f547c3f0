// The library's FP64 reciprocal (gnurbs::fast::rcp) over an array, for tests/test_gpu_rcp.py.
#include <cuda_runtime.h>

#include "nurbs_internal.h"
#include "nurbs_math.cuh"

__global__ void k_rcp(const double* x, double* y, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = gnurbs::fast::rcp<false>(x[i]);
}

extern "C" int rcp_check(const double* x_host, double* y_host, long long n) {
  double *x = nullptr, *y = nullptr;
  cudaError_t e = cudaMalloc(&x, n * sizeof(double));
  if (e == cudaSuccess) e = cudaMalloc(&y, n * sizeof(double));
  if (e == cudaSuccess) e = cudaMemcpy(x, x_host, n * sizeof(double), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_rcp<<<(unsigned)((n + 255) / 256), 256>>>(x, y, n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(y_host, y, n * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(x);
  cudaFree(y);
  return (int)e;
}
