// q[i] = lqm_div_normal(a[i], b[i]) on the device, host arrays in and out.
#include "lqm_eigh.cuh"

__global__ void div_kernel(const double* a, const double* b, double* q, long long m) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < m) q[i] = lqm_div_normal(a[i], b[i]);
}

extern "C" int div_normal(const double* a, const double* b, double* q, long long m) {
  double* d = nullptr;
  if (cudaMalloc(&d, 3 * m * sizeof(double)) != cudaSuccess) return 1;
  cudaMemcpy(d, a, m * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemcpy(d + m, b, m * sizeof(double), cudaMemcpyHostToDevice);
  div_kernel<<<(unsigned)((m + 255) / 256), 256>>>(d, d + m, d + 2 * m, m);
  cudaMemcpy(q, d + 2 * m, m * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}
