// C entry of tests/test_gpu_fp64math.py: the elementary steps of
// marie-tools_gb300/csrc/fp64math.cuh on n host values.
#include <cuda_runtime.h>

#include "../marie-tools_gb300/csrc/fp64math.cuh"

__global__ void k_probe(int what, const double* x, double* a, double* b, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double u, v;
  if (what == 0) u = marie::inv_sqrt(x[i], v);
  else if (what == 1) marie::sin_cos(x[i], &u, &v);
  else marie::sin_cos_small(x[i], &u, &v);
  a[i] = u;
  b[i] = v;
}

extern "C" int fp64math_probe(int what, const double* x, double* a, double* b, int n) {
  double* d = nullptr;
  if (cudaMalloc(&d, 3 * sizeof(double) * n) != cudaSuccess) return 1;
  cudaMemcpy(d, x, sizeof(double) * n, cudaMemcpyHostToDevice);
  k_probe<<<(n + 255) / 256, 256>>>(what, d, d + n, d + 2 * n, n);
  cudaMemcpy(a, d + n, sizeof(double) * n, cudaMemcpyDeviceToHost);
  cudaMemcpy(b, d + 2 * n, sizeof(double) * n, cudaMemcpyDeviceToHost);
  const int st = cudaGetLastError() != cudaSuccess;
  cudaFree(d);
  return st;
}
