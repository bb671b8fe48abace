// The quotients of cov_div.cuh beside CUDA's own division, for
// test_gpu_edges.py: kind 0 div_fast (in: div_range of both operands), 1 div_by
// with the rounded reciprocal.
#include <cuda_runtime.h>

#include "cov_div.cuh"

__global__ void k_quotients(int kind, const double* x, const double* b, int n, double* q, double* ieee, int* in) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  q[i] = kind ? covgpu::div_by(x[i], b[i], __drcp_rn(b[i])) : covgpu::div_fast(x[i], b[i]);
  ieee[i] = __ddiv_rn(x[i], b[i]);
  in[i] = covgpu::div_range(x[i]) && covgpu::div_range(b[i]);
}

extern "C" int quotients(int kind, const double* x, const double* b, int n, double* q, double* ieee, int* in) {
  double* d = nullptr;
  int* di = nullptr;
  const size_t s = (size_t)n * sizeof(double);
  cudaError_t e = cudaMalloc(&d, 4 * s);
  if (e == cudaSuccess) e = cudaMalloc(&di, n * sizeof(int));
  if (e == cudaSuccess) e = cudaMemcpy(d, x, s, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + n, b, s, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) k_quotients<<<(n + 255) / 256, 256>>>(kind, d, d + n, n, d + 2 * (size_t)n, d + 3 * (size_t)n, di);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpy(q, d + 2 * (size_t)n, s, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(ieee, d + 3 * (size_t)n, s, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(in, di, n * sizeof(int), cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(di);
  return (int)e;
}
