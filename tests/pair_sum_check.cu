// The sums of csrc/pair_arith.cuh across a warp: n pairs of sums over 32 lanes.
#include <cuda_runtime.h>

#include "../pynfam_gb300/csrc/pair_arith.cuh"

__global__ void k_check(int n, const float2* a, const float2* b, double* out) {
  const int i = blockIdx.x, l = threadIdx.x;   // grid n, 32 threads
  const double s = pnfam::pair_warp_sums(a[32 * i + l], b[32 * i + l], l);
  if ((l & 15) == 0) out[2 * i + (l >> 4)] = s;
}

// a, b [n][32] pairs; out [n][2]; returns a CUDA error
extern "C" int pair_sum_check(int n, const float* a, const float* b, double* out) {
  const size_t nb = sizeof(float2) * 32 * n;
  float2* d = nullptr;
  double* o = nullptr;
  cudaError_t e = cudaMalloc(&d, 2 * nb);
  if (e == cudaSuccess) e = cudaMalloc(&o, sizeof(double) * 2 * n);
  if (e == cudaSuccess) e = cudaMemcpy(d, a, nb, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + 32 * (size_t)n, b, nb, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_check<<<n, 32>>>(n, d, d + 32 * (size_t)n, o);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, o, sizeof(double) * 2 * n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(o);
  return (int)e;
}
