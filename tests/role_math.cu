// The window kernels' reciprocal square root and reciprocal, entry by entry.
// Built by test_gpu_role_math.py.
#include <cuda_runtime.h>

#include "qz_roles.cuh"

__global__ void k_role_math(const double* x, double* root, double* inv, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    root[i] = qz::role_rsqrt(x[i]);
    inv[i] = qz::role_rcp(x[i]);
  }
}

extern "C" int role_math(const double* x, double* root, double* inv, int n) {
  k_role_math<<<(n + 255) / 256, 256>>>(x, root, inv, n);
  const cudaError_t e = cudaGetLastError();
  return e != cudaSuccess ? (int)e : (int)cudaDeviceSynchronize();
}
