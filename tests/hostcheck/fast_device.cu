// The operations of mhd_fast.cuh on the GPU for tests/test_fast_physics_gpu.py:
// fast_ops as in fast_host.cpp, the fast side formed by a kernel.
#include <cuda_runtime.h>

#include <cmath>

#include "mhd_fast.cuh"

using namespace athb;

static __global__ void k_ops(int op, int n, const double* x, const double* y, double* out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  double h;
  switch (op) {
  case 0: out[k] = recip(x[k]); break;
  case 1: out[k] = root(x[k]); break;
  case 2: out[k] = quot(y[k], x[k], recip(x[k])); break;
  case 3: {
    const double g = root(x[k], h);
    out[k] = recip_of_root(g, h);
    break;
  }
  default: root(x[k], h); out[k] = h;
  }
}

// 0, or the CUDA error
extern "C" int fast_ops(int op, int n, const double* x, const double* y, double* fast, double* plain) {
  for (int k = 0; k < n; k++) {
    switch (op) {
    case 0: plain[k] = 1.0 / x[k]; break;
    case 1: plain[k] = std::sqrt(x[k]); break;
    case 2: plain[k] = y[k] / x[k]; break;
    case 3: plain[k] = 1.0 / std::sqrt(x[k]); break;
    default: plain[k] = 0.5 / std::sqrt(x[k]);
    }
    fast[k] = NAN;
  }
  if (n < 1) return 0;
  double* d = nullptr;
  const size_t b = sizeof(double) * (size_t)n;
  cudaError_t e = cudaMalloc(&d, 3 * b);
  if (e == cudaSuccess) e = cudaMemcpy(d, x, b, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + n, y, b, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_ops<<<(n + 127) / 128, 128>>>(op, n, d, d + n, d + 2 * (size_t)n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(fast, d + 2 * (size_t)n, b, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}
