// The broadened sums' reciprocal by itself, for test_gpu_reciprocal.py.
#include "k_spectrum.cu"

namespace {
__global__ void reciprocals_kernel(const double* x, int n, double* r, double* q) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  r[i] = wtb::reciprocal(x[i]);
  q[i] = 1.0 / x[i];
}
}  // namespace

extern "C" int reciprocals(const double* x, int n, double* r, double* q) {
  if (n < 1) return -1;
  reciprocals_kernel<<<(n + 255) / 256, 256>>>(x, n, r, q);
  const cudaError_t e = cudaGetLastError();
  return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
