// The back-transformation's kernels and its rule by themselves, for test_gpu_dense_eig_kernels.py and
// test_dense_eig_rule.py.
#include "k_dense_eig.cu"

extern "C" int block_columns(int n) {
  size_t smem = 0;
  return wtb::bt_columns(n, &smem);
}

// v: n complex per column (row r of v_j at v[j * n + r], rows j + 2 on read; quantised in place), ncol columns; tau: n - 1;
// Zt: n x n, Z: n x n complex; the first `blocks` blocks of kc columns.
extern "C" int back_transform(wtb::zd* v, int n, int ncol, const wtb::zd* tau, int* exv, const double* Zt, wtb::zd* Z,
                              int kc, int in_smem, int blocks) {
  const size_t smem = in_smem ? (size_t)n * kc * sizeof(longlong2) : 0;
  if (kc < 1 || kc > 16 || smem > 200 * 1024 || ncol > n - 1 || (long)blocks > (n + kc - 1) / kc) return -1;
  cudaError_t e = wtb::raise_smem_limit(reinterpret_cast<const void*>(wtb::tri_backtransform_kernel), smem);
  if (e != cudaSuccess) return (int)e;
  wtb::tri_quantise_kernel<<<ncol, 256>>>(v, n, n, exv);
  wtb::tri_backtransform_kernel<<<blocks, wtb::kBtThreads, smem>>>(v, n, n, tau, exv, Zt, Z, 0, kc, in_smem);
  e = cudaGetLastError();
  return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
