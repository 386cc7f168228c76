// The FP64 projected eigenproblem by itself, for test_gpu_heev64_joint.py: nsys matrices of n x n, n * n apart.
#include "wtb_internal.h"
#include "solver.h"

extern "C" int heev64(const wtb::zd* A, int n, int nwant, int nsys, double* E, wtb::zd* V) {
  wtb::BatchMap bm;
  bm.nsys = nsys;
  const cudaError_t e = wtb::launch_heev_small<double>(A, n, nullptr, n, nwant, E, V, nwant, nullptr, bm, (long)n * n, nwant,
                                                       (long)n * nwant);
  return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
