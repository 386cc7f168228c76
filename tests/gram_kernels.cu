// The FP64 Grams by themselves, for test_gpu_gram64_order.py.
#include "wtb_internal.h"

extern "C" int gram64(const wtb::zd* A, int p, const wtb::zd* B, int q, int nrow, int npart, wtb::zd* out,
                      double* partial) {
  const cudaError_t e = wtb::launch_gram<double>(A, p, p, B, q, q, nrow, out, partial, npart, nullptr);
  return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}

extern "C" int gram_pair64(const wtb::zd* A, const wtb::zd* B, int p, int nrow, int npart, int upper, wtb::zd* M,
                           wtb::zd* G, double* partial) {
  const cudaError_t e = wtb::launch_gram_pair<double>(A, B, p, p, nrow, M, G, partial, npart, nullptr, wtb::BatchMap(), 0,
                                                      upper != 0);
  return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
