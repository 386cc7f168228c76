// Temperature BSE of bsesolvertemp and bsebndstemp (src/module_bse.F90:2649-3263, :1572-1990): the couplings
// weighted by the occupation difference f_v - f_c of the row's transition (fermidisteh, src/module_math.F90:407-421).
// matrizelbsetemp / matrizelbsekqtemp (src/module_bse.F90:575-660, :664-780) give
//   H(i,j) = C(i,j) f_i  (i != j),   H(i,i) = (E_c - E_v) + C(i,i) f_i
// with C the Coulomb part (direct, and at finite Q the exchange); the reference fills the upper triangle and
// ZHEEV 'U' reads its Hermitian completion, E(i,j) = D(i,j) f_min(i,j) with D the unweighted matrix.  Then the
// activities of dielbseptemp (src/module_bse.F90:784-810) for every exciton:
// Re[(sum_j A(j,n) h1(j)) conj(sum_j A(j,n) h2(j) f_j)].
#include <algorithm>

#include "wtb_internal.h"

namespace wtb {

namespace {

// f_v - f_c at temperature temp (K), Fermi level 0; kb is the single-precision literal 8.617330350E-5 and a zero
// temperature is read as 1E-8 (single precision), as fermidisteh does.
__global__ void fermi_weight_kernel(const double* __restrict__ eig_win, int nk, int nv, int nc, double temp,
                                    double* __restrict__ f) {
  const long I = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long dim = (long)nk * nc * nv;
  if (I >= dim) return;
  const int k = (int)(I / (nc * nv)), c = (int)((I / nv) % nc), v = (int)(I % nv);
  const int nb = nv + nc;
  const double ec = eig_win[(size_t)k * nb + nv + c], ev = eig_win[(size_t)k * nb + v];
  const double t = temp == 0.0 ? (double)1e-8f : temp;
  const double kb = (double)8.617330350E-5f;
  const double beta = 1.0 / (kb * t);
  const double fv = 1.0 / (exp(ev * beta) + 1.0);
  const double fc = 1.0 / (exp(ec * beta) + 1.0);
  f[I] = fv - fc;
}

// E = D f_min(i,j) off the diagonal, E(i,i) = dE_i + (D(i,i) - dE_i) f_i (the coupling part of the diagonal
// weighted: V(k_i,k_i) at Q = 0, V(k_i,k_i) - V(Q,0)|<c_i|v_i>|^2 for the finite-Q matrix of matrizelbsekqtemp),
// on the row-major dim x dim D in place.
__global__ void temp_weight_kernel(zd* __restrict__ H, long dim, const double* __restrict__ f,
                                   const double* __restrict__ dE) {
  const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= dim * dim) return;
  const long I = e / dim, J = e % dim;
  if (I == J) {
    H[e] = mk<double>(dE[I] + (H[e].re - dE[I]) * f[I], 0.0);
  } else {
    const double w = f[I < J ? I : J];
    H[e].re *= w;
    H[e].im *= w;
  }
}

// Per exciton n (column n of the row-major eigenvector matrix Z): s_a = sum_i Z(i,n) h_a(i) and
// t_a = sum_i Z(i,n) h_a(i) f_i for a = x y z sp sm, over the rows of chunk blockIdx.y, to part[chunk][20][dim]: the rows
// are split because dim threads alone leave the SMs idle (n = 1,520: 2.72 -> 0.28 ms).
__global__ void __launch_bounds__(128) temp_acts_partial_kernel(const zd* __restrict__ Z, int dim,
                                                                const zd* __restrict__ hr,
                                                                const double* __restrict__ f, int rows,
                                                                double* __restrict__ part) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= dim) return;
  zd s[5], t[5];
#pragma unroll
  for (int a = 0; a < 5; ++a) s[a] = t[a] = mk<double>(0.0, 0.0);
  const int i1 = min(dim, (int)(blockIdx.y + 1) * rows);
#pragma unroll 4
  for (int i = blockIdx.y * rows; i < i1; ++i) {
    const zd z = Z[(size_t)i * dim + n], zf = cscale(z, f[i]);
#pragma unroll
    for (int a = 0; a < 5; ++a) {
      const zd h = hr[(size_t)a * dim + i];
      cfma(s[a], z, h);
      cfma(t[a], zf, h);
    }
  }
  double* o = part + (size_t)blockIdx.y * 20 * dim + n;
#pragma unroll
  for (int a = 0; a < 5; ++a) {
    o[(size_t)(4 * a) * dim] = s[a].re;
    o[(size_t)(4 * a + 1) * dim] = s[a].im;
    o[(size_t)(4 * a + 2) * dim] = t[a].re;
    o[(size_t)(4 * a + 3) * dim] = t[a].im;
  }
}

// The chunks' sums in order, then the eight activities
// xx yy zz (s_a, t_a), xy (s_x, t_y), xz (s_x, t_z), yz (s_y, t_z), sp, sm; xy xz yz zero unless dtfull, sp sm
// zero unless cpol (the reference writes zeros then).
__global__ void __launch_bounds__(64) temp_acts_kernel(const double* __restrict__ part, int nchunk, int dim, int dtfull,
                                                       int cpol, double* __restrict__ acts) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= dim) return;
  double v[20];
#pragma unroll
  for (int q = 0; q < 20; ++q) v[q] = 0.0;
  for (int c = 0; c < nchunk; ++c)
#pragma unroll
    for (int q = 0; q < 20; ++q) v[q] += part[((size_t)c * 20 + q) * dim + n];
  auto re_prod = [&](int a, int b) { return v[4 * a] * v[4 * b + 2] + v[4 * a + 1] * v[4 * b + 3]; };  // Re(s conj(t))
  acts[0 * (size_t)dim + n] = re_prod(0, 0);
  acts[1 * (size_t)dim + n] = re_prod(1, 1);
  acts[2 * (size_t)dim + n] = re_prod(2, 2);
  acts[3 * (size_t)dim + n] = dtfull ? re_prod(0, 1) : 0.0;
  acts[4 * (size_t)dim + n] = dtfull ? re_prod(0, 2) : 0.0;
  acts[5 * (size_t)dim + n] = dtfull ? re_prod(1, 2) : 0.0;
  acts[6 * (size_t)dim + n] = cpol ? re_prod(3, 3) : 0.0;
  acts[7 * (size_t)dim + n] = cpol ? re_prod(4, 4) : 0.0;
}

// chunks of at least 32 rows, about eight CTAs an SM at most
int acts_chunks(int dim) {
  const int blocks = (dim + 127) / 128;
  return std::max(1, std::min((dim + 31) / 32, (152 * 8 + blocks - 1) / blocks));
}

}  // namespace

cudaError_t launch_fermi_weights(const double* eig_win, int nk, int nv, int nc, double temp, double* f,
                                 cudaStream_t s) {
  const long dim = (long)nk * nc * nv;
  fermi_weight_kernel<<<(unsigned)((dim + 255) / 256), 256, 0, s>>>(eig_win, nk, nv, nc, temp, f); ++g_launch_count;
  return cudaGetLastError();
}

cudaError_t launch_temp_weight(zd* H, long dim, const double* f, const double* dE, cudaStream_t s) {
  temp_weight_kernel<<<(unsigned)((dim * dim + 255) / 256), 256, 0, s>>>(H, dim, f, dE); ++g_launch_count;
  return cudaGetLastError();
}

size_t temp_acts_scratch(int dim) { return (size_t)acts_chunks(dim) * 20 * dim; }

cudaError_t launch_temp_acts(const zd* Z, int dim, const zd* hr, const double* f, int dtfull, int cpol, double* part,
                             double* acts, cudaStream_t s) {
  const int nchunk = acts_chunks(dim), rows = (dim + nchunk - 1) / nchunk;
  temp_acts_partial_kernel<<<dim3((dim + 127) / 128, nchunk), 128, 0, s>>>(Z, dim, hr, f, rows, part); ++g_launch_count;
  temp_acts_kernel<<<(dim + 63) / 64, 64, 0, s>>>(part, nchunk, dim, dtfull, cpol, acts); ++g_launch_count;
  return cudaGetLastError();
}

}  // namespace wtb
