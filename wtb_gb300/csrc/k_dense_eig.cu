// All eigenvalues of a dense Hermitian matrix on the device: the stand-in for the LAPACK ZHEEV calls of the
// full-spectrum paths (bsebnds, src/module_bse.F90:1427-1448; the temperature solver's dense path).
//
// 1. Householder tridiagonalisation A = Q T Q^H, lower form, blocked as LAPACK's zhetrd: within a panel of 32 columns
//    the trailing matrix is left as it was, a column is brought up to date from the panel's v and w, and its Hermitian
//    product is corrected by them; after the panel the trailing matrix takes all 32 rank-2 updates at once.  Two
//    launches a column (the Hermitian product by 64 x 64 lower tiles; x and the next column but for a multiple of v,
//    which the next product's loads subtract) and one a panel.  8/3 n^3 multiply-adds: on the FP64 pipe 62 ms at n = 2,304, so the Hermitian product and the trailing
//    update run as exact integer sums of quantised components (below), the rest in FP64.
// 2. Eigenvalues of the real symmetric tridiagonal T by bisection on Sturm counts, as multisection with a few lanes
//    per eigenvalue index where n alone would leave SMs idle, to the FP64 resolution of the Gershgorin interval.
//    Backward stable: |lambda - lambda_exact| <~ n eps ||A||.
#include <cooperative_groups.h>

#include <cfloat>

#include "wtb_internal.h"

namespace wtb {

namespace {

constexpr int kT = 64;    // tile edge of the Hermitian product and the trailing update (absolute tile grid)
constexpr int kNB = 32;   // reflectors a panel
constexpr int kQ = 55;    // bits of a quantised component
constexpr int kExpBad = 100000, kExpZero = -4096;

inline int tiles_of(int n) { return (n + kT - 1) / kT; }
inline size_t lower_tiles(int nT) { return (size_t)nT * (nT + 1) / 2; }

// Quantised arithmetic.  An FP64 warp instruction holds the SM's FP64 pipe for 19 clocks (1.7 lanes a clock), a 32 x 32 +
// 64-bit integer multiply-add for about 1.5, so the products of the reduction run as integers: a component x of a group
// with a common exponent, |x| < 2^ex, is the integer q = rint(x 2^(55 - ex)) = hi 2^28 + lo, |hi| <= 2^27,
// |lo| <= 2^27, and a product takes three multiply-adds (hi hi; hi lo + lo hi; lo lo is below 2^-56 of the largest).
// Every sum of a tile is exact in 64 bits (at most 128 products of 2^54), so the only errors are those of q, 2^-56 of
// the group's largest component, eight times below FP64's own rounding of one product of that size.
__device__ __forceinline__ int exponent_of(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }  // biased

// the biased exponent field of the group's largest component -> ex with |x| < 2^ex
__device__ __forceinline__ int group_ex(int field) {
  return field == 0x7ff ? kExpBad : field == 0 ? kExpZero : field - 1022;
}
__device__ __forceinline__ int2 quantise(double x, int ex) {
  const long long b = __double_as_longlong(x);
  const int f = (int)((b >> 52) & 0x7ff);
  long long m = (b & 0xfffffffffffffll) | 0x10000000000000ll;  // x = m 2^(f - 1075)
  const int sh = f - 1075 + kQ - ex;                            // <= 2 for |x| < 2^ex
  if (f == 0 || ex >= kExpBad || sh < -54) return make_int2(0, 0);
  if (sh >= 0)
    m <<= sh;
  else
    m = (m + (1ll << (-sh - 1))) >> -sh;
  if (b < 0) m = -m;
  const int hi = (int)((m + (1ll << 27)) >> 28);
  return make_int2(hi, (int)(m - ((long long)hi << 28)));
}
__device__ __forceinline__ int4 quantise(zd x, int ex) {
  const int2 r = quantise(x.re, ex), i = quantise(x.im, ex);
  return make_int4(r.x, r.y, i.x, i.y);
}
// 2^e (0 below the range, infinity above; NaN for a group with a component that is not finite)
__device__ __forceinline__ double pow2(int e) {
  if (e > kExpBad / 2) return __longlong_as_double(0x7ff8000000000000ll);
  return scalbn(1.0, e);
}
// an exact sum of products hh 2^56 + cr 2^28 of groups with exponents adding to e, as a double
// (2^28 alone may lie below the range of doubles where 2^56 does not; for products near its end s56 is 2^60 too large
// and the sum, at least 2^-28 or zero, is taken down before it, by its exponent field)
__device__ __forceinline__ double from_sums(long long hh, long long cr, double s56, bool down) {
  double t = fma((double)cr, 0x1p-28, (double)hh);
  if (down && t != 0.0) t = __hiloint2double(__double2hiint(t) - (60 << 20), __double2loint(t));
  return t * s56;
}
__device__ __forceinline__ void mac(long long& hh, long long& cr, int ah, int al, int bh, int bl) {
  hh += (long long)ah * bh;
  cr += (long long)ah * bl;
  cr += (long long)al * bh;
}

// zlarfg for x = A(j+1:n, j): returns tau, beta and the scale 1/(alpha - beta) applied to x(2:m).  By one warp, the four
// quotients on four lanes (a division is a chain of 460 clocks).
struct Reflector {
  zd tau, scale;
  double beta;
};

__device__ __forceinline__ Reflector make_reflector(zd alpha, double xnorm2) {
  Reflector r;
  if (xnorm2 == 0.0 && alpha.im == 0.0) {
    r.tau = mk<double>(0.0, 0.0);
    r.scale = mk<double>(0.0, 0.0);
    r.beta = alpha.re;
    return r;
  }
  const int lane = threadIdx.x & 31;
  const double nrm = sqrt(alpha.re * alpha.re + alpha.im * alpha.im + xnorm2);
  const double beta = alpha.re >= 0.0 ? -nrm : nrm;
  r.beta = beta;
  const double dr = alpha.re - beta, di = alpha.im;
  const double den = dr * dr + di * di;
  // tau = (beta - alpha) / beta, 1 / (alpha - beta) = conj(alpha - beta) / den
  const double q = (lane & 1 ? -di : lane & 2 ? dr : -dr) / (lane & 2 ? den : beta);
  r.tau = mk<double>(__shfl_sync(0xffffffffu, q, 0), __shfl_sync(0xffffffffu, q, 1));
  r.scale = mk<double>(__shfl_sync(0xffffffffu, q, 2), __shfl_sync(0xffffffffu, q, 3));
  return r;
}

// Tile (R, C), R >= C, of the lower triangle of an nT x nT tile grid from the linear index b.
__device__ __forceinline__ void lower_tile(int b, int* R, int* C) {
  int r = (int)((sqrtf(8.0f * (float)b + 1.0f) - 1.0f) * 0.5f);  // FP32 guess, corrected exactly below
  while ((r + 1) * (r + 2) / 2 <= b) ++r;
  while (r * (r + 1) / 2 > b) --r;
  *R = r;
  *C = b - r * (r + 1) / 2;
}

// The column's reflector, what K1's first CTA leaves for K2: om = 1 - sc x1, v = sc x + om e_1 for x = A(j+1:n, j),
// x1 = x's first entry.
struct TriCol {
  zd tau, sc, om, x1;
};

// Programmatic dependent launch: a kernel's CTAs start once every CTA of the one before has called launch_next, and
// wait_previous returns once that kernel has completed.  What that kernel writes changes while this one runs, so no
// pointer of K1, K2 and the functions they call is restrict: such a pointer's loads may be taken from the read-only path
// or moved above the wait.
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// alpha = -(tau/2) sum_b dots[b], the sum split over one warp's lanes in a fixed order.
__device__ __forceinline__ zd her2_alpha(const zd* dots, int ndots, zd tau) {
  zd d = mk<double>(0.0, 0.0);
  for (int b = threadIdx.x & 31; b < ndots; b += 32) d = cadd(d, dots[b]);
  for (int o = 16; o > 0; o >>= 1) {
    d.re += __shfl_xor_sync(0xffffffffu, d.re, o);
    d.im += __shfl_xor_sync(0xffffffffu, d.im, o);
  }
  return cscale(cmul(tau, d), -0.5);
}

// a summed over each half warp, the two components' sums shared out over its lanes: 4 FP64 adds instead of 8.
__device__ __forceinline__ zd half_warp_sum(zd a) {
  const int lane = threadIdx.x & 31;
  const bool im = lane & 8;
  double t = (im ? a.im : a.re) + __shfl_xor_sync(0xffffffffu, im ? a.re : a.im, 8);
  for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  const int base = lane & 16;
  return mk<double>(__shfl_sync(0xffffffffu, t, base), __shfl_sync(0xffffffffu, t, base + 8));
}

constexpr int kRows = 8;     // rows of a CTA of K2, 16 lanes each
constexpr int kDotRows = 512;  // rows of x whose products with one v and w take one CTA of K1
constexpr int kNextRows = 16;  // rows of the next column of a CTA of K1

// K1, column j = j0 + i.  The column brought up to date is x = A(j:n, j) for i = 0, else u - s v_{j-1}, with u and
// the parts of s = 2 Re alpha, alpha = -(tau/2) x_w^H v, from K2 of the column before (w_{j-1} = x_w + alpha v_{j-1}
// has w_{j-1}(j) = x_w(j) + alpha and v_{j-1}(j) = 1).  No scaling of the reflector yet: A v = sc A x + om A(:, j+1).
//   CTA 0: x into column j, the reflector's tau, beta, sc and om.  The next i nch: v_l^H x and w_l^H x over 512 rows
//   each (an SM issues an FP64 instruction every 19 clocks: over all 2,304 rows they outlasted the tiles), the last
//   l's also w_{j-1}.  The next nnext: next(r) = A(r, j+1) - sum_{l < i} (v_l(r) conj(w_l(j+1)) + w_l(r) conj(v_l(j+1)))
//   over 16 rows each, for K2 (FP64 work beside the tiles' integer work; in K2 it took 2 to 3 us).
//   The others, one per lower tile (R, C) of the trailing block: the quantised strict lower triangle's A_RC x_C to
//   the rows of block R and A_RC^H x_R to the rows of block C, as P[other block][row] (a diagonal tile's second
//   product as P[nT][row]), each (slot, row) written once.  A thread sums one row (or column) over a quarter of the
//   tile.  Large trailing blocks are bound by the integer multiply-adds (18 an element) and the tiles' way from L2: 17 us
//   at m = 2,304 where the FP64 product took 55; small ones by the chain of waits and FP64 sums, 7 to 9 us; 11.9 us
//   averaged over the columns of n = 2,304 (14.1 with four real products, two CTAs an SM and one CTA per v and w).
//   Within a panel the tiles' elements are on their way before the kernel before has finished.
__global__ void __launch_bounds__(256, 3) tri_symv_kernel(zd* A, int n, int lda, int j, int i,
                                                       zd* W, const zd* u,
                                                       const zd* xw, const zd* dots,
                                                       const double* sparts, int ndots,
                                                       const int4* Aq, const int* Aex,
                                                       TriCol* col, zd* tau_out,
                                                       double* e_out, zd* g, int nch,
                                                       zd* next, int nnext, zd* P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double s_s;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const zd* vp = A + (size_t)(j - 1) * lda;  // v_{j-1} by absolute row, read for i > 0 only
  auto load_s = [&]() {
    if (i > 0 && warp == 0) {
      double t = 0.0;
      for (int b = lane; b < ndots; b += 32) t += sparts[b];
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == 0) s_s = t;
    }
    __syncthreads();
    return i > 0 ? s_s : 0.0;
  };
  auto x_at = [&](int r, double s) {
    if (i == 0) return A[(size_t)j * lda + r];
    const zd ur = u[r], vr = vp[r];
    return mk<double>(fma(-s, vr.re, ur.re), fma(-s, vr.im, ur.im));
  };
  const int ndot = i * nch;
  if ((int)blockIdx.x > ndot && (int)blockIdx.x <= ndot + nnext) {
    __shared__ zd s_al, vj[kNB], wj[kNB];
    const int l16 = tid & 15, r = j + 1 + ((int)blockIdx.x - ndot - 1) * kNextRows + tid / 16, j0 = j - i;
    wait_previous();
    launch_next();
    if (warp == 0 && i > 0) {
      const zd al = her2_alpha(dots, ndots, tau_out[j - 1]);
      if (tid == 0) s_al = al;
    }
    zd v[2], w[2], a = mk<double>(0.0, 0.0);
    if (r < n) a = A[(size_t)(j + 1) * lda + r];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int l = l16 + 16 * h;
      v[h] = w[h] = mk<double>(0.0, 0.0);
      if (r < n && l < i) {
        v[h] = A[(size_t)(j0 + l) * lda + r];
        w[h] = l < i - 1 ? W[(size_t)l * n + r] : xw[r];
      }
    }
    __syncthreads();
    if (tid < i) {
      const zd v1 = A[(size_t)(j0 + tid) * lda + j + 1];
      zd w1 = tid < i - 1 ? W[(size_t)tid * n + j + 1] : xw[j + 1];
      if (tid == i - 1) cfma(w1, s_al, v1);
      vj[tid] = v1;
      wj[tid] = w1;
    }
    __syncthreads();
    zd t = mk<double>(0.0, 0.0);
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (16 * h < i) {  // uniform
        const int l = l16 + 16 * h;
        if (l == i - 1) cfma(w[h], s_al, v[h]);
        if (l < i) {
          cfmac(t, wj[l], v[h]);
          cfmac(t, vj[l], w[h]);
        }
      }
    t = half_warp_sum(t);
    if (l16 == 0 && r < n) next[r] = mk<double>(a.re - t.re, r == j + 1 ? 0.0 : a.im - t.im);
    return;
  }
  if ((int)blockIdx.x <= ndot) {
    wait_previous();
    launch_next();
    const double s = load_s();
    zd* red = reinterpret_cast<zd*>(smem_raw);
    if (blockIdx.x == 0) {
      double t = 0.0;
      __shared__ zd s_x1;
      for (int r = j + tid; r < n; r += 256) {
        zd x = x_at(r, s);
        if (r == j) x.im = 0.0;
        if (r == j + 1) s_x1 = x;
        if (r > j + 1) t = fma(x.re, x.re, fma(x.im, x.im, t));
        if (i > 0 || r == j) A[(size_t)j * lda + r] = x;
      }
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      double* rd = reinterpret_cast<double*>(smem_raw);
      if (lane == 0) rd[warp] = t;
      __syncthreads();
      if (warp == 0 && j + 1 < n) {
        t = rd[lane & 7];
        for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        const zd x1 = s_x1;
        const Reflector R = make_reflector(x1, t);
        if (lane == 0) {
          tau_out[j] = R.tau;
          e_out[j] = R.beta;
          col->tau = R.tau;
          col->sc = R.scale;
          const zd sa = cmul(R.scale, x1);
          col->om = mk<double>(1.0 - sa.re, -sa.im);
          col->x1 = x1;
        }
      }
      return;
    }
    const int ch = (blockIdx.x - 1) % nch, l = (blockIdx.x - 1) / nch;
    const zd* v = A + (size_t)(j - i + l) * lda;
    zd* w = W + (size_t)l * n;
    const bool fresh = l == i - 1;  // w_{j-1} is still x_w + alpha v_{j-1}
    zd alpha = mk<double>(0.0, 0.0);
    if (fresh) {
      if (warp == 0) {
        const zd al = her2_alpha(dots, ndots, tau_out[j - 1]);
        if (tid == 0) red[0] = al;
      }
      __syncthreads();
      alpha = red[0];
      __syncthreads();  // red is written again below
    }
    zd gv = mk<double>(0.0, 0.0), gw = gv;
    for (int r = j + 1 + ch * kDotRows + tid; r < min(n, j + 1 + (ch + 1) * kDotRows); r += 256) {
      const zd x = x_at(r, s), vr = v[r];
      zd wr;
      if (fresh) {
        wr = xw[r];
        cfma(wr, alpha, vr);
        w[r] = wr;
      } else {
        wr = w[r];
      }
      cfmac(gv, vr, x);
      cfmac(gw, wr, x);
    }
    for (int o = 16; o > 0; o >>= 1) {
      gv.re += __shfl_xor_sync(0xffffffffu, gv.re, o);
      gv.im += __shfl_xor_sync(0xffffffffu, gv.im, o);
      gw.re += __shfl_xor_sync(0xffffffffu, gw.re, o);
      gw.im += __shfl_xor_sync(0xffffffffu, gw.im, o);
    }
    if (lane == 0) {
      red[2 * warp] = gv;
      red[2 * warp + 1] = gw;
    }
    __syncthreads();
    if (tid < 2) {
      zd t = red[tid];
      for (int q = 1; q < 8; ++q) t = cadd(t, red[2 * q + tid]);
      g[ch * 2 * kNB + 2 * l + tid] = t;
    }
    return;
  }
  constexpr int kPad = kT + 1;                       // conflict-free columns and rows
  int4* tile = reinterpret_cast<int4*>(smem_raw);    // [column][row]
  int4* xa = tile + kT * kPad;                       // rows' 64 entries of x, then the columns': re, im - re
  int2* xb = reinterpret_cast<int2*>(xa + 2 * kT);   // re + im
  long long* sums = reinterpret_cast<long long*>(smem_raw);  // [2][4 quarters][4][kT], over the tile once it is used
  const int nT = (n + kT - 1) / kT, C0 = (j + 1) / kT;
  int R, C;
  lower_tile(blockIdx.x - ndot - nnext - 1, &R, &C);
  R += C0;
  C += C0;
  const size_t t = (size_t)R * (R + 1) / 2 + C;
  const int4* src = Aq + t * kT * kT;
  // Aq was written by the panel's update: for i > 0 at least two kernels ago, complete before the one before this
  // could start it
  if (i == 0) wait_previous();
  for (int e = tid; e < kT * kT; e += 256)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(tile + (e / kT) * kPad + e % kT)),
                 "l"(src + e)
                 : "memory");
  asm volatile("cp.async.commit_group;" ::: "memory");
  if (i > 0) wait_previous();
  launch_next();
  __shared__ int s_f[4];  // largest exponent fields of x over the halves of the two blocks
  zd z = mk<double>(0.0, 0.0), zv = z;
  if (tid < 2 * kT) {
    const int r = (tid < kT ? R : C) * kT + tid % kT;
    if (r > j && r < n) {
      z = i == 0 ? A[(size_t)j * lda + r] : u[r];
      if (i > 0) zv = vp[r];
    }
  }
  const double s = load_s();
  if (tid < 2 * kT) {
    if (i > 0) z = mk<double>(fma(-s, zv.re, z.re), fma(-s, zv.im, z.im));
    const int f = __reduce_max_sync(0xffffffffu, max(exponent_of(z.re), exponent_of(z.im)));
    if (lane == 0) s_f[warp] = f;
  }
  __syncthreads();
  const int exR = group_ex(max(s_f[0], s_f[1])), exC = group_ex(max(s_f[2], s_f[3]));
  if (tid < 2 * kT) {
    const int4 q = quantise(z, tid < kT ? exR : exC);
    xa[tid] = make_int4(q.x, q.y, q.z - q.x, q.w - q.y);
    xb[tid] = make_int2(q.x + q.z, q.y + q.w);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  const int row = tid % kT, q0 = (tid / kT) * (kT / 4);
  // a complex product by three real ones (all exact, so the sums are those of four): with s = b.re (a.re + a.im),
  // a b = s - a.im (b.re + b.im) + i (s + a.re (b.im - b.re)), and conj(a) b the same with -a.im
  long long o[2][4];
#pragma unroll
  for (int second = 0; second < 2; ++second) {
    long long sh = 0, sl = 0, ph = 0, pl = 0, mh = 0, ml = 0;
    if (!second) {
#pragma unroll 4
      for (int c = q0; c < q0 + kT / 4; ++c) {
        const int4 a = tile[c * kPad + row], b = xa[kT + c];
        const int2 p = xb[kT + c];
        mac(sh, sl, a.x + a.z, a.y + a.w, b.x, b.y);
        mac(ph, pl, a.z, a.w, p.x, p.y);
        mac(mh, ml, a.x, a.y, b.z, b.w);
      }
      ph = -ph;
      pl = -pl;
    } else {
#pragma unroll 4
      for (int r = q0; r < q0 + kT / 4; ++r) {
        const int4 a = tile[row * kPad + r], b = xa[r];
        const int2 p = xb[r];
        mac(sh, sl, a.x - a.z, a.y - a.w, b.x, b.y);
        mac(ph, pl, a.z, a.w, p.x, p.y);
        mac(mh, ml, a.x, a.y, b.z, b.w);
      }
    }
    o[second][0] = sh + ph;
    o[second][1] = sl + pl;
    o[second][2] = sh + mh;
    o[second][3] = sl + ml;
  }
  __syncthreads();
#pragma unroll
  for (int second = 0; second < 2; ++second)
#pragma unroll
    for (int c = 0; c < 4; ++c) sums[((second * 4 + tid / kT) * 4 + c) * kT + row] = o[second][c];
  __syncthreads();
  const int second = tid / kT, out = (second ? C : R) * kT + row;
  if (tid < 2 * kT && out < n) {
    const int e56 = Aex[t] + (second ? exR : exC) - 2 * kQ + 56;
    const bool down = e56 < -960 && e56 > -1200;
    const double s56 = pow2(e56 + (down ? 60 : 0));
    const long long* q = sums + second * 16 * kT + row;
    long long v[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) v[c] = (q[c * kT] + q[(4 + c) * kT]) + (q[(8 + c) * kT] + q[(12 + c) * kT]);
    const int slot = second ? (R == C ? nT : R) : C;
    P[(size_t)slot * n + out] = mk<double>(from_sums(v[0], v[1], s56, down), from_sums(v[2], v[3], s56, down));
  }
}

// K2: x_w = tau (A v - sum_l v_l (w_l^H v) + w_l (v_l^H v)) with A v = sc (P + diag x) + om A(:, j+1), v into column
// j, the parts of conj(x_w) v and of -Re(tau conj(x_w) v) by CTA, and, unless column j ends its panel (next null), of
// the next column
//   u = next - v conj(x_w(j+1)) - x_w,
// with x_w(j+1) formed by every CTA for itself (a ninth row).  FP64 instructions hold the pipe whatever the number of
// lanes that take part, so the sums over lanes are shared out (half_warp_sum) and the nine rows' remaining arithmetic
// is done by nine lanes of one warp.  7.1 us averaged over the columns of n = 2,304 (8.1 with the sums of next formed
// here); the two kernels took the place of three (32 us a column) that brought the next column up to date by
// themselves: n = 2,304 84 -> 71 ms, and 65 with both as they are.
__global__ void __launch_bounds__(16 * (kRows + 2)) tri_x_kernel(zd* A, int n, int lda, int j, int i,
                                                                 const zd* next,
                                                                 const zd* W,
                                                                 const zd* P,
                                                                 const TriCol* col,
                                                                 const zd* g, int nch,
                                                                 zd* u,
                                                                 zd* xw, zd* dots,
                                                                 double* sparts) {
  __shared__ zd gv[kNB], gw[kNB], sx[kRows + 1];
  const int tid = threadIdx.x, lane = tid & 15, half = tid / 16, j0 = j - i;
  wait_previous();
  launch_next();
  const zd tau = col->tau, sc = col->sc, om = col->om;
  if (tid < 2 * i) {
    const int l = tid >> 1;
    const zd at = (tid & 1) ? W[(size_t)l * n + j + 1] : A[(size_t)(j0 + l) * lda + j + 1];
    zd gs = g[tid];
    for (int c = 1; c < nch; ++c) gs = cadd(gs, g[c * 2 * kNB + tid]);
    zd t = cmul(sc, gs);
    cfma(t, om, cconj(at));
    ((tid & 1) ? gw : gv)[l] = t;  // v_l^H v, w_l^H v
  }
  const int nT = (n + kT - 1) / kT, C0 = (j + 1) / kT;
  auto row_of = [&](int h) { return h < kRows ? j + 1 + (int)blockIdx.x * kRows + h : h == kRows ? j + 1 : n; };
  const int r = row_of(half), q = row_of(tid <= kRows ? tid : kRows + 1);
  zd x = mk<double>(0.0, 0.0), a1 = x, un = x;
  double dg = 0.0;
  if (q < n) {  // for the last part, on their way meanwhile
    x = q == j + 1 ? col->x1 : A[(size_t)j * lda + q];  // CTA 0 overwrites row j + 1
    dg = A[(size_t)q * lda + q].re;
    a1 = A[(size_t)(j + 1) * lda + q];
    if (next) un = next[q];
  }
  zd y = mk<double>(0.0, 0.0);
  if (r < n)
    for (int t = C0 + lane; t <= nT; t += 16) y = cadd(y, P[(size_t)t * n + r]);
  __syncthreads();
  zd acc = mk<double>(0.0, 0.0);
  if (r < n) {
    acc = cmul(sc, y);
    for (int l = lane; l < i; l += 16) {
      const zd v = A[(size_t)(j0 + l) * lda + r], w = W[(size_t)l * n + r];
      cfma(acc, mk<double>(-v.re, -v.im), gw[l]);
      cfma(acc, mk<double>(-w.re, -w.im), gv[l]);
    }
  }
  acc = half_warp_sum(acc);
  if (lane == 0 && half <= kRows) sx[half] = acc;
  __syncthreads();
  if (tid >= 32) return;
  zd xr = mk<double>(0.0, 0.0), v = xr, d = xr;
  if (q < n) {
    acc = sx[tid];
    if (q == j + 1) a1.im = 0.0;
    v = q == j + 1 ? mk<double>(1.0, 0.0) : cmul(sc, x);
    cfma(acc, sc, cscale(x, dg));
    cfma(acc, om, a1);
    xr = cmul(tau, acc);
  }
  const zd x1 = mk<double>(__shfl_sync(0xffffffffu, xr.re, kRows), __shfl_sync(0xffffffffu, xr.im, kRows));
  if (q < n && tid < kRows) {
    xw[q] = xr;
    A[(size_t)j * lda + q] = v;
    if (next) {
      zd un1 = csub(un, xr);
      cfma(un1, mk<double>(-v.re, -v.im), cconj(x1));
      u[q] = un1;
    }
    d = cmulc(xr, v);
  }
  for (int o = kRows / 2; o > 0; o >>= 1) {
    d.re += __shfl_xor_sync(0xffffffffu, d.re, o);
    d.im += __shfl_xor_sync(0xffffffffu, d.im, o);
  }
  if (tid == 0) {
    dots[blockIdx.x] = d;
    sparts[blockIdx.x] = -cmul(tau, d).re;
  }
}

// After a panel (columns j1 - 32 .. j1 - 1): A(r, c) -= sum_l v_l(r) conj(w_l(c)) + w_l(r) conj(v_l(c))
// for r >= c >= j1, one cluster of two CTAs per 64 x 64 tile (32 columns each: one CTA's time is 80 us for the last
// tiles), the products quantised, then the tile's own quantised form (strict lower triangle) for the next panel's
// Hermitian products, on the larger exponent of the two.  reflectors = 0: only that.  512 threads, 4 entries each.  A complex
// product a conj(b) takes three real ones: with s = b.re (a.re + a.im), it is s - a.im (b.re - b.im)
// + i (s - a.re (b.re + b.im)), all exact.  Bound by the integer multiply-adds (576 an entry), 9 of a
// CTA's 39 us its loads and the quantising: 350 us at m = 2,240, where four real products on whole tiles took 399 and 32
// FP64 rank-2 updates 1.6 ms; averaged over the panels of n = 2,304 176 -> 148 us.
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(512, 1)
    tri_update_kernel(zd* __restrict__ A, int n, int lda, int j1, int reflectors, const zd* __restrict__ tau,
                      const zd* __restrict__ W, const zd* __restrict__ xw, const zd* __restrict__ dots, int ndots,
                      int4* __restrict__ Aq, int* __restrict__ Aex) {
  namespace cg = cooperative_groups;
  cg::cluster_group clu = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int kH = kT / 2;
  int4* vR = reinterpret_cast<int4*>(smem_raw);  // [kNB][kT] each
  int4* wR = vR + kNB * kT;
  int4* vC = wR + kNB * kT;  // [kNB][kH] each
  int4* wC = vC + kNB * kH;
  __shared__ zd s_alpha;
  __shared__ int s_exv, s_exw, s_ext;
  const int tid = threadIdx.x, C0 = j1 / kT, c0 = (blockIdx.x & 1) * kH;
  int R, C;
  lower_tile(blockIdx.x / 2, &R, &C);
  R += C0;
  C += C0;
  if (tid == 0) s_exv = s_exw = s_ext = 0;
  if (reflectors && tid < 32) {
    const zd al = her2_alpha(dots, ndots, tau[j1 - 1]);
    if (tid == 0) s_alpha = al;
  }
  __syncthreads();
  const int tr = tid % 16, tc = tid / 16;
  long long rh[4], rc[4], ih[4], ic[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) rh[e] = rc[e] = ih[e] = ic[e] = 0;
  double scale = 0.0;
  if (reflectors) {
    // v and w of the tile's rows, then of its columns: all loads in flight at once, quantised once the largest exponent
    // is known
    constexpr int kG = kT + kH, kE = kG * kNB / 512;
    auto at = [&](int rr) { return rr < kT ? R * kT + rr : C * kT + c0 + rr - kT; };
    zd v[kE], w[kE];
#pragma unroll
    for (int q = 0; q < kE; ++q) {
      const int e = tid + 512 * q, l = e / kG, r = at(e % kG);
      v[q] = w[q] = mk<double>(0.0, 0.0);
      if (r >= j1 && r < n) {
        v[q] = A[(size_t)(j1 - kNB + l) * lda + r];
        w[q] = l < kNB - 1 ? W[(size_t)l * n + r] : xw[r];
      }
    }
    int fv = 0, fw = 0;
    const zd alpha = s_alpha;
#pragma unroll
    for (int q = 0; q < kE; ++q) {
      if ((tid + 512 * q) / kG == kNB - 1) cfma(w[q], alpha, v[q]);  // still x - (tau/2)(x^H v) v
      fv = max(fv, max(exponent_of(v[q].re), exponent_of(v[q].im)));
      fw = max(fw, max(exponent_of(w[q].re), exponent_of(w[q].im)));
    }
    fv = __reduce_max_sync(0xffffffffu, fv);
    fw = __reduce_max_sync(0xffffffffu, fw);
    if ((tid & 31) == 0) {
      atomicMax(&s_exv, fv);
      atomicMax(&s_exw, fw);
    }
    __syncthreads();
    const int exv = group_ex(s_exv), exw = group_ex(s_exw);
#pragma unroll
    for (int q = 0; q < kE; ++q) {
      const int e = tid + 512 * q, l = e / kG, rr = e % kG;
      *(rr < kT ? wR + l * kT + rr : wC + l * kH + rr - kT) = quantise(w[q], exw);
      *(rr < kT ? vR + l * kT + rr : vC + l * kH + rr - kT) = quantise(v[q], exv);
    }
    __syncthreads();
    long long sh[4], sl[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) sh[e] = sl[e] = 0;
    auto product = [&](int e, const int4& a, const int2& as, const int4& b, const int2& bd, const int2& bs) {
      mac(sh[e], sl[e], as.x, as.y, b.x, b.y);
      mac(rh[e], rc[e], a.z, a.w, bd.x, bd.y);
      mac(ih[e], ic[e], a.x, a.y, bs.x, bs.y);
    };
    auto sum = [](const int4& a) { return make_int2(a.x + a.z, a.y + a.w); };
    auto dif = [](const int4& a) { return make_int2(a.x - a.z, a.y - a.w); };
    for (int l = 0; l < kNB; ++l) {
      const int4 v2 = vC[l * kH + tc], w2 = wC[l * kH + tc];
      const int2 vs = sum(v2), vd = dif(v2), ws = sum(w2), wd = dif(w2);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int4 v = vR[l * kT + tr + 16 * e], w = wR[l * kT + tr + 16 * e];
        product(e, v, sum(v), w2, wd, ws);
        product(e, w, sum(w), v2, vd, vs);
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      rh[e] = sh[e] - rh[e];
      rc[e] = sl[e] - rc[e];
      ih[e] = sh[e] - ih[e];
      ic[e] = sl[e] - ic[e];
    }
    scale = pow2(exw + exv - 2 * kQ + 56);
  }
  // the new entries, and the tile's largest exponent off the diagonal
  zd a[4];
  int f = 0;
  const int c = C * kT + c0 + tc;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int r = R * kT + tr + 16 * e;
    a[e] = mk<double>(0.0, 0.0);
    if (r < n && c >= j1 && r >= c) {
      zd* p = A + (size_t)c * lda + r;
      a[e] = *p;
      if (reflectors) {  // the low sums carried into the high ones, rounded at 2^-54 of the largest product
        const long long hr = rh[e] + ((rc[e] + (1ll << 27)) >> 28), hi = ih[e] + ((ic[e] + (1ll << 27)) >> 28);
        a[e].re = fma(-(double)hr, scale, a[e].re);
        a[e].im = r == c ? 0.0 : fma(-(double)hi, scale, a[e].im);
        *p = a[e];
      }
      if (r == c)
        a[e] = mk<double>(0.0, 0.0);
      else
        f = max(f, max(exponent_of(a[e].re), exponent_of(a[e].im)));
    }
  }
  f = __reduce_max_sync(0xffffffffu, f);
  if ((tid & 31) == 0) atomicMax(&s_ext, f);
  clu.sync();
  const int ex = group_ex(max(s_ext, *clu.map_shared_rank(&s_ext, clu.block_rank() ^ 1)));
  const size_t t = (size_t)R * (R + 1) / 2 + C;
  if (tid == 0 && c0 == 0) Aex[t] = ex;
#pragma unroll
  for (int e = 0; e < 4; ++e) Aq[t * kT * kT + (c0 + tc) * kT + tr + 16 * e] = quantise(a[e], ex);
  clu.sync();  // the peer has read s_ext
}

// A(j,i) = conj(A(i,j)) for i < j (the upper triangle is the input, as ZHEEV 'U' reads it); real diagonal.
__global__ void mirror_upper_kernel(zd* __restrict__ A, int n, int lda) {
  const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long)n * n) return;
  const int i = (int)(e % n), j = (int)(e / n);  // element (i, j), column-major
  if (i > j) A[(size_t)j * lda + i] = cconj(A[(size_t)i * lda + j]);
  else if (i == j) A[(size_t)j * lda + i].im = 0.0;
}

// d(i) = Re A(i,i); Gershgorin bounds and scale of T (one CTA).
__global__ void __launch_bounds__(1024) tri_finish_kernel(const zd* __restrict__ A, int n, int lda,
                                                          double* __restrict__ d, const double* __restrict__ e,
                                                          double* __restrict__ bounds) {
  double lo = INFINITY, hi = -INFINITY;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double di = A[(size_t)i * lda + i].re;
    d[i] = di;
    const double el = i > 0 ? fabs(e[i - 1]) : 0.0, er = i < n - 1 ? fabs(e[i]) : 0.0;
    lo = fmin(lo, di - el - er);
    hi = fmax(hi, di + el + er);
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  __shared__ double s_lo[32], s_hi[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    s_lo[warp] = lo;
    s_hi[warp] = hi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < (int)(blockDim.x >> 5); ++i) {
      lo = fmin(lo, s_lo[i]);
      hi = fmax(hi, s_hi[i]);
    }
    const double tnorm = fmax(fabs(lo), fabs(hi));
    // widen by a few ulps of the norm so that the end eigenvalues are strictly inside
    const double pad = 2.0 * (double)n * DBL_EPSILON * fmax(tnorm, 1e-300) + DBL_MIN;
    bounds[0] = lo - pad;
    bounds[1] = hi + pad;
    const int k = min(max(ilogb(fmax(fabs(bounds[0]), fabs(bounds[1]))) + 1, -1000), 1000);
    bounds[2] = scalbn(1.0, -k);  // T times this has entries and eigenvalues of at most 1
  }
}

// Number of eigenvalues of the scaled T below x: the sign changes of p_0 = 1, p_{i+1} = (d_i - x) p_i - e_{i-1}^2 p_{i-1}
// (the leading minors; Givens' recurrence, each p_i the exact one of a T whose entries differ by a few ulp).  One
// multiply-add of latency and three FP64 instructions a row, against a division's chain of 460 clocks and eleven
// instructions for the ratios q_i = p_{i+1} / p_i (all eigenvalues at n = 2,304: 20 -> 6.9 ms).  T is scaled to entries of at
// most 1.  A row takes the pair (p_i, p_{i-1}) up by at most two bits; every eighth row rescales it by a power of two.  A
// zero p_i counts as of the other sign than its predecessor (a zero pivot replaced by a small negative one) and goes on at
// the end of the range, far below a predecessor of an ordinary size.  Eight rows that leave the pair below 2^-900, after a
// zero without couplings or differences d_i - x of nearly nothing, are done again with zeros as -2^-110 of their
// predecessor and differences below 2^-54 as -2^-54 (T off by a quarter of an ulp of its norm): 110 bits a row at most.  (A
// zero of a size of its own beside a predecessor as small made the count wrong by one: a row of [[c, b], [b, a]] beside an
// uncoupled row c, at x = c.)
__device__ __forceinline__ int sturm_count(const double* __restrict__ d, const double* __restrict__ e2, int n,
                                           double x) {
  auto zero = [](double p) { return (__double_as_longlong(p) << 1) == 0; };
  auto pivot = [](double t) { return (__double2hiint(t) & 0x7fffffff) < (1023 - 54) << 20 ? -0x1p-54 : t; };
  double p0 = 1.0, p1 = pivot(d[0] - x);
  int cnt = (unsigned)__double2hiint(p1) >> 31;
  auto field = [&]() { return max((__double2hiint(p0) >> 20) & 0x7ff, (__double2hiint(p1) >> 20) & 0x7ff); };
  auto next = [&](double p) {
    cnt += (unsigned)(__double2hiint(p) ^ __double2hiint(p1)) >> 31;
    p0 = p1;
    p1 = p;
  };
  int e = field();
  for (int i0 = 1; i0 < n; i0 += 8) {
    const double sc = __hiloint2double((2046 - e) << 20, 0);  // 2^(1023 - e): the larger one to [1, 2)
    p0 *= sc;
    p1 *= sc;
    const double q0 = p0, q1 = p1;
    const int c0 = cnt, i1 = min(i0 + 8, n);
#pragma unroll 8
    for (int i = i0; i < i1; ++i) {
      const double p = fma(d[i] - x, p1, -(e2[i - 1] * p0));
      next(zero(p) ? __hiloint2double((__double2hiint(p1) & 0x80000000) ^ (int)0x80100000, 0) : p);  // -+ 2^-1022
    }
    e = field();
    if (e < 1023 - 900) {
      p0 = q0;
      p1 = q1;
      cnt = c0;
#pragma unroll 1
      for (int i = i0; i < i1; ++i) {
        const double p = fma(pivot(d[i] - x), p1, -(e2[i - 1] * p0));
        const int neg = __double2hiint(p1) ^ (int)0x80000000;
        next(zero(p) ? __hiloint2double(neg - (110 << 20), __double2loint(p1)) : p);
      }
      e = field();
    }
  }
  return cnt;
}

// The same in FP32, rescaled every fourth row (24 bits a row); a zero goes on as 2^-40, since these counts only say where
// to look first.
__device__ __forceinline__ int sturm_count(const float* __restrict__ d, const float* __restrict__ e2, int n, float x) {
  auto nonzero = [](float p, float before) {
    return p == 0.0f ? __int_as_float((__float_as_int(before) & 0x80000000) ^ (int)0xab800000) : p;  // -+ 2^-40
  };
  float p0 = 1.0f, p1 = nonzero(d[0] - x, 1.0f);
  int cnt = (unsigned)__float_as_int(p1) >> 31;
  for (int i0 = 1; i0 < n; i0 += 4) {
    const int e = max((__float_as_int(p0) >> 23) & 0xff, (__float_as_int(p1) >> 23) & 0xff);
    const float sc = __int_as_float(max(254 - e, 1) << 23);
    p0 *= sc;
    p1 *= sc;
    const int i1 = min(i0 + 4, n);
#pragma unroll 4
    for (int i = i0; i < i1; ++i) {
      const float p = nonzero(fmaf(d[i] - x, p1, -(e2[i - 1] * p0)), p1);
      cnt += (unsigned)(__float_as_int(p) ^ __float_as_int(p1)) >> 31;
      p0 = p1;
      p1 = p;
    }
  }
  return cnt;
}

// ds, e2: T scaled by the power of two that brings its Gershgorin interval to at most 1 in magnitude (bounds[2]), and
// both rounded to FP32
__global__ void tri_scale_kernel(const double* __restrict__ d, const double* __restrict__ e, int n,
                                 const double* __restrict__ bounds, double* __restrict__ ds, double* __restrict__ e2,
                                 float* __restrict__ dsf, float* __restrict__ e2f) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double s = bounds[2];
  ds[i] = d[i] * s;
  dsf[i] = (float)ds[i];
  if (i < n - 1) {
    const double es = e[i] * s;
    e2[i] = es * es;
    e2f[i] = (float)e2[i];
  }
}

// The k-th smallest eigenvalue (k = 0..n-1) by multisection with L lanes per k (L a power of two <= 32): the L
// lanes evaluate the Sturm count at L interior points of the bracket, which shrinks (L+1)-fold per pass, to the
// resolution 2 eps max|bound|.  The count is non-decreasing in x, so the points with count <= k form a prefix
// of the group and the new bracket is read off the ballot.  L = 1 is plain bisection (the fewest counts); the
// launcher raises L only until the GPU's SMs all have work, since a Sturm count queues on the SM's FP64 pipe.  Groups
// that have converged idle until their whole warp has.
// The first 20 bits come from FP32 counts of the rounded T (an FP32 instruction costs a sixtieth): their bracket,
// widened by 2^-18 for the rounding (entries of at most 1, each off by a few 2^-24), is only where the first FP64
// points lie, from its one end to the other inside the Gershgorin interval; the FP64 counts decide.  n = 1,520:
// 4.6 -> 3.8 ms, 2,304: 6.9 -> 5.4.
__global__ void __launch_bounds__(128) tri_multisect_kernel(const double* __restrict__ d,
                                                            const double* __restrict__ e2, int n,
                                                            const float* __restrict__ df,
                                                            const float* __restrict__ e2f,
                                                            const double* __restrict__ bounds,
                                                            double* __restrict__ W, int L) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const int k = tid / L, g = lane % L, base = lane - g;
  const unsigned gmask = L == 32 ? 0xffffffffu : (((1u << L) - 1u) << base);
  const double sc = bounds[2];
  double lo = bounds[0] * sc, hi = bounds[1] * sc;
  const double tol = 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi));
  bool done = k >= n;
  float lof = (float)lo, hif = (float)hi;
  for (int it = 0; it < 24; ++it) {
    const bool narrow = done || !(hif - lof > 0x1p-19f);
    if (__all_sync(0xffffffffu, narrow)) break;
    const float xf = lof + (hif - lof) / (float)(L + 1) * (float)(g + 1);
    const int cnt = narrow ? 0 : sturm_count(df, e2f, n, xf);
    const unsigned bal = __ballot_sync(0xffffffffu, !narrow && cnt <= k);
    const int nlo = __popc(bal & gmask);
    const float xlo = __shfl_sync(0xffffffffu, xf, base + max(nlo - 1, 0));
    const float xhi = __shfl_sync(0xffffffffu, xf, base + min(nlo, L - 1));
    if (!narrow) {
      lof = nlo > 0 ? xlo : lof;
      hif = nlo < L ? xhi : hif;
    }
  }
  const double first = (double)lof - 0x1p-18, last = (double)hif + 0x1p-18;
  const int nfirst = L > 1 ? 1 : 2;  // passes over the FP32 bracket
  for (int it = 0; it < 256; ++it) {
    if (!done && !(hi - lo > tol)) done = true;
    if (__all_sync(0xffffffffu, done)) break;
    const double h = (hi - lo) / (double)(L + 1);
    double x = lo + h * (double)(g + 1);
    if (it < nfirst) {
      x = L > 1 ? first + (last - first) / (double)(L - 1) * (double)g : it == 0 ? first : last;
      x = fmin(fmax(x, lo), hi);
    }
    const int cnt = done ? 0 : sturm_count(d, e2, n, x);
    const unsigned bal = __ballot_sync(0xffffffffu, !done && cnt <= k);
    const int nlo = __popc(bal & gmask);
    const double xlo = __shfl_sync(0xffffffffu, x, base + max(nlo - 1, 0));
    const double xhi = __shfl_sync(0xffffffffu, x, base + min(nlo, L - 1));
    if (!done) {
      const double nl = nlo > 0 ? xlo : lo;
      const double nh = nlo < L ? xhi : hi;
      if (nl == lo && nh == hi && it >= nfirst)
        done = true;  // no representable progress
      else {
        lo = nl;
        hi = nh;
      }
    }
  }
  if (k < n && g == 0) W[k] = 0.5 * (lo + hi) / sc;
}

// ----------------------------------------------------------------------------- eigenvectors
// Inverse iteration on T for every eigenvalue (dstein's method): Gaussian elimination with partial pivoting of
// T - lambda I, three solves from a deterministic start vector, each normalised.  Eigenvalues closer than
// 1e-7 ||T|| to their predecessor form a cluster, handled by one thread in order: later members are shifted
// apart by 10 eps ||T|| and reorthogonalised against the earlier ones after every solve (a degenerate pair
// then spans its eigenspace).  Outside clusters the vectors are orthogonal to eps ||T|| / gap <= 2e-9.
// One thread per cluster start; its scratch (6 arrays of n) is interleaved across the batch's threads so the
// row loops are coalesced.  Zt(i, k) = Zt[i * n + k] (row-major real).
// A thread's rows are one chain, so its latency is the time: the elimination carries its row in registers, the solves
// load eight rows of their operands before they use the first, one division a row (the pivot's reciprocal), and a CTA
// is one warp, so that the warps spread over the SMs.  n = 1,520: 11.2 -> 3.7 ms.
constexpr int kInvIters = 3;

// deterministic start entries in [-1, 1): splitmix64 of (k, i)
__device__ __forceinline__ double start_entry(unsigned long long k, unsigned long long i) {
  unsigned long long z = k * 0x9E3779B97F4A7C15ull + (i + 1) * 0xD1B54A32D192ED03ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return (double)(z >> 11) * (2.0 / 9007199254740992.0) - 1.0;
}

__global__ void __launch_bounds__(32) tri_invit_kernel(const double* __restrict__ d, const double* __restrict__ e,
                                                       int n, const double* __restrict__ W,
                                                       const double* __restrict__ bounds, int k0, int nb,
                                                       double* __restrict__ work, double* __restrict__ Zt) {
  constexpr int U = 8;  // rows whose operands are loaded together
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int k = k0 + t;
  if (t >= nb || k >= n) return;
  const double tnorm = fmax(fmax(fabs(bounds[0]), fabs(bounds[1])), DBL_MIN);
  const double ortol = 1e-7 * tnorm;
  if (k > 0 && W[k] - W[k - 1] < ortol) return;  // inside a cluster started by an earlier thread
  int kend = k + 1;
  while (kend < n && W[kend] - W[kend - 1] < ortol) ++kend;
  const size_t st = (size_t)nb;
  double* ra = work + t;             // reciprocal of the diagonal of U
  double* b = ra + (size_t)n * st;   // first superdiagonal of U
  double* dd = b + (size_t)n * st;   // second superdiagonal of U
  double* c = dd + (size_t)n * st;   // multipliers
  double* pv = c + (size_t)n * st;   // 1 where rows i, i+1 were swapped
  double* y = pv + (size_t)n * st;   // iterate
#define AT(arr, i) arr[(size_t)(i) * st]
  // Smaller pivots go on as +-tiny, which moves T by that much at one entry, another for every eigenvalue: at an ulp of the
  // norm it was the largest of the errors that turn two close eigenvalues' vectors towards one another (random n = 333,
  // exact shifts: ||Z^T Z - I|| 6.1e-14, with a sixteenth 3.0e-14, the same below).  Its reciprocal stays in range.
  const double tiny = fmax(0x1p-56 * tnorm, fmin(DBL_EPSILON * tnorm, DBL_MIN));
  double lam_prev = 0.0;
  for (int q = k; q < kend; ++q) {
    double lam = W[q];
    if (q > k && lam - lam_prev < 10.0 * DBL_EPSILON * tnorm) lam = lam_prev + 10.0 * DBL_EPSILON * tnorm;
    lam_prev = lam;
    // T - lam I = P L U, row i in (ai, bi)
    double ai = d[0] - lam, bi = n > 1 ? e[0] : 0.0;
    for (int i = 0; i < n; ++i) {
      const bool more = i + 1 < n;
      const double sub = more ? e[i] : 0.0;
      const double a1 = more ? d[i + 1] - lam : 0.0, b1 = i + 2 < n ? e[i + 1] : 0.0;
      const bool keep = fabs(ai) >= fabs(sub);
      double piv = keep ? ai : sub;
      if (fabs(piv) < tiny) piv = piv < 0.0 ? -tiny : tiny;
      const double rp = 1.0 / piv, m = (keep ? sub : ai) * rp;
      AT(ra, i) = rp;
      AT(c, i) = m;
      AT(pv, i) = keep ? 0.0 : 1.0;
      AT(b, i) = keep ? bi : a1;
      AT(dd, i) = keep ? 0.0 : b1;
      AT(y, i) = start_entry((unsigned long long)q, (unsigned long long)i);
      const double an = keep ? a1 - m * bi : bi - m * a1;
      bi = keep ? b1 : -m * b1;
      ai = an;
    }
    for (int it = 0; it < kInvIters; ++it) {
      double cur = AT(y, 0);
      for (int i0 = 0; i0 + 1 < n; i0 += U) {
        double cc[U], pp[U], yy[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int i = min(i0 + u, n - 2);
          cc[u] = AT(c, i);
          pp[u] = AT(pv, i);
          yy[u] = AT(y, i + 1);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (i0 + u + 1 < n) {
            const double first = pp[u] != 0.0 ? yy[u] : cur, second = pp[u] != 0.0 ? cur : yy[u];
            AT(y, i0 + u) = first;
            cur = second - cc[u] * first;
          }
      }
      AT(y, n - 1) = cur;
      double y1 = 0.0, y2 = 0.0, mx = 0.0;  // rows i + 1 and i + 2
      for (int i0 = n - 1; i0 >= 0; i0 -= U) {
        double aa[U], bb[U], ee[U], yy[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int i = max(i0 - u, 0);
          aa[u] = AT(ra, i);
          bb[u] = AT(b, i);
          ee[u] = AT(dd, i);
          yy[u] = AT(y, i);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (i0 - u >= 0) {
            const double x = (yy[u] - bb[u] * y1 - ee[u] * y2) * aa[u];
            AT(y, i0 - u) = x;
            mx = fmax(mx, fabs(x));
            y2 = y1;
            y1 = x;
          }
      }
      if (q > k) {
        // against the cluster's earlier members
        for (int p = k; p < q; ++p) {
          double dot = 0.0;
          for (int i = 0; i < n; ++i) dot += AT(y, i) * Zt[(size_t)i * n + p];
          for (int i = 0; i < n; ++i) AT(y, i) -= dot * Zt[(size_t)i * n + p];
        }
        mx = 0.0;
        for (int i = 0; i < n; ++i) mx = fmax(mx, fabs(AT(y, i)));
      }
      // to unit length
      const double sc = mx > 0.0 ? 1.0 / mx : 1.0;
      double nrm2 = 0.0;
#pragma unroll 8
      for (int i = 0; i < n; ++i) {
        const double v = AT(y, i) * sc;
        nrm2 = fma(v, v, nrm2);
      }
      const double f = sc / sqrt(nrm2);
      double* out = it + 1 < kInvIters ? y : Zt + q;
      const size_t so = it + 1 < kInvIters ? st : (size_t)n;
      for (int i0 = 0; i0 < n; i0 += U) {
        double yy[U];
#pragma unroll
        for (int u = 0; u < U; ++u) yy[u] = AT(y, min(i0 + u, n - 1));
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (i0 + u < n) out[(size_t)(i0 + u) * so] = yy[u] * f;
      }
    }
  }
#undef AT
}

// The reflectors quantised in place for the back-transformation: v_j(1:) (rows j + 2 ..) of column j as int4 with the
// exponent exv[j]; v_j(0) = 1 is implied.  One CTA per column.  A column's sum v^H z of the high limbs is at most
// 2^55 sqrt(2 n) (z has unit length): one bit less in v keeps it in 64 bits beyond 16,384 rows.
__global__ void __launch_bounds__(256) tri_quantise_kernel(zd* __restrict__ A, int n, int lda, int* __restrict__ exv) {
  __shared__ int s_f;
  const int j = blockIdx.x, tid = threadIdx.x;
  zd* v = A + (size_t)j * lda;
  if (tid == 0) s_f = 0;
  __syncthreads();
  int f = 0;
  for (int r = j + 2 + tid; r < n; r += 256) f = max(f, max(exponent_of(v[r].re), exponent_of(v[r].im)));
  f = __reduce_max_sync(0xffffffffu, f);
  if ((tid & 31) == 0) atomicMax(&s_f, f);
  __syncthreads();
  const int ex = group_ex(s_f) + (n > 16384 ? 1 : 0);
  if (tid == 0) exv[j] = ex;
  int4* q = reinterpret_cast<int4*>(v);
  for (int r = j + 2 + tid; r < n; r += 256) q[r] = quantise(v[r], ex);
}

// Z = Q Zt with Q = H_0 H_1 ... H_{n-2}, H_j = I - tau_j v_j v_j^H: the reflectors applied from j = n-2 down to 0 to
// every column.  A CTA owns kc columns for the whole sweep, so the columns need no synchronisation between CTAs.  The
// columns are held in fixed point, 64-bit integers in units of 2^-60 (they have unit length throughout), in shared
// memory where they fit, else in Z itself; a thread owns the same rows of its column for every reflector.  v^H z and
// v f run as exact integer sums (kQ above; the two 32-bit halves of z are its limbs, the lower one shortened to 28
// bits; f quantised with an exponent of its own), f = tau v^H z itself in FP64.  Rounding: 2^-61 an update and entry, where FP64 has 2^-53 of the entry; v^H z
// to 2^-56 of its terms.  Bound by the integer multiply-adds (24 an entry and reflector; the FP64 form 8 on a pipe
// a twelfth as fast).  n = 1,520: 38.9 -> 15.3 ms.
// Z(i, k) = Z[i * n + k] (row-major), conjugated at the end when the solver worked on conj(H).
// A row adds up to 2^56.6 to a low sum, so it is carried into the high one every kBtFold rows of a thread; columns in
// shared memory have at most 50 and go without (the nested loop took n = 1,520 from 50.5 to 52.3 ms).
constexpr int kBtThreads = 256, kBtFold = 64;
__device__ __forceinline__ void carry(long long& hh, long long& cr) {
  hh += cr >> 28;
  cr &= (1ll << 28) - 1;
}
__global__ void __launch_bounds__(kBtThreads) tri_backtransform_kernel(const zd* __restrict__ A, int n, int lda,
                                                                       const zd* __restrict__ tau,
                                                                       const int* __restrict__ exv,
                                                                       const double* __restrict__ Zt,
                                                                       zd* __restrict__ Z, int conj_out, int kc,
                                                                       int in_smem) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ long long red[2][kBtThreads];
  __shared__ int4 fq[32];
  __shared__ int exf[32], bad[32];
  const int tid = threadIdx.x, nsl = kBtThreads / kc, c = tid % kc, sl = tid / kc;
  const int k0 = blockIdx.x * kc, k = k0 + c;
  const bool on = sl < nsl && k < n;
  longlong2* z = in_smem ? reinterpret_cast<longlong2*>(smem_raw) + c : reinterpret_cast<longlong2*>(Z) + k;
  const size_t ldz = in_smem ? kc : n;
  if (tid < 32) bad[tid] = 0;
  __syncthreads();
  if (on)
    for (int i = sl; i < n; i += nsl) {
      const double x = Zt[(size_t)i * n + k];
      if (!(fabs(x) <= 2.0)) bad[c] = 1;
      longlong2 zi;
      zi.x = __double2ll_rn(x * 1152921504606846976.0);  // 2^60
      zi.y = 0;
      z[i * ldz] = zi;
    }
  for (int j = n - 2; j >= 0; --j) {
    const zd tj = tau[j];
    if (tj.re == 0.0 && tj.im == 0.0) continue;  // uniform
    const int4* v = reinterpret_cast<const int4*>(A + (size_t)j * lda);
    const int ex = exv[j];
    const int i0 = j + 2 + ((sl - (j + 2)) % nsl + nsl) % nsl;  // this thread's first row from j + 2 on
    const bool head = on && (j + 1) % nsl == sl;                // it owns row j + 1
    long long rh = 0, rc = 0, ih = 0, ic = 0;
    auto row = [&](int i) {  // conj(v) z
      const int4 a = v[i];
      const longlong2 zi = z[i * ldz];
      const int xl = (int)zi.x, yl = (int)zi.y;
      const int xh = (int)(zi.x >> 32) + (xl < 0), yh = (int)(zi.y >> 32) + (yl < 0);
      const int xs = xl >> 4, ys = yl >> 4;
      mac(rh, rc, a.x, a.y, xh, xs);
      mac(rh, rc, a.z, a.w, yh, ys);
      mac(ih, ic, a.x, a.y, yh, ys);
      mac(ih, ic, -a.z, -a.w, xh, xs);
    };
    if (on && in_smem)
      for (int i = i0; i < n; i += nsl) row(i);
    else if (on)
      for (int i = i0; i < n;) {
        const int i1 = (int)min((long)n, i + (long)kBtFold * nsl);
        for (; i < i1; i += nsl) row(i);
        carry(rh, rc);
        carry(ih, ic);
      }
    red[0][tid] = rh + ((rc + (1ll << 27)) >> 28);
    red[1][tid] = ih + ((ic + (1ll << 27)) >> 28);
    __syncthreads();
    // the sums of a column's slices, eight lanes each, then f
    if (tid < 8 * kc) {
      const int cc = tid >> 3, l = tid & 7;
      long long sr = 0, si = 0;
      for (int q = l; q < nsl; q += 8) {
        sr += red[0][q * kc + cc];
        si += red[1][q * kc + cc];
      }
      const unsigned m = 0xffu << (tid & 24);  // the column's eight lanes: their trip counts above may differ
      for (int o = 4; o > 0; o >>= 1) {
        sr += __shfl_xor_sync(m, sr, o);
        si += __shfl_xor_sync(m, si, o);
      }
      if (l == 0 && k0 + cc < n) {
        const longlong2 z0 = (in_smem ? reinterpret_cast<longlong2*>(smem_raw) + cc
                                      : reinterpret_cast<longlong2*>(Z) + k0 + cc)[(size_t)(j + 1) * ldz];
        constexpr double u60 = 1.0 / 1152921504606846976.0;
        const double sv = pow2(ex - kQ);
        const zd p = mk<double>(fma((double)sr, sv, (double)z0.x * u60), fma((double)si, sv, (double)z0.y * u60));
        const zd f = cmul(tj, p);
        const bool ok = fabs(f.re) < 4.0 && fabs(f.im) < 4.0;
        if (!ok) bad[cc] = 1;
        const int ef = ok ? group_ex(max(exponent_of(f.re), exponent_of(f.im))) : kExpZero;
        exf[cc] = ef;
        fq[cc] = quantise(f, ef);
      }
    }
    __syncthreads();
    if (on) {
      const int4 f = fq[c];
      const int eh = exf[c] + 5;  // f's unit, and (below) the high sums' one, in units of z: 2^eh, 2^sh
      if (head && eh > -62) {  // z -= f
        longlong2 zi = z[(size_t)(j + 1) * ldz];
        const long long fx = ((long long)f.x << 28) + f.y, fy = ((long long)f.z << 28) + f.w;
        zi.x -= eh >= 0 ? fx << eh : (fx + (1ll << (-eh - 1))) >> -eh;
        zi.y -= eh >= 0 ? fy << eh : (fy + (1ll << (-eh - 1))) >> -eh;
        z[(size_t)(j + 1) * ldz] = zi;
      }
      const int sh = ex + eh + 1;
      for (int i = i0; i < n; i += nsl) {  // z -= v f
        const int4 a = v[i];
        longlong2 zi = z[i * ldz];
        long long xh = 0, xc = 0, yh = 0, yc = 0;
        mac(xh, xc, a.x, a.y, f.x, f.y);
        mac(xh, xc, -a.z, -a.w, f.z, f.w);
        mac(yh, yc, a.x, a.y, f.z, f.w);
        mac(yh, yc, a.z, a.w, f.x, f.y);
        if (sh >= 0) {
          zi.x -= (xh << sh) + ((xc + (1ll << (27 - sh))) >> (28 - sh));
          zi.y -= (yh << sh) + ((yc + (1ll << (27 - sh))) >> (28 - sh));
        } else if (sh > -62) {
          const long long half = 1ll << (-sh - 1);
          zi.x -= (xh + (xc >> 28) + half) >> -sh;
          zi.y -= (yh + (yc >> 28) + half) >> -sh;
        }
        z[i * ldz] = zi;
      }
    }
  }
  __syncthreads();
  if (on) {
    constexpr double u60 = 1.0 / 1152921504606846976.0;
    const double nan = bad[c] ? __longlong_as_double(0x7ff8000000000000ll) : 0.0;
    for (int i = sl; i < n; i += nsl) {
      const longlong2 zi = z[i * ldz];
      const double re = (double)zi.x * u60 + nan, im = (double)zi.y * u60 + nan;
      Z[(size_t)i * n + k] = mk<double>(re, conj_out ? -im : im);
    }
  }
}

// Columns a CTA of the back-transformation: the fewest rounds of CTAs times columns, with the ~2,500 clocks of a
// reflector's reduction hidden where several CTAs share an SM, and the fewer columns where two counts tie.  0: the
// columns do not fit shared memory.  Measured with 1 to 8 columns at 34 sizes from 300 to 4,096: the least time, or
// within 14 % of it (0.72 ms with 1, 0.68 with 2 at 300; 2.44, 2.12 at 700; 10.5, 11.2 and 8.0 with 3 at 1,300; 13.5, 14.4
// and 16.4 at 1,459; 18.7, 16.6 and 17.5 at 1,600; 46.2, 54.8 and 59.6 at 2,304).
inline int bt_columns(int n, size_t* smem) {
  int best = 0;
  double cost = 0.0;
  for (int kc = 1; kc <= 16; ++kc) {
    const size_t b = (size_t)n * kc * sizeof(longlong2);
    if (b > 200 * 1024) break;
    // an SM's 228 KB, of which a CTA takes its columns, 4.75 KB for the sums and 1 KB for the system
    const int res = (int)std::min<size_t>(4, (228 * 1024) / (b + 5888));
    const long ctas = (n + kc - 1) / kc, rounds = (ctas + 152L * res - 1) / (152L * res);
    const double work = 0.5 * n * kc * 24.0 / 21.0, t = rounds * std::max(res * work, work + 2500.0);
    if (!best || t < cost * (1.0 - 1e-9)) {
      best = kc;
      cost = t;
      *smem = b;
    }
  }
  return best;
}

}  // namespace

// The reduction's buffers in one scratch block.
struct TriScratch {
  zd *xw, *u, *next, *tau, *dots, *g, *W, *P;
  double *sparts, *e, *d, *ds, *e2, *bounds;
  float *dsf, *e2f;
  TriCol* col;
  int *Aex, *exv;
  int4* Aq;
  size_t bytes;
  TriScratch(int n, void* base) {
    const int nT = tiles_of(n);
    const size_t nd = (size_t)(n + kRows - 1) / kRows, nt = lower_tiles(nT);
    unsigned char* p = reinterpret_cast<unsigned char*>(base);
    auto take = [&](size_t b) {
      unsigned char* q = p;
      p += (b + 15) & ~(size_t)15;
      return q;
    };
    Aq = reinterpret_cast<int4*>(take(nt * kT * kT * sizeof(int4)));
    P = reinterpret_cast<zd*>(take((size_t)(nT + 1) * n * sizeof(zd)));
    W = reinterpret_cast<zd*>(take((size_t)kNB * n * sizeof(zd)));
    xw = reinterpret_cast<zd*>(take(n * sizeof(zd)));
    u = reinterpret_cast<zd*>(take(n * sizeof(zd)));
    next = reinterpret_cast<zd*>(take(n * sizeof(zd)));
    tau = reinterpret_cast<zd*>(take(n * sizeof(zd)));
    dots = reinterpret_cast<zd*>(take(nd * sizeof(zd)));
    g = reinterpret_cast<zd*>(take((size_t)(n + kDotRows - 1) / kDotRows * 2 * kNB * sizeof(zd)));
    col = reinterpret_cast<TriCol*>(take(sizeof(TriCol)));
    sparts = reinterpret_cast<double*>(take(nd * sizeof(double)));
    e = reinterpret_cast<double*>(take(n * sizeof(double)));
    d = reinterpret_cast<double*>(take(n * sizeof(double)));
    ds = reinterpret_cast<double*>(take(n * sizeof(double)));
    e2 = reinterpret_cast<double*>(take(n * sizeof(double)));
    bounds = reinterpret_cast<double*>(take(4 * sizeof(double)));
    dsf = reinterpret_cast<float*>(take(n * sizeof(float)));
    e2f = reinterpret_cast<float*>(take(n * sizeof(float)));
    Aex = reinterpret_cast<int*>(take(nt * sizeof(int)));
    exv = reinterpret_cast<int*>(take(n * sizeof(int)));
    bytes = (size_t)(p - reinterpret_cast<unsigned char*>(base));
  }
};

size_t dense_eig_scratch(int n) { return TriScratch(n, nullptr).bytes; }

constexpr size_t kSymvSmem = sizeof(int4) * (kT * (kT + 1) + 2 * kT) + sizeof(int2) * 2 * kT;
constexpr size_t kUpdateSmem = sizeof(int4) * 3 * kNB * kT;

cudaError_t dense_eig_prepare() {
  cudaError_t err = raise_smem_limit(reinterpret_cast<const void*>(tri_symv_kernel), kSymvSmem);
  if (err == cudaSuccess) err = raise_smem_limit(reinterpret_cast<const void*>(tri_update_kernel), kUpdateSmem);
  return err;
}

// The reduction: per column the two kernels, per panel the trailing update.
static cudaError_t tridiagonalise(zd* A, int n, int lda, const TriScratch& t, cudaStream_t s) {
  cudaError_t err = dense_eig_prepare();
  if (err != cudaSuccess) return err;
  const int nT = tiles_of(n);
  int ndots = 0;
  auto update = [&](int j1, int reflectors) {
    const unsigned ctas = 2 * (unsigned)lower_tiles(nT - j1 / kT);
    tri_update_kernel<<<ctas, 512, kUpdateSmem, s>>>(A, n, lda, j1, reflectors, t.tau, t.W, t.xw, t.dots, ndots, t.Aq,
                                                     t.Aex);
    ++g_launch_count;
  };
  cudaLaunchAttribute early = {};
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  auto launch = [&](auto kernel, unsigned grid, unsigned threads, size_t smem, auto... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &early;
    cfg.numAttrs = 1;
    ++g_launch_count;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
  };
  update(0, 0);
  int i = 0;
  for (int j = 0; j < n; ++j) {
    const bool last = j + 1 == n;  // the last column has a diagonal entry only
    const unsigned tiles = last ? 0 : (unsigned)lower_tiles(nT - (j + 1) / kT);
    const int nch = (n - j - 1 + kDotRows - 1) / kDotRows;
    const int nnext = i + 1 < kNB ? (n - j - 1 + kNextRows - 1) / kNextRows : 0;  // a panel's last column has no next
    err = launch(tri_symv_kernel, tiles + 1 + (unsigned)(i * nch + nnext), 256, kSymvSmem, A, n, lda, j, i, t.W, t.u, t.xw, t.dots,
                 t.sparts, ndots, t.Aq, t.Aex, t.col, t.tau, t.e, t.g, nch, t.next, nnext, t.P);
    if (err != cudaSuccess || last) break;
    ndots = (n - j - 1 + kRows - 1) / kRows;
    err = launch(tri_x_kernel, (unsigned)ndots, 16 * (kRows + 2), 0, A, n, lda, j, i, nnext ? t.next : (const zd*)nullptr, t.W, t.P,
                 t.col, t.g, nch, t.u, t.xw, t.dots, t.sparts);
    if (err != cudaSuccess) break;
    if (++i == kNB) {
      update(j + 1, 1);
      i = 0;
    }
  }
  return err == cudaSuccess ? cudaGetLastError() : err;
}

static int invit_batch(int n) {
  const long nb = (1L << 25) / (6L * n);  // the inverse-iteration scratch stays near 256 MB
  return (int)std::max(1L, std::min((long)n, nb));
}

size_t dense_eigvec_scratch(int n) {
  return sizeof(double) * ((size_t)n * n + (size_t)6 * n * invit_batch(n));
}

cudaError_t launch_dense_eigvals(zd* A, int n, int lda, bool upper_only, double* W, void* scratch,
                                 cudaStream_t s) {
  return launch_dense_eig(A, n, lda, upper_only, W, nullptr, false, scratch, nullptr, s);
}

cudaError_t launch_dense_eig(zd* A, int n, int lda, bool upper_only, double* W, zd* Z, bool conj_vectors,
                             void* scratch, void* vscratch, cudaStream_t s) {
  if (Z && !vscratch) return cudaErrorInvalidValue;
  if (n < 1 || lda < n) return cudaErrorInvalidValue;
  const TriScratch t(n, scratch);
  zd* tau = t.tau;
  double *e = t.e, *d = t.d, *ds = t.ds, *e2 = t.e2, *bounds = t.bounds;
  if (upper_only) {
    mirror_upper_kernel<<<(unsigned)(((long)n * n + 255) / 256), 256, 0, s>>>(A, n, lda); ++g_launch_count;
  }
  const cudaError_t err = tridiagonalise(A, n, lda, t, s);
  if (err != cudaSuccess) return err;
  tri_finish_kernel<<<1, 1024, 0, s>>>(A, n, lda, d, e, bounds); ++g_launch_count;
  tri_scale_kernel<<<(n + 255) / 256, 256, 0, s>>>(d, e, n, bounds, ds, e2, t.dsf, t.e2f); ++g_launch_count;
  int L = 1;  // about two warps per SM
  while (L < 32 && (long)n * L < 152L * 64) L *= 2;
  tri_multisect_kernel<<<(unsigned)(((long)n * L + 127) / 128), 128, 0, s>>>(ds, e2, n, t.dsf, t.e2f, bounds, W,
                                                                             L); ++g_launch_count;
  if (Z) {
    double* Zt = reinterpret_cast<double*>(vscratch);
    double* work = Zt + (size_t)n * n;
    const int nb = invit_batch(n);
    for (int k0 = 0; k0 < n; k0 += nb) {
      tri_invit_kernel<<<(nb + 31) / 32, 32, 0, s>>>(d, e, n, W, bounds, k0, nb, work, Zt); ++g_launch_count;
    }
    if (n > 1) {
      tri_quantise_kernel<<<n - 1, 256, 0, s>>>(A, n, lda, t.exv); ++g_launch_count;
    }
    size_t smem = 0;
    const int fit = bt_columns(n, &smem), kc = fit ? fit : 8;
    if (!fit) smem = 0;
    const cudaError_t eb = raise_smem_limit(reinterpret_cast<const void*>(tri_backtransform_kernel), smem);
    if (eb != cudaSuccess) return eb;
    tri_backtransform_kernel<<<(n + kc - 1) / kc, kBtThreads, smem, s>>>(A, n, lda, tau, t.exv, Zt, Z,
                                                                         conj_vectors ? 1 : 0, kc, fit ? 1 : 0);
    ++g_launch_count;
  }
  return cudaGetLastError();
}

}  // namespace wtb
