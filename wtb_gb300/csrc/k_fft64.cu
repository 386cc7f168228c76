// FP64 form of the contraction T = V Z on a Monkhorst-Pack mesh of one, two or three dimensions.
//
// On the mesh V(k, k') = s(k - k') (coulomb_stencil_kernel), so each column of T = V Z is the linear convolution of
// the stencil with the column of Z on the n1 x n2 x n3 mesh: a cyclic convolution of size P_d >= 2 n_d - 1 per
// dimension, T = IDFT(S o DFT(z)) with S the transform of the wrapped stencil over P1 P2 P3.  The stencil is real, so
// the re and im rows n = 2q, 2q + 1 of Z go through one complex transform.
//
// The FP64 pipe bounds every FP64 kernel of this part (2 multiply-adds a clock and SM, 1/64 of the FP32 rate), so the
// design counts FP64 instructions and nothing else; index arithmetic, shared memory and barriers are cheap beside
// them.  Each length P = R1 R2 with coprime R1, R2 <= 16 runs as a Good-Thomas (prime-factor) transform: element
// (R2 a + R1 b) mod P is slot (a, b), an R1-point DFT over a and an R2-point DFT over b give X[k] with k = k1 mod R1,
// k2 mod R2 in slot (k1, k2), with no twiddle factors at all.  The frequencies stay in that order; the spectrum is
// stored in it.  The lengths come from the table in plan_length (15 x 8 = 120 for 60 points: 17.8 FP64 instructions a
// point against 21 for the radix-2 128).  At 60 x 60 a column takes about 0.83 M FP64 instructions where the product
// takes 26 M.
//
// One CTA per complex column.  The mesh is taken as m1 x m2 x m3 with unit dimensions dropped (2D: m2 = 1):
//   A. rows: DFT over the innermost dimension, m1 m2 rows of P3 slots in shared memory;
//   B. batches of the P3 planes (2D: columns): plane to a P1 x P2 scratch, DFT over dimension 2, over dimension 1,
//      times S, inverse over dimension 1, over dimension 2; the m1 x m2 results on the mesh go back to the rows;
//   C. inverse rows; the m3 results on the mesh go to T.
// The second factor of dimension 1, the product with S and the inverse's first factor stay in registers.
// Measured per 16-column application: 3.04 ms at 48 x 45, w = 12 (2,304 columns of 0.61 M FP64 instructions: 73 % of
// the FP64 pipe's issue rate; the product 37.3 ms), 4.48 ms at 11^3, w = 16 (the product 24.5 ms), 0.40 ms at 30 x 30,
// w = 8 (3.9 ms).
#include "wtb_internal.h"

#include <algorithm>

namespace wtb {
namespace {

typedef double2 d2;
__device__ __forceinline__ d2 D(double a, double b) { return make_double2(a, b); }
__device__ __forceinline__ d2 add(d2 a, d2 b) { return D(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ d2 sub(d2 a, d2 b) { return D(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ d2 mi(d2 a) { return D(a.y, -a.x); }  // -i a
__device__ __forceinline__ d2 axpy(double c, d2 a, d2 b) { return D(fma(c, a.x, b.x), fma(c, a.y, b.y)); }  // c a + b
__device__ __forceinline__ d2 scal(double c, d2 a) { return D(c * a.x, c * a.y); }
// a - i c b
__device__ __forceinline__ d2 submi(double c, d2 b, d2 a) { return D(fma(c, b.y, a.x), fma(-c, b.x, a.y)); }

__device__ __forceinline__ void dft2(d2& a, d2& b) {
  const d2 t = a;
  a = add(t, b);
  b = sub(t, b);
}
__device__ __forceinline__ void dft3(d2& a, d2& b, d2& c) {
  constexpr double S = 0.86602540378443864676;  // sin(2 pi / 3)
  const d2 p = add(b, c), m = sub(b, c), h = axpy(-0.5, p, a);
  a = add(a, p);
  b = submi(S, m, h);
  c = submi(-S, m, h);
}
__device__ __forceinline__ void dft4(d2& a, d2& b, d2& c, d2& e) {
  const d2 t0 = add(a, c), t1 = sub(a, c), t2 = add(b, e), t3 = mi(sub(b, e));
  a = add(t0, t2);
  c = sub(t0, t2);
  b = add(t1, t3);
  e = sub(t1, t3);
}
// X_k = x0 + sum_j p_j cos(2 pi j k / R) - i sum_j m_j sin(2 pi j k / R), p_j = x_j + x_{R-j}, m_j = x_j - x_{R-j}
__device__ __forceinline__ void dft5(d2 (&x)[5]) {
  constexpr double C1 = 0.30901699437494742410, C2 = -0.80901699437494742410;
  constexpr double S1 = 0.95105651629515357212, S2 = 0.58778525229247312917;
  const d2 p1 = add(x[1], x[4]), p2 = add(x[2], x[3]), m1 = sub(x[1], x[4]), m2 = sub(x[2], x[3]);
  const d2 a1 = axpy(C2, p2, axpy(C1, p1, x[0])), a2 = axpy(C1, p2, axpy(C2, p1, x[0]));
  const d2 b1 = axpy(S2, m2, scal(S1, m1)), b2 = axpy(-S1, m2, scal(S2, m1));
  x[0] = add(x[0], add(p1, p2));
  x[1] = add(a1, mi(b1));
  x[4] = sub(a1, mi(b1));
  x[2] = add(a2, mi(b2));
  x[3] = sub(a2, mi(b2));
}
__device__ __forceinline__ void dft7(d2 (&x)[7]) {
  constexpr double C1 = 0.62348980185873353053, C2 = -0.22252093395631440429, C3 = -0.90096886790241912624;
  constexpr double S1 = 0.78183148246802980871, S2 = 0.97492791218182360702, S3 = 0.43388373911755812048;
  const d2 p1 = add(x[1], x[6]), p2 = add(x[2], x[5]), p3 = add(x[3], x[4]);
  const d2 m1 = sub(x[1], x[6]), m2 = sub(x[2], x[5]), m3 = sub(x[3], x[4]);
  const d2 a1 = axpy(C3, p3, axpy(C2, p2, axpy(C1, p1, x[0])));
  const d2 a2 = axpy(C1, p3, axpy(C3, p2, axpy(C2, p1, x[0])));
  const d2 a3 = axpy(C2, p3, axpy(C1, p2, axpy(C3, p1, x[0])));
  const d2 b1 = axpy(S3, m3, axpy(S2, m2, scal(S1, m1)));
  const d2 b2 = axpy(-S1, m3, axpy(-S3, m2, scal(S2, m1)));
  const d2 b3 = axpy(S2, m3, axpy(-S1, m2, scal(S3, m1)));
  x[0] = add(x[0], add(p1, add(p2, p3)));
  x[1] = add(a1, mi(b1));
  x[6] = sub(a1, mi(b1));
  x[2] = add(a2, mi(b2));
  x[5] = sub(a2, mi(b2));
  x[3] = add(a3, mi(b3));
  x[4] = sub(a3, mi(b3));
}
// times exp(-2 pi i j / N) = c - i s
__device__ __forceinline__ d2 tw(d2 a, double c, double s) {
  return D(fma(s, a.y, c * a.x), fma(-s, a.x, c * a.y));
}
__device__ __forceinline__ void dft8(d2 (&x)[8]) {
  constexpr double R = 0.70710678118654752440;
  dft4(x[0], x[2], x[4], x[6]);
  dft4(x[1], x[3], x[5], x[7]);
  // odd half: X order of x[1], x[3], x[5], x[7] is k = 0, 1, 2, 3
  const d2 o1 = D(R * (x[3].x + x[3].y), R * (x[3].y - x[3].x)), o2 = mi(x[5]);
  const d2 o3 = D(R * (x[7].y - x[7].x), -R * (x[7].x + x[7].y));
  const d2 e0 = x[0], e1 = x[2], e2 = x[4], e3 = x[6], o0 = x[1];
  x[0] = add(e0, o0);
  x[4] = sub(e0, o0);
  x[1] = add(e1, o1);
  x[5] = sub(e1, o1);
  x[2] = add(e2, o2);
  x[6] = sub(e2, o2);
  x[3] = add(e3, o3);
  x[7] = sub(e3, o3);
}
__device__ __forceinline__ void dft9(d2 (&x)[9]) {
  constexpr double c1 = 0.76604444311897803520, s1 = 0.64278760968653932632;  // 2 pi / 9
  constexpr double c2 = 0.17364817766693034885, s2 = 0.98480775301220805937;  // 4 pi / 9
  constexpr double c4 = -0.93969262078590838405, s4 = 0.34202014332566873304;  // 8 pi / 9
  dft3(x[0], x[3], x[6]);
  dft3(x[1], x[4], x[7]);
  dft3(x[2], x[5], x[8]);
  x[4] = tw(x[4], c1, s1);
  x[7] = tw(x[7], c2, s2);
  x[5] = tw(x[5], c2, s2);
  x[8] = tw(x[8], c4, s4);
  dft3(x[0], x[1], x[2]);
  dft3(x[3], x[4], x[5]);
  dft3(x[6], x[7], x[8]);
  // x[3 c + d] holds X[c + 3 d]
  d2 t = x[1]; x[1] = x[3]; x[3] = t;
  t = x[2]; x[2] = x[6]; x[6] = t;
  t = x[5]; x[5] = x[7]; x[7] = t;
}
__device__ __forceinline__ void dft16(d2 (&x)[16]) {
  constexpr double C = 0.92387953251128675613, S = 0.38268343236508977173, R = 0.70710678118654752440;
#pragma unroll
  for (int a = 0; a < 4; ++a) dft4(x[a], x[a + 4], x[a + 8], x[a + 12]);
  // x[a + 4 c]: twiddle by W_16^(a c)
  x[5] = tw(x[5], C, S);
  x[9] = D(R * (x[9].x + x[9].y), R * (x[9].y - x[9].x));
  x[13] = tw(x[13], S, C);
  x[6] = D(R * (x[6].x + x[6].y), R * (x[6].y - x[6].x));
  x[10] = mi(x[10]);
  x[14] = D(R * (x[14].y - x[14].x), -R * (x[14].x + x[14].y));
  x[7] = tw(x[7], S, C);
  x[11] = D(R * (x[11].y - x[11].x), -R * (x[11].x + x[11].y));
  x[15] = tw(x[15], -C, -S);
#pragma unroll
  for (int c = 0; c < 4; ++c) dft4(x[4 * c], x[4 * c + 1], x[4 * c + 2], x[4 * c + 3]);
  d2 y[16];  // x[4 c + e] holds X[c + 4 e]
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int e = 0; e < 4; ++e) y[c + 4 * e] = x[4 * c + e];
#pragma unroll
  for (int k = 0; k < 16; ++k) x[k] = y[k];
}

template <int R>
__device__ __forceinline__ void dft(d2 (&x)[R]);

// R = A B, coprime: the prime-factor transform in registers (all indices are compile-time constants)
template <int A, int B>
__device__ __forceinline__ void dft_pf(d2 (&x)[A * B]) {
  constexpr int R = A * B;
  d2 y[B][A];
#pragma unroll
  for (int b = 0; b < B; ++b) {
#pragma unroll
    for (int a = 0; a < A; ++a) y[b][a] = x[(B * a + A * b) % R];
    dft<A>(y[b]);
  }
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    d2 z[B];
#pragma unroll
    for (int b = 0; b < B; ++b) z[b] = y[b][k1];
    dft<B>(z);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) {
      // the frequency k < R with k = k1 mod A and k = k2 mod B
      int k = k1;
#pragma unroll
      for (int t = 0; t < B; ++t)
        if ((k1 + A * t) % B == k2) k = k1 + A * t;
      x[k] = z[k2];
    }
  }
}

template <int R>
__device__ __forceinline__ void dft(d2 (&x)[R]) {
  if constexpr (R == 2) dft2(x[0], x[1]);
  else if constexpr (R == 3) dft3(x[0], x[1], x[2]);
  else if constexpr (R == 4) dft4(x[0], x[1], x[2], x[3]);
  else if constexpr (R == 5) dft5(x);
  else if constexpr (R == 7) dft7(x);
  else if constexpr (R == 8) dft8(x);
  else if constexpr (R == 9) dft9(x);
  else if constexpr (R == 10) dft_pf<2, 5>(x);
  else if constexpr (R == 12) dft_pf<3, 4>(x);
  else if constexpr (R == 15) dft_pf<3, 5>(x);
  else if constexpr (R == 16) dft16(x);
}

__device__ __forceinline__ d2 swp(d2 a) { return D(a.y, a.x); }

// One R-point DFT: x[m] = load(m), store(m, X[m]).  INV: the unnormalised inverse, as the forward transform of the
// sequence with re and im exchanged.
template <int R, bool INV, class L, class St>
__device__ __forceinline__ void one_dft(const L& load, const St& store) {
  d2 x[R];
#pragma unroll
  for (int m = 0; m < R; ++m) x[m] = INV ? swp(load(m)) : load(m);
  dft<R>(x);
#pragma unroll
  for (int m = 0; m < R; ++m) store(m, INV ? swp(x[m]) : x[m]);
}

template <bool INV, class L, class St>
__device__ __forceinline__ void any_dft(int R, const L& load, const St& store) {
  switch (R) {  // uniform over the CTA
    case 1: one_dft<1, INV>(load, store); break;
    case 2: one_dft<2, INV>(load, store); break;
    case 3: one_dft<3, INV>(load, store); break;
    case 4: one_dft<4, INV>(load, store); break;
    case 5: one_dft<5, INV>(load, store); break;
    case 7: one_dft<7, INV>(load, store); break;
    case 8: one_dft<8, INV>(load, store); break;
    case 9: one_dft<9, INV>(load, store); break;
    case 10: one_dft<10, INV>(load, store); break;
    case 12: one_dft<12, INV>(load, store); break;
    case 15: one_dft<15, INV>(load, store); break;
    default: one_dft<16, INV>(load, store); break;
  }
}

// R-point DFT, product with the spectrum values sp(m), inverse R-point DFT
template <int R, class L, class Sp, class St>
__device__ __forceinline__ void one_mul(const L& load, const Sp& sp, const St& store) {
  d2 x[R];
#pragma unroll
  for (int m = 0; m < R; ++m) x[m] = load(m);
  dft<R>(x);
#pragma unroll
  for (int m = 0; m < R; ++m) {
    const d2 s = sp(m);
    x[m] = D(fma(x[m].x, s.y, x[m].y * s.x), fma(x[m].x, s.x, -x[m].y * s.y));  // re and im exchanged
  }
  dft<R>(x);
#pragma unroll
  for (int m = 0; m < R; ++m) store(m, swp(x[m]));
}
template <class L, class Sp, class St>
__device__ __forceinline__ void any_mul(int R, const L& load, const Sp& sp, const St& store) {
  switch (R) {
    case 1: one_mul<1>(load, sp, store); break;
    case 2: one_mul<2>(load, sp, store); break;
    case 3: one_mul<3>(load, sp, store); break;
    case 4: one_mul<4>(load, sp, store); break;
    case 5: one_mul<5>(load, sp, store); break;
    case 7: one_mul<7>(load, sp, store); break;
    case 8: one_mul<8>(load, sp, store); break;
    case 9: one_mul<9>(load, sp, store); break;
    case 10: one_mul<10>(load, sp, store); break;
    case 12: one_mul<12>(load, sp, store); break;
    case 15: one_mul<15>(load, sp, store); break;
    default: one_mul<16>(load, sp, store); break;
  }
}

__device__ __forceinline__ int slot_of(int a, int b, int R1, int R2, int P) {
  const int t = R2 * a + R1 * b;
  return t < P ? t : t - P;
}

__global__ void __launch_bounds__(256) fft64_conv_kernel(Fft64Plan pl, const double* __restrict__ Z, int ldz,
                                                         const d2* __restrict__ spec, double* __restrict__ T, int ldt) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int m1 = pl.m[0], m2 = pl.m[1], m3 = pl.m[2], nrow = m1 * m2;
  const int P1 = pl.P[0], P2 = pl.P[1], P3 = pl.P[2];
  const int A1 = pl.R1[0], B1 = pl.R2[0], A2 = pl.R1[1], B2 = pl.R2[1], A3 = pl.R1[2], B3 = pl.R2[2];
  d2* Sb = reinterpret_cast<d2*>(smem_raw);  // [nrow][P3]
  d2* G = Sb + nrow * P3;                    // [batch][P1][P2]
  const int tid = threadIdx.x, nt = blockDim.x, q = blockIdx.x;
  const double* zre = Z + (size_t)(2 * q) * ldz;
  const double* zim = zre + ldz;
  const d2 zero = D(0.0, 0.0);
  // A. rows: over a (from global memory), then over b
  for (int it = tid; it < nrow * B3; it += nt) {
    const int b = it % B3, r = it / B3;
    d2* row = Sb + r * P3;
    const double *pr = zre + r * m3, *pi = zim + r * m3;
    any_dft<false>(
        A3,
        [&](int a) {
          const int l = slot_of(a, b, A3, B3, P3);
          return l < m3 ? D(pr[l], pi[l]) : zero;
        },
        [&](int a, d2 v) { row[slot_of(a, b, A3, B3, P3)] = v; });
  }
  __syncthreads();
  if (B3 > 1) {
    for (int it = tid; it < nrow * A3; it += nt) {
      const int a = it % A3;
      d2* row = Sb + (it / A3) * P3;
      any_dft<false>(
          B3, [&](int b) { return row[slot_of(a, b, A3, B3, P3)]; },
          [&](int b, d2 v) { row[slot_of(a, b, A3, B3, P3)] = v; });
    }
    __syncthreads();
  }
  // B. planes w0 .. w0 + np - 1.  The plane index runs fastest over the threads.
  const int PP = P1 * P2;
  for (int w0 = 0; w0 < P3; w0 += pl.batch) {
    const int np = min(pl.batch, P3 - w0);
    if (P2 > 1) {  // forward rows of every plane (m1 of them)
      for (int it = tid; it < np * m1 * B2; it += nt) {
        const int p = it % np, t = it / np, b = t % B2, i = t / B2;
        d2* row = G + p * PP + i * P2;
        any_dft<false>(
            A2,
            [&](int a) {
              const int j = slot_of(a, b, A2, B2, P2);
              return j < m2 ? Sb[(i * m2 + j) * P3 + w0 + p] : zero;
            },
            [&](int a, d2 v) { row[slot_of(a, b, A2, B2, P2)] = v; });
      }
      __syncthreads();
      if (B2 > 1) {
        for (int it = tid; it < np * m1 * A2; it += nt) {
          const int p = it % np, t = it / np, a = t % A2, i = t / A2;
          d2* row = G + p * PP + i * P2;
          any_dft<false>(
              B2, [&](int b) { return row[slot_of(a, b, A2, B2, P2)]; },
              [&](int b, d2 v) { row[slot_of(a, b, A2, B2, P2)] = v; });
        }
        __syncthreads();
      }
    }
    const bool two = P2 > 1;
    if (B1 > 1) {
      // columns: over a, from the mesh rows (the others are zero)
      for (int it = tid; it < np * P2 * B1; it += nt) {
        const int p = it % np, t = it / np, v = t % P2, b = t / P2;
        d2* col = G + p * PP + v;
        any_dft<false>(
            A1,
            [&](int a) {
              const int i = slot_of(a, b, A1, B1, P1);
              return i < m1 ? (two ? col[i * P2] : Sb[i * P3 + w0 + p]) : zero;
            },
            [&](int a, d2 x) { col[slot_of(a, b, A1, B1, P1) * P2] = x; });
      }
      __syncthreads();
      // over b, times the spectrum, inverse over b
      for (int it = tid; it < np * P2 * A1; it += nt) {
        const int p = it % np, t = it / np, v = t % P2, a = t / P2;
        d2* col = G + p * PP + v;
        const d2* sp = spec + (size_t)v * P3 + w0 + p;
        any_mul(
            B1, [&](int b) { return col[slot_of(a, b, A1, B1, P1) * P2]; },
            [&](int b) { return sp[(size_t)slot_of(a, b, A1, B1, P1) * P2 * P3]; },
            [&](int b, d2 x) { col[slot_of(a, b, A1, B1, P1) * P2] = x; });
      }
      __syncthreads();
      // inverse over a; the mesh rows stay
      for (int it = tid; it < np * P2 * B1; it += nt) {
        const int p = it % np, t = it / np, v = t % P2, b = t / P2;
        d2* col = G + p * PP + v;
        any_dft<true>(
            A1, [&](int a) { return col[slot_of(a, b, A1, B1, P1) * P2]; },
            [&](int a, d2 x) {
              const int i = slot_of(a, b, A1, B1, P1);
              if (i < m1) {
                if (two)
                  col[i * P2] = x;
                else
                  Sb[i * P3 + w0 + p] = x;
              }
            });
      }
      __syncthreads();
    } else {  // P1 = A1: the whole column in registers
      for (int it = tid; it < np * P2; it += nt) {
        const int p = it % np, v = it / np;
        d2* col = G + p * PP + v;
        const d2* sp = spec + (size_t)v * P3 + w0 + p;
        any_mul(
            A1, [&](int i) { return i < m1 ? (two ? col[i * P2] : Sb[i * P3 + w0 + p]) : zero; },
            [&](int i) { return sp[(size_t)i * P2 * P3]; },
            [&](int i, d2 x) {
              if (i < m1) {
                if (two)
                  col[i * P2] = x;
                else
                  Sb[i * P3 + w0 + p] = x;
              }
            });
      }
      __syncthreads();
    }
    if (two) {  // inverse rows of every plane; the mesh columns go back
      if (B2 > 1) {
        for (int it = tid; it < np * m1 * A2; it += nt) {
          const int p = it % np, t = it / np, a = t % A2, i = t / A2;
          d2* row = G + p * PP + i * P2;
          any_dft<true>(
              B2, [&](int b) { return row[slot_of(a, b, A2, B2, P2)]; },
              [&](int b, d2 v) { row[slot_of(a, b, A2, B2, P2)] = v; });
        }
        __syncthreads();
      }
      for (int it = tid; it < np * m1 * B2; it += nt) {
        const int p = it % np, t = it / np, b = t % B2, i = t / B2;
        const d2* row = G + p * PP + i * P2;
        any_dft<true>(
            A2, [&](int a) { return row[slot_of(a, b, A2, B2, P2)]; },
            [&](int a, d2 v) {
              const int j = slot_of(a, b, A2, B2, P2);
              if (j < m2) Sb[(i * m2 + j) * P3 + w0 + p] = v;
            });
      }
      __syncthreads();
    }
  }
  // C. inverse rows
  if (B3 > 1) {
    for (int it = tid; it < nrow * A3; it += nt) {
      const int a = it % A3;
      d2* row = Sb + (it / A3) * P3;
      any_dft<true>(
          B3, [&](int b) { return row[slot_of(a, b, A3, B3, P3)]; },
          [&](int b, d2 v) { row[slot_of(a, b, A3, B3, P3)] = v; });
    }
    __syncthreads();
  }
  for (int it = tid; it < nrow * B3; it += nt) {
    const int b = it % B3, r = it / B3;
    const d2* row = Sb + r * P3;
    double* out = T + (size_t)r * m3 * ldt + 2 * q;
    any_dft<true>(
        A3, [&](int a) { return row[slot_of(a, b, A3, B3, P3)]; },
        [&](int a, d2 v) {
          const int l = slot_of(a, b, A3, B3, P3);
          if (l < m3) *reinterpret_cast<d2*>(out + (size_t)l * ldt) = v;
        });
  }
}

// out[o][slot][i] = scale sum_l in[o][l][i] W_P^(f(slot) (l - (n - 1))), l < 2 n - 1, f(slot) the frequency in the
// slot (k1 mod R1, k2 mod R2): one dimension of the spectrum, W_P^m from a shared table.  first: in is the real stencil.
__global__ void __launch_bounds__(128) fft64_spec_kernel(const double* __restrict__ in, int first, int outer, int inner,
                                                         int n, int P, int R1, int R2, double scale,
                                                         d2* __restrict__ out) {
  __shared__ double wr[256], wi[256];
  for (int m = threadIdx.x; m < P; m += blockDim.x) {
    double sn, cs;
    sincospi(2.0 * m / P, &sn, &cs);
    wr[m] = cs;
    wi[m] = -sn;
  }
  __syncthreads();
  const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long)outer * P * inner) return;
  const int i = (int)(e % inner), slot = (int)((e / inner) % P);
  const long o = e / ((long)inner * P);
  // the frequency k with slot = (R2 k1 + R1 k2) mod P, k1 = k mod R1, k2 = k mod R2: the inverse of k -> slot
  int f = 0;
  for (int k = 0; k < P; ++k)
    if ((R2 * (k % R1) + R1 * (k % R2)) % P == slot) f = k;
  const int L = 2 * n - 1;
  double re = 0.0, im = 0.0;
  int m = (int)(((-(long)f * (n - 1)) % P + P) % P);
  for (int l = 0; l < L; ++l) {
    const size_t a = ((size_t)o * L + l) * inner + i;
    if (first) {
      const double x = in[a];
      re = fma(x, wr[m], re);
      im = fma(x, wi[m], im);
    } else {
      const d2 x = reinterpret_cast<const d2*>(in)[a];
      re = fma(x.x, wr[m], fma(-x.y, wi[m], re));
      im = fma(x.x, wi[m], fma(x.y, wr[m], im));
    }
    m += f;
    if (m >= P) m -= P;
  }
  out[e] = D(re * scale, im * scale);
}

// FP64 instructions of an R-point DFT (complex additions two, products by a constant folded into multiply-adds)
int dft_cost(int R) {
  switch (R) {
    case 1: return 0;
    case 2: return 4;
    case 3: return 12;
    case 4: return 16;
    case 5: return 36;
    case 7: return 72;
    case 8: return 56;
    case 9: return 88;
    case 10: return 2 * 36 + 5 * 4;
    case 12: return 4 * 12 + 3 * 16;
    case 15: return 5 * 12 + 3 * 36;
    default: return 168;
  }
}

// The cheapest P = R1 R2 >= 2 n - 1 with coprime factors (an R of one factor only: R2 = 1)
bool plan_length(int n, int* P, int* R1, int* R2, long* cost) {
  static const int kR[] = {1, 2, 3, 4, 5, 7, 8, 9, 10, 12, 15, 16};
  auto gcd = [](int a, int b) {
    while (b) {
      const int t = a % b;
      a = b;
      b = t;
    }
    return a;
  };
  if (n == 1) {
    *P = *R1 = *R2 = 1;
    *cost = 0;
    return true;
  }
  long best = -1;
  for (int a : kR)
    for (int b : kR) {
      if (b > a || a * b < 2 * n - 1 || gcd(a, b) != 1) continue;
      const long c = (long)b * dft_cost(a) + (long)a * dft_cost(b);
      if (best < 0 || c < best || (c == best && a * b < *P)) {
        best = c;
        *P = a * b;
        *R1 = a;
        *R2 = b;
      }
    }
  *cost = best;
  return best >= 0;
}

constexpr size_t kFft64Smem = 220 * 1024;  // dynamic shared memory of one CTA at most

}  // namespace

// The plan of an n1 x n2 x n3 mesh, or false where the transforms do not fit one CTA (the caller then multiplies by
// the table).  *per_column: FP64 instructions of one complex column.
bool fft64_plan(int n1, int n2, int n3, Fft64Plan* pl, double* per_column) {
  const int n[3] = {n1, n2, n3};
  int d[3], nd = 0;
  for (int i = 0; i < 3; ++i) {
    if (n[i] < 1) return false;
    if (n[i] > 1) d[nd++] = n[i];
  }
  pl->m[0] = nd >= 2 ? d[0] : 1;
  pl->m[1] = nd == 3 ? d[1] : 1;
  pl->m[2] = nd >= 1 ? d[nd - 1] : 1;
  long c[3];
  for (int i = 0; i < 3; ++i)
    if (!plan_length(pl->m[i], &pl->P[i], &pl->R1[i], &pl->R2[i], &c[i])) return false;
  const size_t rows = sizeof(double2) * pl->m[0] * pl->m[1] * pl->P[2], plane = sizeof(double2) * pl->P[0] * pl->P[1];
  // planes a batch: enough items for the CTA's 256 threads in the pass with the fewest (P1 P2 / 16 a plane), and no
  // more shared memory than leaves room for a second CTA where the rows alone do
  int batch = (int)std::max<long>(1, (256L * 16 + pl->P[0] * pl->P[1] - 1) / (pl->P[0] * pl->P[1]));
  batch = std::min(batch, pl->P[2]);
  const size_t room = rows + plane <= 110 * 1024 ? 110 * 1024 : kFft64Smem;
  while (batch > 1 && rows + batch * plane > room) --batch;
  if (rows + batch * plane > kFft64Smem) return false;
  // equal batches
  const int nb = (pl->P[2] + batch - 1) / batch;
  pl->batch = (pl->P[2] + nb - 1) / nb;
  pl->smem = rows + pl->batch * plane;
  if (per_column)
    *per_column = 2.0 * pl->m[0] * pl->m[1] * c[2] + pl->P[2] * (2.0 * pl->m[0] * c[1] + 2.0 * pl->P[1] * c[0]) +
                  4.0 * pl->P[0] * pl->P[1] * pl->P[2];
  return true;
}

size_t fft64_spec_size(const Fft64Plan& pl) { return (size_t)pl.P[0] * pl.P[1] * pl.P[2]; }

size_t fft64_work_size(const Fft64Plan& pl) {
  return (size_t)(2 * pl.m[0] - 1) * (2 * pl.m[1] - 1 + pl.P[1]) * pl.P[2];
}

cudaError_t launch_fft64_spectrum(const Fft64Plan& pl, const double* stencil, zd* work, zd* spec, cudaStream_t s) {
  const int L1 = 2 * pl.m[0] - 1, L2 = 2 * pl.m[1] - 1;
  d2* sp = reinterpret_cast<d2*>(spec);
  d2* wk = reinterpret_cast<d2*>(work);
  d2* wk2 = wk + (size_t)L1 * L2 * pl.P[2];
  auto grid = [](long n) { return (unsigned)((n + 127) / 128); };
  // stencil [L1][L2][L3] -> [L1][L2][P3] -> [L1][P2][P3] -> spec [P1][P2][P3]
  fft64_spec_kernel<<<grid((long)L1 * L2 * pl.P[2]), 128, 0, s>>>(stencil, 1, L1 * L2, 1, pl.m[2], pl.P[2], pl.R1[2],
                                                                  pl.R2[2], 1.0, wk);
  ++g_launch_count;
  fft64_spec_kernel<<<grid((long)L1 * pl.P[1] * pl.P[2]), 128, 0, s>>>(
      reinterpret_cast<const double*>(wk), 0, L1, pl.P[2], pl.m[1], pl.P[1], pl.R1[1], pl.R2[1], 1.0, wk2);
  ++g_launch_count;
  fft64_spec_kernel<<<grid((long)pl.P[0] * pl.P[1] * pl.P[2]), 128, 0, s>>>(
      reinterpret_cast<const double*>(wk2), 0, 1, pl.P[1] * pl.P[2], pl.m[0], pl.P[0], pl.R1[0], pl.R2[0],
      1.0 / ((double)pl.P[0] * pl.P[1] * pl.P[2]), sp);
  ++g_launch_count;
  return cudaGetLastError();
}

cudaError_t launch_fft64_conv(const Fft64Plan& pl, const double* Z, int ldz, int npairs, const zd* spec, double* T,
                              int ldt, cudaStream_t s) {
  if (npairs < 1) return cudaSuccess;
  if (ldt & 1) return cudaErrorInvalidValue;
  cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(fft64_conv_kernel), pl.smem);
  if (e != cudaSuccess) return e;
  // small meshes: no more threads than the largest pass has items
  const long a = (long)pl.m[0] * pl.m[1] * pl.R1[2], b = (long)pl.batch * pl.P[1] * pl.R1[0];
  const int nt = (int)std::min(256L, (std::max(a, b) + 31) / 32 * 32);
  fft64_conv_kernel<<<npairs, nt, pl.smem, s>>>(pl, Z, ldz, reinterpret_cast<const d2*>(spec), T, ldt);
  ++g_launch_count;
  return cudaGetLastError();
}

}  // namespace wtb
