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
// k2 mod R2 in slot (k1, k2), with no twiddle factors at all; other factors run with twiddles between them (96 = 8 x 12
// for 48 points).  The frequencies stay in that order; the spectrum is stored in it.  Half of a transform's input is
// zero and half of its output unused: where the first factor is 2, 4, 8, 10 or 16 and the mesh at most P / 2 long, of
// the two elements that its first radix-2 stage would add, one is always zero, whatever the second factor's index, so
// that stage takes sign changes only (and its inverse one addition of two).  At 60 x 60 a column takes about 0.78 M
// FP64 instructions where the product takes 26 M.
//
// One CTA per complex column.  The mesh is taken as m1 x m2 x m3 with unit dimensions dropped (2D: m2 = 1):
//   A. rows: DFT over the innermost dimension, m1 m2 rows of P3 slots in shared memory;
//   B. batches of the P3 planes (2D: columns): plane to a P1 x P2 scratch, DFT over dimension 2, over dimension 1,
//      times S, inverse over dimension 1, over dimension 2; the m1 x m2 results on the mesh go back to the rows;
//   C. inverse rows; the m3 results on the mesh go to T.
// The second factor of dimension 1, the product with S and the inverse's first factor stay in registers.
// Measured per 16-column application: 2.45 ms at 48 x 45, w = 12 (2,304 columns of 0.52 M FP64 instructions; the FP64
// pipe busy 79 % of the cycles; without the pruned stages and 96 points 3.04 ms of 0.61 M; the product 37.3 ms), 4.20 ms
// at 11^3, w = 16 (4.48 and 24.5 ms).
//
// All rows of a column stay in one CTA's shared memory, so a mesh has a plan up to 80 x 80 (60 x 113, 120 x 56), 18^3 and
// 120 points in one dimension; larger ones take the product.
#include "wtb_internal.h"

#include <algorithm>
#include <numeric>
#include <vector>

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

__device__ __forceinline__ d2 neg_if(d2 a, bool neg) {  // on the sign bits: no FP64 instruction
  const int f = neg ? (int)0x80000000 : 0;
  return D(__hiloint2double(__double2hiint(a.x) ^ f, __double2loint(a.x)),
           __hiloint2double(__double2hiint(a.y) ^ f, __double2loint(a.y)));
}

// times exp(-2 pi i a / R), R = 4, 8, 16
template <int R>
__device__ __forceinline__ d2 tw_const(d2 x, int a) {
  constexpr double C = 0.92387953251128675613, S = 0.38268343236508977173, Q = 0.70710678118654752440;
  switch (a * (16 / R)) {  // compile-time
    case 0: return x;
    case 1: return tw(x, C, S);
    case 2: return D(Q * (x.x + x.y), Q * (x.y - x.x));
    case 3: return tw(x, S, C);
    case 4: return mi(x);
    case 5: return tw(x, -S, C);
    case 6: return D(Q * (x.y - x.x), -Q * (x.x + x.y));
    default: return tw(x, -C, S);
  }
}

// The first factor R = 2 H of a transform of which only one element of every pair (a, a + H) is on the mesh (the pair is
// P / 2 apart, the mesh at most P / 2 long): the first radix-2 stage takes no additions.  from(a, &neg): the pair's
// element on the mesh, neg if it is the second.  to(m, X[m]).
template <int R, class L, class St>
__device__ __forceinline__ void half_in(const L& from, const St& to) {
  constexpr int H = R / 2;
  d2 e[H], o[H];
#pragma unroll
  for (int t = 0; t < H; ++t) {
    // R = 10 = 2 * 5 by the prime-factor map (e, o over t of the elements 2 t mod 10), else by twiddles
    const int a = R == 10 ? 2 * t % H : t;
    bool neg;
    e[t] = from(a, &neg);
    o[t] = neg_if(e[t], R == 10 ? neg != (2 * t >= H) : neg);
    if constexpr (R != 10) o[t] = tw_const<R>(o[t], t);
  }
  if constexpr (H > 1) {
    dft<H>(e);
    dft<H>(o);
  }
#pragma unroll
  for (int k = 0; k < H; ++k) {
    if constexpr (R == 10) {  // X[k], k = 0 or 1 mod 2 and k = t mod 5
      to(k % 2 ? k + 5 : k, e[k]);
      to(k % 2 ? k : k + 5, o[k]);
    } else {
      to(2 * k, e[k]);
      to(2 * k + 1, o[k]);
    }
  }
}
// Its inverse: from(m) = X[m], of every pair the element on the mesh.  to(a, &, value, value if it is the second).
template <int R, class L, class St>
__device__ __forceinline__ void half_out(const L& from, const St& to) {
  constexpr int H = R / 2;
  d2 e[H], o[H];
#pragma unroll
  for (int k = 0; k < H; ++k) {
    e[k] = swp(from(R == 10 ? (k % 2 ? k + 5 : k) : 2 * k));
    o[k] = swp(from(R == 10 ? (k % 2 ? k : k + 5) : 2 * k + 1));
  }
  if constexpr (H > 1) {
    dft<H>(e);
    dft<H>(o);
  }
#pragma unroll
  for (int t = 0; t < H; ++t) {
    const int a = R == 10 ? 2 * t % H : t;
    if constexpr (R != 10) o[t] = tw_const<R>(o[t], t);
    to(a, [&](bool neg) { return swp(add(e[t], neg_if(o[t], R == 10 ? neg != (2 * t >= H) : neg))); });
  }
}

// The first factor of a forward transform from the mesh, put(a, X): element a is at l = idx(a) < P, of which l < n are
// on the mesh (get(l)), the others zero.
template <class I, class L, class St>
__device__ __forceinline__ void mesh_in(int R, bool half, int P, int n, const I& idx, const L& get, const St& put) {
  if (!half) {
    any_dft<false>(
        R,
        [&](int a) {
          const int l = idx(a);
          return l < n ? get(l) : D(0.0, 0.0);
        },
        put);
    return;
  }
  const int Q = P / 2;
  auto from = [&](int a, bool* neg) {
    int l = idx(a);
    *neg = l >= Q;
    l -= *neg ? Q : 0;
    return l < n ? get(l) : D(0.0, 0.0);
  };
  switch (R) {
    case 2: half_in<2>(from, put); break;
    case 4: half_in<4>(from, put); break;
    case 8: half_in<8>(from, put); break;
    case 10: half_in<10>(from, put); break;
    default: half_in<16>(from, put); break;
  }
}
// The first factor of an inverse transform, last to run: get(a), put(l, x) for the elements on the mesh.
template <class I, class L, class St>
__device__ __forceinline__ void mesh_out(int R, bool half, int P, int n, const I& idx, const L& get, const St& put) {
  if (!half) {
    any_dft<true>(R, get, [&](int a, d2 v) {
      const int l = idx(a);
      if (l < n) put(l, v);
    });
    return;
  }
  const int Q = P / 2;
  auto to = [&](int a, const auto& value) {
    int l = idx(a);
    const bool neg = l >= Q;
    l -= neg ? Q : 0;
    if (l < n) put(l, value(neg));
  };
  switch (R) {
    case 2: half_out<2>(get, to); break;
    case 4: half_out<4>(get, to); break;
    case 8: half_out<8>(get, to); break;
    case 10: half_out<10>(get, to); break;
    default: half_out<16>(get, to); break;
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

// slot (a, b) of a transform with the strides sa, sb of its factors
__device__ __forceinline__ int slot_of(int a, int b, int sa, int sb, int P) {
  const int t = sa * a + sb * b;
  return t < P ? t : t - P;
}

__global__ void __launch_bounds__(256) fft64_conv_kernel(Fft64Plan pl, const double* __restrict__ Z, int ldz,
                                                         const d2* __restrict__ spec, double* __restrict__ T, int ldt) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int m1 = pl.m[0], m2 = pl.m[1], m3 = pl.m[2], nrow = m1 * m2;
  const int P1 = pl.P[0], P2 = pl.P[1], P3 = pl.P[2];
  const int A1 = pl.R1[0], B1 = pl.R2[0], A2 = pl.R1[1], B2 = pl.R2[1], A3 = pl.R1[2], B3 = pl.R2[2];
  const int C1 = pl.ct[0] ? 1 : A1, C2 = pl.ct[1] ? 1 : A2, C3 = pl.ct[2] ? 1 : A3;  // the second factors' strides
  d2* Sb = reinterpret_cast<d2*>(smem_raw);  // [nrow][P3]
  d2* G = Sb + nrow * P3;                    // [batch][P1][P2]
  d2* tw1 = G + pl.batch * P1 * P2;          // the twiddle tables of the dimensions that have one
  d2* tw2 = tw1 + (pl.ct[0] ? P1 : 0);
  d2* tw3 = tw2 + (pl.ct[1] ? P2 : 0);
  const int tid = threadIdx.x, nt = blockDim.x, q = blockIdx.x;
  {
    const d2* table = spec + (size_t)P1 * P2 * P3;
    if (pl.ct[0])
      for (int i = tid; i < P1; i += nt) tw1[i] = table[i];
    if (pl.ct[1])
      for (int i = tid; i < P2; i += nt) tw2[i] = table[P1 + i];
    if (pl.ct[2])
      for (int i = tid; i < P3; i += nt) tw3[i] = table[P1 + P2 + i];
    if (pl.ct[0] || pl.ct[1] || pl.ct[2]) __syncthreads();
  }
  auto fwd = [](const d2* t, bool ct, int i, d2 v) {
    if (!ct) return v;
    const d2 w = t[i];
    return tw(v, w.x, w.y);
  };
  auto inv = [](const d2* t, bool ct, int i, d2 v) {
    if (!ct) return v;
    const d2 w = t[i];
    return D(fma(-w.y, v.y, w.x * v.x), fma(w.y, v.x, w.x * v.y));
  };
  const double* zre = Z + (size_t)(2 * q) * ldz;
  const double* zim = zre + ldz;
  // A. rows: over a (from global memory), then over b
  for (int it = tid; it < nrow * B3; it += nt) {
    const int b = it % B3, r = it / B3;
    d2* row = Sb + r * P3;
    const double *pr = zre + r * m3, *pi = zim + r * m3;
    mesh_in(
        A3, pl.half[2], P3, m3, [&](int a) { return slot_of(a, b, B3, C3, P3); },
        [&](int l) { return D(pr[l], pi[l]); },
        [&](int a, d2 v) { row[slot_of(a, b, B3, C3, P3)] = fwd(tw3, pl.ct[2], a * b, v); });
  }
  __syncthreads();
  if (B3 > 1) {
    for (int it = tid; it < nrow * A3; it += nt) {
      const int a = it % A3;
      d2* row = Sb + (it / A3) * P3;
      any_dft<false>(
          B3, [&](int b) { return row[slot_of(a, b, B3, C3, P3)]; },
          [&](int b, d2 v) { row[slot_of(a, b, B3, C3, P3)] = v; });
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
        mesh_in(
            A2, pl.half[1], P2, m2, [&](int a) { return slot_of(a, b, B2, C2, P2); },
            [&](int j) { return Sb[(i * m2 + j) * P3 + w0 + p]; },
            [&](int a, d2 v) { row[slot_of(a, b, B2, C2, P2)] = fwd(tw2, pl.ct[1], a * b, v); });
      }
      __syncthreads();
      if (B2 > 1) {
        for (int it = tid; it < np * m1 * A2; it += nt) {
          const int p = it % np, t = it / np, a = t % A2, i = t / A2;
          d2* row = G + p * PP + i * P2;
          any_dft<false>(
              B2, [&](int b) { return row[slot_of(a, b, B2, C2, P2)]; },
              [&](int b, d2 v) { row[slot_of(a, b, B2, C2, P2)] = v; });
        }
        __syncthreads();
      }
    }
    const bool two = P2 > 1;
    if (B1 > 1) {
      // columns: over a, from the mesh rows (the others are zero).  With P2 > 1 the mesh elements of an item are among
      // its own slots in G (of a pair's two, both are slots of the same b)
      for (int it = tid; it < np * P2 * B1; it += nt) {
        const int p = it % np, t = it / np, v = t % P2, b = t / P2;
        d2* col = G + p * PP + v;
        mesh_in(
            A1, pl.half[0], P1, m1, [&](int a) { return slot_of(a, b, B1, C1, P1); },
            [&](int i) { return two ? col[i * P2] : Sb[i * P3 + w0 + p]; },
            [&](int a, d2 x) { col[slot_of(a, b, B1, C1, P1) * P2] = fwd(tw1, pl.ct[0], a * b, x); });
      }
      __syncthreads();
      // over b, times the spectrum, inverse over b
      for (int it = tid; it < np * P2 * A1; it += nt) {
        const int p = it % np, t = it / np, v = t % P2, a = t / P2;
        d2* col = G + p * PP + v;
        const d2* sp = spec + (size_t)v * P3 + w0 + p;
        any_mul(
            B1, [&](int b) { return col[slot_of(a, b, B1, C1, P1) * P2]; },
            [&](int b) { return sp[(size_t)slot_of(a, b, B1, C1, P1) * P2 * P3]; },
            [&](int b, d2 x) { col[slot_of(a, b, B1, C1, P1) * P2] = x; });
      }
      __syncthreads();
      // inverse over a; the mesh rows stay
      for (int it = tid; it < np * P2 * B1; it += nt) {
        const int p = it % np, t = it / np, v = t % P2, b = t / P2;
        d2* col = G + p * PP + v;
        mesh_out(
            A1, pl.half[0], P1, m1, [&](int a) { return slot_of(a, b, B1, C1, P1); },
            [&](int a) { return inv(tw1, pl.ct[0], a * b, col[slot_of(a, b, B1, C1, P1) * P2]); },
            [&](int i, d2 x) {
              if (two)
                col[i * P2] = x;
              else
                Sb[i * P3 + w0 + p] = x;
            });
      }
      __syncthreads();
    } else {  // P1 = A1: the whole column in registers
      for (int it = tid; it < np * P2; it += nt) {
        const int p = it % np, v = it / np;
        d2* col = G + p * PP + v;
        const d2* sp = spec + (size_t)v * P3 + w0 + p;
        any_mul(
            A1, [&](int i) { return i < m1 ? (two ? col[i * P2] : Sb[i * P3 + w0 + p]) : D(0.0, 0.0); },
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
              B2, [&](int b) { return row[slot_of(a, b, B2, C2, P2)]; },
              [&](int b, d2 v) { row[slot_of(a, b, B2, C2, P2)] = v; });
        }
        __syncthreads();
      }
      for (int it = tid; it < np * m1 * B2; it += nt) {
        const int p = it % np, t = it / np, b = t % B2, i = t / B2;
        const d2* row = G + p * PP + i * P2;
        mesh_out(
            A2, pl.half[1], P2, m2, [&](int a) { return slot_of(a, b, B2, C2, P2); },
            [&](int a) { return inv(tw2, pl.ct[1], a * b, row[slot_of(a, b, B2, C2, P2)]); },
            [&](int j, d2 v) { Sb[(i * m2 + j) * P3 + w0 + p] = v; });
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
          B3, [&](int b) { return row[slot_of(a, b, B3, C3, P3)]; },
          [&](int b, d2 v) { row[slot_of(a, b, B3, C3, P3)] = v; });
    }
    __syncthreads();
  }
  for (int it = tid; it < nrow * B3; it += nt) {
    const int b = it % B3, r = it / B3;
    const d2* row = Sb + r * P3;
    double* out = T + (size_t)r * m3 * ldt + 2 * q;
    mesh_out(
        A3, pl.half[2], P3, m3, [&](int a) { return slot_of(a, b, B3, C3, P3); },
        [&](int a) { return inv(tw3, pl.ct[2], a * b, row[slot_of(a, b, B3, C3, P3)]); },
        [&](int l, d2 v) { *reinterpret_cast<d2*>(out + (size_t)l * ldt) = v; });
  }
}

// out[o][slot][i] = scale sum_l in[o][l][i] W_P^(f(slot) (l - (n - 1))), l < 2 n - 1, f(slot) the frequency in the
// slot: one dimension of the spectrum, W_P^m from a shared table, which also goes to table (the twiddle factors of a
// transform with ct).  first: in is the real stencil.
__global__ void __launch_bounds__(128) fft64_spec_kernel(const double* __restrict__ in, int first, int outer, int inner,
                                                         int n, int P, int R1, int R2, int ct, double scale,
                                                         d2* __restrict__ out, d2* __restrict__ table) {
  __shared__ double wr[256], wi[256];
  for (int m = threadIdx.x; m < P; m += blockDim.x) {
    double sn, cs;
    sincospi(2.0 * m / P, &sn, &cs);
    wr[m] = cs;
    wi[m] = -sn;
    if (blockIdx.x == 0) table[m] = D(cs, sn);
  }
  __syncthreads();
  const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long)outer * P * inner) return;
  const int i = (int)(e % inner), slot = (int)((e / inner) % P);
  const long o = e / ((long)inner * P);
  // slot = (R2 k1 + R1 k2) mod P of the frequency k, k1 = k mod R1, k2 = k mod R2 (inverted by search), or with ct
  // R2 k1 + k2 of k = k1 + R1 k2
  int f = ct ? slot / R2 + R1 * (slot % R2) : 0;
  for (int k = 0; k < P && !ct; ++k)
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

// The time of a plan in FP64 instructions at the pipe's rate: 0.556 of its instructions and this for every R-point DFT.
// Fitted (root mean square error 4.5 %) to the measured times of 717 plans of ten meshes, 7^3 to 48 x 45: large powers
// of two keep the pipe busiest, 3, 5, 10 and 15 points least.
double dft_time(int R) {
  switch (R) {
    case 1: return 0.0;
    case 2: return 4.5;
    case 3: return 11.4;
    case 4: return 11.9;
    case 5: return 25.4;
    case 7: return 40.8;
    case 8: return 29.6;
    case 9: return 54.2;
    case 10: return 62.2;
    case 12: return 56.6;
    case 15: return 121.8;
    default: return 93.0;
  }
}
constexpr double kInstrTime = 0.556;

// A transform of one dimension: its length P = R1 R2, the kinds of its factors, and the FP64 instructions and the time
// of a forward and an inverse.
struct Length {
  int P = 0, R1 = 1, R2 = 1, half = 0, ct = 0;
  double cost = 0.0, time = 0.0;
};

// Lengths P >= 2 n - 1 for n mesh points, none of them both longer and slower than another.  Coprime factors need no
// twiddles; others (ct) do, P complex products each way.  half: the mesh takes at most half of P and R1 has a half
// form.
std::vector<Length> lengths(int n) {
  static const int kR[] = {16, 15, 12, 10, 9, 8, 7, 5, 4, 3, 2, 1};  // the larger factor first where two plans tie
  std::vector<Length> best;
  if (n == 1) {
    best.resize(1);
    best[0].P = 1;
    return best;
  }
  Length by_p[257];  // the cheapest of each length
  for (int a : kR)
    for (int b : kR) {
      const int P = a * b;
      // one factor alone makes one item a row and most lanes idle: up to 5 points only.  1,024 columns with and without
      // two factors in their place, of 29 meshes with a dimension of at most 8: 6 x 6 20.6 and 57.8 us, 8 x 8 24.9 and
      // 115.5, 8 x 1 10.6 and 29.0, 30 x 8 100.7 and 151.1, 4^3 63.6 and 78.2, 8^3 337 and 357, 7^3 and 24 x 24 x 2 the
      // same; only with the short one beside two longer ones a single factor is ahead, 12 x 12 x 4 422 and 380
      if (a == 1 || (b == 1 && a > 5) || P < 2 * n - 1) continue;
      const bool ct = b > 1 && std::gcd(a, b) != 1;
      long in = dft_cost(a), out = in;
      const bool half = b > 1 && 2 * n <= P && (a == 2 || a == 4 || a == 8 || a == 10 || a == 16);
      if (half) {  // two DFTs of R / 2, the twiddles between, and one addition of two per pair on the way out
        static const int kTw[] = {0, 0, 0, 0, 0, 0, 0, 0, 8, 0, 0, 0, 0, 0, 0, 0, 24};
        in = 2 * dft_cost(a / 2) + kTw[a];
        out = in + a;
      }
      Length x;
      x.P = P;
      x.R1 = a;
      x.R2 = b;
      x.half = half ? 1 : 0;
      x.ct = ct ? 1 : 0;
      x.cost = (double)b * (in + out) + 2.0 * a * dft_cost(b) + (ct ? 8.0 * P : 0.0);
      x.time = kInstrTime * x.cost + 2.0 * b * dft_time(a) + 2.0 * a * dft_time(b);
      if (by_p[P].P == 0 || x.time < by_p[P].time) by_p[P] = x;
    }
  for (const Length& x : by_p)
    if (x.P && (best.empty() || x.time < best.back().time)) best.push_back(x);
  return best;
}

constexpr size_t kFft64Smem = 220 * 1024;   // dynamic shared memory of one CTA at most
constexpr size_t kFft64Smem2 = 110 * 1024;  // of one of two CTAs an SM
constexpr int kFft64Mesh = 120;             // mesh points of a dimension at most

// Batches of planes and shared memory for the lengths in pl; false where they do not fit.
bool fft64_batches(Fft64Plan* pl) {
  size_t rows = sizeof(double2) * pl->m[0] * pl->m[1] * pl->P[2];
  const size_t plane = sizeof(double2) * pl->P[0] * pl->P[1];
  for (int i = 0; i < 3; ++i)
    if (pl->ct[i]) rows += sizeof(double2) * pl->P[i];
  // planes a batch: enough items for the CTA's 256 threads in the pass with the fewest (P1 P2 / 16 a plane), and no
  // more shared memory than leaves room for a second CTA where the rows alone do
  int batch = (int)std::max<long>(1, (256L * 16 + pl->P[0] * pl->P[1] - 1) / (pl->P[0] * pl->P[1]));
  batch = std::min(batch, pl->P[2]);
  const size_t room = rows + plane <= kFft64Smem2 ? kFft64Smem2 : kFft64Smem;
  while (batch > 1 && rows + batch * plane > room) --batch;
  if (rows + batch * plane > kFft64Smem) return false;
  // equal batches
  const int nb = (pl->P[2] + batch - 1) / batch;
  pl->batch = (pl->P[2] + nb - 1) / nb;
  pl->smem = rows + pl->batch * plane;
  return true;
}

}  // namespace

// The plan of an n1 x n2 x n3 mesh, or false where the transforms do not fit one CTA (the caller then multiplies by
// the table).  *per_column: FP64 instructions of one complex column.  The lengths of the three dimensions are chosen
// together (a longer one adds transforms to the others): the least time, plans that leave an SM one CTA counted half
// as much again (its FP64 pipe idles between the passes).
bool fft64_plan(int n1, int n2, int n3, Fft64Plan* pl, double* per_column) {
  const int n[3] = {n1, n2, n3};
  int d[3], nd = 0;
  for (int i = 0; i < 3; ++i) {
    if (n[i] < 1 || n[i] > kFft64Mesh) return false;
    if (n[i] > 1) d[nd++] = n[i];
  }
  Fft64Plan t;
  t.m[0] = nd >= 2 ? d[0] : 1;
  t.m[1] = nd == 3 ? d[1] : 1;
  t.m[2] = nd >= 1 ? d[nd - 1] : 1;
  const std::vector<Length> L[3] = {lengths(t.m[0]), lengths(t.m[1]), lengths(t.m[2])};
  double best = 0.0;
  for (const Length& x : L[0])
    for (const Length& y : L[1])
      for (const Length& z : L[2]) {
        const Length* l[3] = {&x, &y, &z};
        for (int i = 0; i < 3; ++i) {
          t.P[i] = l[i]->P;
          t.R1[i] = l[i]->R1;
          t.R2[i] = l[i]->R2;
          t.half[i] = l[i]->half;
          t.ct[i] = l[i]->ct;
        }
        auto column = [&](double Length::*what, double product) {
          return (double)t.m[0] * t.m[1] * (z.*what) + z.P * ((double)t.m[0] * (y.*what) + (double)y.P * (x.*what)) +
                 product * x.P * y.P * z.P;
        };
        double time = column(&Length::time, 4.0 * kInstrTime);
        if ((best > 0.0 && time >= best) || !fft64_batches(&t)) continue;
        if (t.smem > kFft64Smem2) time *= 1.5;
        if (best == 0.0 || time < best) {
          best = time;
          *pl = t;
          if (per_column) *per_column = column(&Length::cost, 4.0);
        }
      }
  return best > 0.0;
}

// the spectrum, then the dimensions' twiddle tables
size_t fft64_spec_size(const Fft64Plan& pl) {
  return (size_t)pl.P[0] * pl.P[1] * pl.P[2] + pl.P[0] + pl.P[1] + pl.P[2];
}

size_t fft64_work_size(const Fft64Plan& pl) {
  return (size_t)(2 * pl.m[0] - 1) * (2 * pl.m[1] - 1 + pl.P[1]) * pl.P[2];
}

cudaError_t launch_fft64_spectrum(const Fft64Plan& pl, const double* stencil, zd* work, zd* spec, cudaStream_t s) {
  const int L1 = 2 * pl.m[0] - 1, L2 = 2 * pl.m[1] - 1;
  d2* sp = reinterpret_cast<d2*>(spec);
  d2* wk = reinterpret_cast<d2*>(work);
  d2* wk2 = wk + (size_t)L1 * L2 * pl.P[2];
  d2* table = sp + (size_t)pl.P[0] * pl.P[1] * pl.P[2];
  auto grid = [](long n) { return (unsigned)((n + 127) / 128); };
  // stencil [L1][L2][L3] -> [L1][L2][P3] -> [L1][P2][P3] -> spec [P1][P2][P3]
  fft64_spec_kernel<<<grid((long)L1 * L2 * pl.P[2]), 128, 0, s>>>(stencil, 1, L1 * L2, 1, pl.m[2], pl.P[2], pl.R1[2],
                                                                  pl.R2[2], pl.ct[2], 1.0, wk,
                                                                  table + pl.P[0] + pl.P[1]);
  ++g_launch_count;
  fft64_spec_kernel<<<grid((long)L1 * pl.P[1] * pl.P[2]), 128, 0, s>>>(
      reinterpret_cast<const double*>(wk), 0, L1, pl.P[2], pl.m[1], pl.P[1], pl.R1[1], pl.R2[1],
      pl.ct[1], 1.0, wk2, table + pl.P[0]);
  ++g_launch_count;
  fft64_spec_kernel<<<grid((long)pl.P[0] * pl.P[1] * pl.P[2]), 128, 0, s>>>(
      reinterpret_cast<const double*>(wk2), 0, 1, pl.P[1] * pl.P[2], pl.m[0], pl.P[0], pl.R1[0], pl.R2[0],
      pl.ct[0], 1.0 / ((double)pl.P[0] * pl.P[1] * pl.P[2]), sp, table);
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
