// qla_mfunc.cuh -- colour-matrix functions for Nc = 3 as engine OPs
// (QLA_F3/D3 M_veq_exp_M, M_veq_sqrt_M, M_veq_inverse_M, C_veq_det_M).
//
//  det, inverse: the reference's closed cofactor forms
//    (lib/perl/code-templates/C_eq_det_M.c:70-84, M_eq_inverse_M.c:79-119),
//    restated with explicitly rounded operations in the site precision:
//    bit-identical to the reference for F3 and D3.
//  sqrt: the reference's Newton iteration (M_eq_sqrt_M.c:139-180, with the
//    Gauss-Jordan solve of M_eq_M_inverse_M.c:108-135) in the site precision,
//    the template's own arithmetic (matrices in float for F3, |a|_F and the
//    stopping norm in double, FLT_EPSILON / DBL_EPSILON threshold):
//    bit-identical to QLA_F3 and QLA_D3.
//  exp: Cayley-Hamilton-reduced Taylor series with FP64 coefficients.  With
//    B = A / 2^k (|B|_F <= 1) and B^3 = c2 B^2 + c1 B + c0 1, a polynomial in B
//    is h0 1 + h1 B + h2 B^2, and B times it is h2 c0, h0 + h2 c1, h1 + h2 c2:
//    Horner's scheme on the triple (h0, h1, h2) sums the series in twelve fused
//    multiply-adds per term, with no eigenvalues involved, so nearly degenerate
//    spectra need no special case; then k squarings.  D3: all of it in FP64 (21
//    terms).  F3: only the coefficients in FP64 (16 terms); B^2, the assembly
//    and the squarings in FP32.  The reference's F3/D3 use a rational
//    approximation with scaling (M_eq_exp_M.c:302-367); agreement is checked
//    against its FP64 (D3) result.
#pragma once
#include "qla_engine.cuh"

namespace qlab {

template <typename R>
using C9 = Cx<R>[9];

__device__ __forceinline__ Cx<double> cd(Cx<float> v) { return Cx<double>{(double)v.re, (double)v.im}; }
__device__ __forceinline__ Cx<double> cd(Cx<double> v) { return v; }
template <typename R>
__device__ __forceinline__ Cx<R> cround(Cx<double> v) {
  return Cx<R>{(R)v.re, (R)v.im};
}

// explicitly rounded complex helpers (qla_complex.h order)
template <typename R>
__device__ __forceinline__ Cx<R> cmul(Cx<R> a, Cx<R> b) {  // c_eq_c_times_c
  return Cx<R>{rsub(rmul(a.re, b.re), rmul(a.im, b.im)), radd(rmul(a.re, b.im), rmul(a.im, b.re))};
}
template <typename R>
__device__ __forceinline__ void cmms(Cx<R>& c, Cx<R> a, Cx<R> b) {  // c_meq_c_times_c
  c.re = rsub(c.re, rsub(rmul(a.re, b.re), rmul(a.im, b.im)));
  c.im = rsub(c.im, radd(rmul(a.re, b.im), rmul(a.im, b.re)));
}
template <typename R>
__device__ __forceinline__ void cpms(Cx<R>& c, Cx<R> a, Cx<R> b) {  // c_peq_c_times_c
  c.re = radd(c.re, rsub(rmul(a.re, b.re), rmul(a.im, b.im)));
  c.im = radd(c.im, radd(rmul(a.re, b.im), rmul(a.im, b.re)));
}
template <typename R>
__device__ __forceinline__ R cnorm2(Cx<R> a) {
  return radd(rmul(a.re, a.re), rmul(a.im, a.im));
}

// r = a * b for 3x3 (M_eq_M_times_M order: x = 0; x += a_ik b_kj)
template <typename R>
__device__ __forceinline__ void mat3_mul(Cx<R> (&r)[9], const Cx<R> (&a)[9], const Cx<R> (&b)[9]) {
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      Cx<R> x{R(0), R(0)};
#pragma unroll
      for (int k = 0; k < 3; k++) cpms(x, a[i * 3 + k], b[k * 3 + j]);
      r[i * 3 + j] = x;
    }
}

// sum |a_ij|^2, each term in R, summed in double (the templates' maxev2)
template <typename R>
__device__ __forceinline__ double fnorm2_3(const Cx<R> (&a)[9]) {
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < 9; k++) s = __dadd_rn(s, (double)cnorm2(a[k]));
  return s;
}

// ---------------------------------------------------------------------------
// C_eq_det_M (nc = 3)
template <typename R>
__device__ __forceinline__ Cx<R> det3(const Cx<R> (&a)[9]) {
  Cx<R> det2 = cmul(a[0], a[4]);
  cmms(det2, a[1], a[3]);
  Cx<R> det1 = cmul(a[2], a[3]);
  cmms(det1, a[0], a[5]);
  Cx<R> det0 = cmul(a[1], a[5]);
  cmms(det0, a[2], a[4]);
  Cx<R> det = cmul(det2, a[8]);
  cpms(det, det1, a[7]);
  cpms(det, det0, a[6]);
  return det;
}

template <typename R_>
struct DetOp {
  using R = R_;
  static constexpr int NIN = 1, N0 = 9, N1 = 0, N2 = 0, NOUT = 1, NACC = 0;
  __device__ __forceinline__ static void apply(const SiteParams&, const Cx<R> (&a)[9], const Cx<R> (&)[1],
                                               const Cx<R> (&)[1], Cx<R> (&y)[1]) {
    y[0] = det3(a);
  }
  __device__ static void accum(const SiteParams&, const Cx<R> (&)[9], const Cx<R> (&)[1], const Cx<R> (&)[1],
                               double*) {}
  __device__ static void finish(const SiteParams&, const double*) {}
};

// ---------------------------------------------------------------------------
// M_eq_inverse_M (nc = 3): cofactors times 1/det
template <typename R>
__device__ __forceinline__ void inv3(Cx<R> (&x)[9], const Cx<R> (&a)[9]) {
  Cx<R> det2 = cmul(a[0], a[4]);
  cmms(det2, a[1], a[3]);
  Cx<R> det1 = cmul(a[2], a[3]);
  cmms(det1, a[0], a[5]);
  Cx<R> det0 = cmul(a[1], a[5]);
  cmms(det0, a[2], a[4]);
  Cx<R> det = cmul(det2, a[8]);
  cpms(det, det1, a[7]);
  cpms(det, det0, a[6]);
  // QLA_c_eq_r_div_c(idet, 1, det): t = 1/|det|^2; idet = t*conj(det)
  const R t = rdiv(R(1), cnorm2(det));
  const Cx<R> idet{rmul(t, det.re), rmul(-t, det.im)};
#define QLAB_SET(i0, j0, i1, j1, i2, j2)              \
  {                                                   \
    Cx<R> d_ = cmul(a[i1 * 3 + j1], a[i2 * 3 + j2]);  \
    cmms(d_, a[i1 * 3 + j2], a[i2 * 3 + j1]);         \
    x[i0 * 3 + j0] = cmul(d_, idet);                  \
  }
  QLAB_SET(0, 0, 1, 1, 2, 2);
  QLAB_SET(0, 1, 2, 1, 0, 2);
  x[2] = cmul(det0, idet);
  QLAB_SET(1, 0, 1, 2, 2, 0);
  QLAB_SET(1, 1, 2, 2, 0, 0);
  x[5] = cmul(det1, idet);
  QLAB_SET(2, 0, 1, 0, 2, 1);
  QLAB_SET(2, 1, 2, 0, 0, 1);
  x[8] = cmul(det2, idet);
#undef QLAB_SET
}

template <typename R_>
struct InverseOp {
  using R = R_;
  static constexpr int NIN = 1, N0 = 9, N1 = 0, N2 = 0, NOUT = 9, NACC = 0;
  __device__ __forceinline__ static void apply(const SiteParams&, const Cx<R> (&a)[9], const Cx<R> (&)[1],
                                               const Cx<R> (&)[1], Cx<R> (&x)[9]) {
    inv3(x, a);
  }
  __device__ static void accum(const SiteParams&, const Cx<R> (&)[9], const Cx<R> (&)[1], const Cx<R> (&)[1],
                               double*) {}
  __device__ static void finish(const SiteParams&, const double*) {}
};

// ---------------------------------------------------------------------------
// x = a^-1 b, Gauss-Jordan with partial pivoting (M_eq_M_inverse_M.c:108-135)
// for NB right-hand-side columns, rows swapped physically (same arithmetic
// as the template's row permutation).  Result written into d (in place of
// the right-hand side).
template <typename R, int NB = 3>
__device__ __forceinline__ void gj_solve3(Cx<R> (&c)[9], Cx<R> (&d)[3 * NB]) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    R rmax = cnorm2(c[k * 3 + k]);
    int imax = k;
#pragma unroll
    for (int i = k + 1; i < 3; i++) {
      const R rr = cnorm2(c[i * 3 + k]);
      if (rr > rmax) {
        rmax = rr;
        imax = i;
      }
    }
#pragma unroll
    for (int i = k + 1; i < 3; i++) {
      if (imax == i) {
#pragma unroll
        for (int j = 0; j < 3; j++) {
          const Cx<R> t = c[k * 3 + j];
          c[k * 3 + j] = c[i * 3 + j];
          c[i * 3 + j] = t;
        }
#pragma unroll
        for (int j = 0; j < NB; j++) {
          const Cx<R> t = d[k * NB + j];
          d[k * NB + j] = d[i * NB + j];
          d[i * NB + j] = t;
        }
      }
    }
    rmax = rdiv(R(1), rmax);
    const Cx<R> s{rmul(rmax, c[k * 3 + k].re), -rmul(rmax, c[k * 3 + k].im)};
    c[k * 3 + k] = s;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      if (i == k) continue;
      const Cx<R> t = cmul(s, c[i * 3 + k]);
#pragma unroll
      for (int j = k + 1; j < 3; j++) cmms(c[i * 3 + j], t, c[k * 3 + j]);
#pragma unroll
      for (int j = 0; j < NB; j++) cmms(d[i * NB + j], t, d[k * NB + j]);
    }
  }
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < NB; j++) d[i * NB + j] = cmul(c[i * 3 + i], d[i * NB + j]);
}

// Newton loop of M_eq_sqrt_M.c:158-171 / M_eq_invsqrt_M.c:160-173 in the
// site precision R, the templates' own arithmetic (QLA_F3 in float, QLA_D3 in
// double): e <- -1/2 e x^-1 e, x += e until |e|_F^2 <= EPS (FLT_EPSILON or
// DBL_EPSILON; the norm's terms in R, summed in double) or 20 iterations.
template <typename R>
__device__ __forceinline__ void newton_sqrt3(Cx<R> (&x)[9], Cx<R> (&e)[9]) {
  const double eps = sizeof(R) == 4 ? 1.1920928955078125e-07 : 2.220446049250313080847e-16;
  Cx<R> c[9], d[9];
  int nit = 0;
  double enorm;
  do {
    nit++;
#pragma unroll
    for (int k = 0; k < 9; k++) {
      c[k] = x[k];
      d[k] = e[k];
    }
    gj_solve3(c, d);    // d = x^-1 e
    mat3_mul(c, e, d);  // c = e x^-1 e
#pragma unroll
    for (int k = 0; k < 9; k++) {
      e[k] = Cx<R>{rmul(R(-0.5), c[k].re), rmul(R(-0.5), c[k].im)};
      x[k] = Cx<R>{radd(x[k].re, e[k].re), radd(x[k].im, e[k].im)};
    }
    enorm = fnorm2_3(e);
  } while (nit < 20 && enorm > eps);
}

// M_eq_sqrt_M in the site precision R: r = sqrt(a).  ds = |a|_F is formed in
// double and enters as (R)(1/ds) and (R)sqrt(ds), as the template's
// M_eq_d_times_M does (QLA_Real rr = d).
template <typename R>
__device__ __forceinline__ void sqrt3(Cx<R> (&r)[9], const Cx<R> (&a)[9]) {
  double ds = fnorm2_3(a);
  if (ds == 0.0) {
#pragma unroll
    for (int k = 0; k < 9; k++) r[k] = Cx<R>{R(0), R(0)};
    return;
  }
  ds = __dsqrt_rn(ds);
  Cx<R> x[9], e[9];
  const R inv = (R)__ddiv_rn(1.0, ds);
#pragma unroll
  for (int k = 0; k < 9; k++) {
    x[k] = Cx<R>{rmul(inv, a[k].re), rmul(inv, a[k].im)};  // x = a / ds
    const R dg = (k % 4 == 0) ? R(0.5) : R(0);               // e = 0.5 1 - 0.5 x
    e[k] = Cx<R>{radd(dg, rmul(R(-0.5), x[k].re)), radd(R(0), rmul(R(-0.5), x[k].im))};
    x[k] = Cx<R>{radd(x[k].re, e[k].re), radd(x[k].im, e[k].im)};
  }
  newton_sqrt3(x, e);
  const R sds = (R)__dsqrt_rn(ds);
#pragma unroll
  for (int k = 0; k < 9; k++) r[k] = Cx<R>{rmul(sds, x[k].re), rmul(sds, x[k].im)};
}

// M_eq_sqrt_M (Newton) in the site precision: bit-identical to QLA_F3 / QLA_D3
template <typename R_>
struct SqrtOp {
  using R = R_;
  static constexpr int NIN = 1, N0 = 9, N1 = 0, N2 = 0, NOUT = 9, NACC = 0;
  __device__ static void apply(const SiteParams&, const Cx<R> (&a)[9], const Cx<R> (&)[1], const Cx<R> (&)[1],
                               Cx<R> (&r)[9]) {
    sqrt3(r, a);
  }
  __device__ static void accum(const SiteParams&, const Cx<R> (&)[9], const Cx<R> (&)[1], const Cx<R> (&)[1],
                               double*) {}
  __device__ static void finish(const SiteParams&, const double*) {}
};

// plain complex arithmetic (the compiler may fuse multiply-adds): for the
// F3 exp, whose result is not tied to the reference's rounding sequence
template <typename T>
__device__ __forceinline__ Cx<T> cmul_fast(Cx<T> a, Cx<T> b) {
  return Cx<T>{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
template <typename T>
__device__ __forceinline__ void mat3_mul_fast(Cx<T> (&r)[9], const Cx<T> (&a)[9], const Cx<T> (&b)[9]) {
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      Cx<T> x = cmul_fast(a[i * 3], b[j]);
#pragma unroll
      for (int k = 1; k < 3; k++) {
        const Cx<T> t = cmul_fast(a[i * 3 + k], b[k * 3 + j]);
        x.re += t.re;
        x.im += t.im;
      }
      r[i * 3 + j] = x;
    }
}
template <typename T>
__device__ __forceinline__ Cx<T> det3_fast(const Cx<T> (&a)[9]) {
  Cx<T> m0 = cmul_fast(a[4], a[8]), m1 = cmul_fast(a[5], a[7]);
  Cx<T> n0 = cmul_fast(a[3], a[8]), n1 = cmul_fast(a[5], a[6]);
  Cx<T> o0 = cmul_fast(a[3], a[7]), o1 = cmul_fast(a[4], a[6]);
  const Cx<T> c0{m0.re - m1.re, m0.im - m1.im}, c1{n0.re - n1.re, n0.im - n1.im}, c2{o0.re - o1.re, o0.im - o1.im};
  const Cx<T> t0 = cmul_fast(a[0], c0), t1 = cmul_fast(a[1], c1), t2 = cmul_fast(a[2], c2);
  return Cx<T>{t0.re - t1.re + t2.re, t0.im - t1.im + t2.im};
}

// ---------------------------------------------------------------------------
// M_eq_exp_M: Cayley-Hamilton-reduced Taylor series (see header).  The kernel is
// bound by the FP64 pipe.  (Summing the terms from the first up, with the powers
// of B by the same recurrence, took 28 unfused operations per term instead of
// 12: F3 on 24^3 x 48 sites 49 us, 31 so.)

// 1/j! for j = 0 .. 20
__device__ __constant__ const double kInvFact[21] = {
    1.0, 1.0, 1.0 / 2.0, 1.0 / 6.0, 1.0 / 24.0, 1.0 / 120.0, 1.0 / 720.0, 1.0 / 5040.0, 1.0 / 40320.0, 1.0 / 362880.0,
    1.0 / 3628800.0, 1.0 / 39916800.0, 1.0 / 479001600.0, 1.0 / 6227020800.0, 1.0 / 87178291200.0,
    1.0 / 1307674368000.0, 1.0 / 20922789888000.0, 1.0 / 355687428096000.0, 1.0 / 6402373705728000.0,
    1.0 / 121645100408832000.0, 1.0 / 2432902008176640000.0};

// x + a b, fused
__device__ __forceinline__ Cx<double> cfma(Cx<double> a, Cx<double> b, Cx<double> x) {
  return Cx<double>{fma(a.re, b.re, fma(-a.im, b.im, x.re)), fma(a.re, b.im, fma(a.im, b.re, x.im))};
}

// f0, f1, f2 with sum_{j <= LAST} B^j / j! = f0 1 + f1 B + f2 B^2
template <int LAST>
__device__ __forceinline__ void exp_coefficients(const Cx<double> (&b)[9], Cx<double>& f0, Cx<double>& f1,
                                                 Cx<double>& f2) {
  const Cx<double> trb{b[0].re + b[4].re + b[8].re, b[0].im + b[4].im + b[8].im};
  Cx<double> trb2{0.0, 0.0};  // tr B^2 = sum_ik b_ik b_ki
#pragma unroll
  for (int i = 0; i < 3; i++) {
    trb2 = cfma(b[i * 4], b[i * 4], trb2);
#pragma unroll
    for (int k = i + 1; k < 3; k++) {
      const Cx<double> u = b[i * 3 + k], v = b[k * 3 + i];
      const Cx<double> u2{2.0 * u.re, 2.0 * u.im};
      trb2 = cfma(u2, v, trb2);
    }
  }
  // B^3 = c2 B^2 + c1 B + c0 1  (Cayley-Hamilton)
  const Cx<double> c2 = trb;
  const Cx<double> c1{-0.5 * (trb.re * trb.re - trb.im * trb.im - trb2.re), -0.5 * (2.0 * trb.re * trb.im - trb2.im)};
  const Cx<double> c0 = det3_fast(b);
  f0 = Cx<double>{kInvFact[LAST - 2], 0.0};
  f1 = Cx<double>{kInvFact[LAST - 1], 0.0};
  f2 = Cx<double>{kInvFact[LAST], 0.0};
#pragma unroll
  for (int j = LAST - 3; j >= 0; j--) {
    const Cx<double> n0 = cfma(f2, c0, Cx<double>{kInvFact[j], 0.0});
    const Cx<double> n1 = cfma(f2, c1, f0);
    f2 = cfma(f2, c2, f1);
    f0 = n0;
    f1 = n1;
  }
}

template <typename R_>
struct ExpOp {
  using R = R_;
  static constexpr int NIN = 1, N0 = 9, N1 = 0, N2 = 0, NOUT = 9, NACC = 0;
  // last power of the series: F3 B^15 (the neglected tail is below 1/16! =
  // 5e-14 of the result's scale when |B|_F <= 1), D3 B^20 (2e-20)
  static constexpr int kLast = sizeof(R) == 4 ? 15 : 20;
  __device__ static void apply(const SiteParams&, const Cx<R> (&a)[9], const Cx<R> (&)[1], const Cx<R> (&)[1],
                               Cx<R> (&r)[9]) {
    double fn = 0.0;
#pragma unroll
    for (int k = 0; k < 9; k++) fn = fma((double)a[k].im, (double)a[k].im, fma((double)a[k].re, (double)a[k].re, fn));
    // B = A / 2^ks with |B|_F^2 <= 1: fn < 2^E, so ks = ceil(E / 2) suffices
    int ks = 0;
    if (fn > 1.0) {
      const int E = ((__double2hiint(fn) >> 20) & 0x7ff) - 1022;
      ks = (E + 1) >> 1;
      if (ks > 60) ks = 60;
    }
    const R sc = (R)__hiloint2double((1023 - ks) << 20, 0);  // 2^-ks, exact
    Cx<R> b[9];
    Cx<double> bd[9];
#pragma unroll
    for (int k = 0; k < 9; k++) {
      b[k] = Cx<R>{a[k].re * sc, a[k].im * sc};
      bd[k] = cd(b[k]);
    }
    Cx<double> f0, f1, f2;
    exp_coefficients<kLast>(bd, f0, f1, f2);
    // B^2, the assembly and the squarings in the site precision
    const Cx<R> g0{(R)f0.re, (R)f0.im}, g1{(R)f1.re, (R)f1.im}, g2{(R)f2.re, (R)f2.im};
    Cx<R> b2[9];
    mat3_mul_fast(b2, b, b);
#pragma unroll
    for (int k = 0; k < 9; k++) {
      Cx<R> t = cmul_fast(g1, b[k]);
      const Cx<R> u = cmul_fast(g2, b2[k]);
      t.re += u.re;
      t.im += u.im;
      if (k % 4 == 0) {
        t.re += g0.re;
        t.im += g0.im;
      }
      r[k] = t;
    }
    for (int s = 0; s < ks; s++) {
      mat3_mul_fast(b2, r, r);
#pragma unroll
      for (int k = 0; k < 9; k++) r[k] = b2[k];
    }
  }
  __device__ static void accum(const SiteParams&, const Cx<R> (&)[9], const Cx<R> (&)[1], const Cx<R> (&)[1],
                               double*) {}
  __device__ static void finish(const SiteParams&, const double*) {}
};

}  // namespace qlab
