// qla_ewise.cuh -- the element-wise level-1 families: every output complex
// number depends on the same-position complex number of one or two source
// records (or of the source's adjoint / transpose) and on an optional scalar
// (a constant passed by pointer, or a per-site complex / real field):
//
//   r (eqop) a                      copy, conj, i*a, adjoint, transpose
//   r (eqop) s * b                  s complex or real constant / field, and
//                                   the conj(s), conj(b) forms
//   r = a + b, a - b, s*b + c, s*b - c
//   C / R (eqop) per-site dot products and norms (field outputs)
//   M (eqop) a b^+                  outer product of two ColorVectors
// (lib/perl/build_qla.pl:1256-1335 constant and field multiples, :403-469
// adjoint/transpose/conj copies, :1338-1420 sums and combinations,
// :2358-2460 site-local dot products; QLA complex macro forms
// include/qla_complex.h:140-460).
//
// Map ops run one thread per output complex number: consecutive threads move
// consecutive 8-B (F3) / 16-B (D3) elements of the AoS records, coalesced for
// every record type including the 1152-B DiracPropagator, which does not fit
// one thread's registers.  Each element is computed with the reference's
// macro for its (eqop, form), every multiply and add rounded separately, so
// results are bit-identical.  Local dot products run one thread per site and
// accumulate in FP64 like the reference's QLA_D temporaries.
#pragma once
#include "qla_api.cuh"
#include "qla_launch.cuh"
#include "qla_ops.cuh"

namespace qlab {

enum EwShape : int {
  EW_COPY = 0, EW_CONJ, EW_I, EW_CT, EW_CTA, EW_CAT, EW_CATA, EW_RT, EW_RTA,
  EW_PLUS, EW_MINUS, EW_RT_PLUS, EW_RT_MINUS, EW_CT_PLUS, EW_CT_MINUS
};
enum EwPerm : int { PERM_ID = 0, PERM_M = 1, PERM_P = 2 };     // source element order
enum EwScal : int { SC_NONE = 0, SC_CONST = 1, SC_FIELD = 2 };  // where the scalar comes from

struct EwParams {
  void* out;
  Opnd b, c;           // first and second field source
  Opnd s;              // per-site scalar field (one complex or one real per site)
  const int* gang;
  long long n;
  int eqop;
  const void* sptr;    // constant scalar: device pointer, or nullptr to use sre/sim
  double sre, sim;
};

// element e of a record of the source in the requested order: PERM_M reads
// the transposed 3x3 matrix, PERM_P the spin-colour transposed propagator
template <int PERM, int NE>
__device__ __forceinline__ int perm_elem(int e) {
  if constexpr (PERM == PERM_M) {
    return (e % 3) * 3 + e / 3;
  } else if constexpr (PERM == PERM_P) {
    return (e % 12) * 12 + e / 12;  // (ic,is | jc,js) -> (jc,js | ic,is)
  } else {
    return e;
  }
}

template <typename R>
__device__ __forceinline__ const Cx<R>* rec_ptr(const Opnd& o, long long k, int ne) {
  return (o.mode == OM_PTR) ? static_cast<const Cx<R>*>(o.ptrs[k]) : static_cast<const Cx<R>*>(o.base) + k * ne;
}

template <typename R, int SHAPE>
__device__ __forceinline__ Cx<R> ew_apply(int eqop, Cx<R> x, Cx<R> s, Cx<R> b, Cx<R> c) {
  // t = the value the eq form assigns; peq / meq add / subtract it with one
  // rounding per component; eqm forms are written out as the macros write them
  if constexpr (SHAPE == EW_COPY) {
    switch (eqop) {
      case EQ: return b;
      case EQM: return Cx<R>{-b.re, -b.im};
      case PEQ: return Cx<R>{radd(x.re, b.re), radd(x.im, b.im)};
      default: return Cx<R>{rsub(x.re, b.re), rsub(x.im, b.im)};
    }
  } else if constexpr (SHAPE == EW_CONJ) {
    switch (eqop) {
      case EQ: return Cx<R>{b.re, -b.im};
      case EQM: return Cx<R>{-b.re, b.im};
      case PEQ: return Cx<R>{radd(x.re, b.re), rsub(x.im, b.im)};
      default: return Cx<R>{rsub(x.re, b.re), radd(x.im, b.im)};
    }
  } else if constexpr (SHAPE == EW_I) {
    switch (eqop) {
      case EQ: return Cx<R>{-b.im, b.re};
      case EQM: return Cx<R>{b.im, -b.re};
      case PEQ: return Cx<R>{rsub(x.re, b.im), radd(x.im, b.re)};
      default: return Cx<R>{radd(x.re, b.im), rsub(x.im, b.re)};
    }
  } else if constexpr (SHAPE == EW_RT || SHAPE == EW_RTA) {
    const R tr = rmul(s.re, b.re), ti = rmul(s.re, b.im);
    const R ti_c = SHAPE == EW_RTA ? -ti : ti;  // conj(b): the imaginary part enters negated
    switch (eqop) {
      case EQ: return Cx<R>{tr, ti_c};
      case EQM: return Cx<R>{-tr, -ti_c};
      case PEQ: return SHAPE == EW_RTA ? Cx<R>{radd(x.re, tr), rsub(x.im, ti)} : Cx<R>{radd(x.re, tr), radd(x.im, ti)};
      default: return SHAPE == EW_RTA ? Cx<R>{rsub(x.re, tr), radd(x.im, ti)} : Cx<R>{rsub(x.re, tr), rsub(x.im, ti)};
    }
  } else if constexpr (SHAPE == EW_CT || SHAPE == EW_CTA || SHAPE == EW_CAT || SHAPE == EW_CATA) {
    R re, im;  // the eq-form value
    if constexpr (SHAPE == EW_CT) {
      if (eqop == EQM)
        return Cx<R>{radd(rmul(-s.re, b.re), rmul(s.im, b.im)), rsub(rmul(-s.re, b.im), rmul(s.im, b.re))};
      re = rsub(rmul(s.re, b.re), rmul(s.im, b.im));
      im = radd(rmul(s.re, b.im), rmul(s.im, b.re));
    } else if constexpr (SHAPE == EW_CTA) {  // s * conj(b)
      if (eqop == EQM)
        return Cx<R>{rsub(rmul(-s.re, b.re), rmul(s.im, b.im)), radd(rmul(-s.im, b.re), rmul(s.re, b.im))};
      re = radd(rmul(s.re, b.re), rmul(s.im, b.im));
      im = rsub(rmul(s.im, b.re), rmul(s.re, b.im));
    } else if constexpr (SHAPE == EW_CAT) {  // conj(s) * b
      if (eqop == EQM)
        return Cx<R>{rsub(rmul(-s.re, b.re), rmul(s.im, b.im)), radd(rmul(-s.re, b.im), rmul(s.im, b.re))};
      re = radd(rmul(s.re, b.re), rmul(s.im, b.im));
      im = rsub(rmul(s.re, b.im), rmul(s.im, b.re));
    } else {  // conj(s) * conj(b)
      if (eqop == EQM)
        return Cx<R>{radd(rmul(-s.re, b.re), rmul(s.im, b.im)), radd(rmul(s.re, b.im), rmul(s.im, b.re))};
      re = rsub(rmul(s.re, b.re), rmul(s.im, b.im));
      im = rsub(rmul(-s.re, b.im), rmul(s.im, b.re));
    }
    switch (eqop) {
      case EQ: return Cx<R>{re, im};
      case PEQ: return Cx<R>{radd(x.re, re), radd(x.im, im)};
      default: return Cx<R>{rsub(x.re, re), rsub(x.im, im)};
    }
  } else if constexpr (SHAPE == EW_PLUS) {
    return Cx<R>{radd(b.re, c.re), radd(b.im, c.im)};
  } else if constexpr (SHAPE == EW_MINUS) {
    return Cx<R>{rsub(b.re, c.re), rsub(b.im, c.im)};
  } else if constexpr (SHAPE == EW_RT_PLUS) {
    return Cx<R>{radd(rmul(s.re, b.re), c.re), radd(rmul(s.re, b.im), c.im)};
  } else if constexpr (SHAPE == EW_RT_MINUS) {
    return Cx<R>{rsub(rmul(s.re, b.re), c.re), rsub(rmul(s.re, b.im), c.im)};
  } else if constexpr (SHAPE == EW_CT_PLUS) {
    return Cx<R>{radd(rsub(rmul(s.re, b.re), rmul(s.im, b.im)), c.re),
                 radd(radd(rmul(s.re, b.im), rmul(s.im, b.re)), c.im)};
  } else {  // EW_CT_MINUS
    return Cx<R>{rsub(rsub(rmul(s.re, b.re), rmul(s.im, b.im)), c.re),
                 rsub(radd(rmul(s.re, b.im), rmul(s.im, b.re)), c.im)};
  }
}

template <typename R, int NE, int SHAPE, int PERM, int SCAL, bool SREAL>
__global__ void __launch_bounds__(256) ew_kernel(const EwParams p) {
  overlap_begin();
  constexpr bool TWO = SHAPE == EW_PLUS || SHAPE == EW_MINUS || SHAPE >= EW_RT_PLUS;
  const long long total = p.n * NE;
  const bool load = (p.eqop == PEQ || p.eqop == MEQ);
  Cx<R> sc{R(0), R(0)};
  if constexpr (SCAL == SC_CONST) {
    if (p.sptr) {
      if constexpr (SREAL)
        sc.re = *static_cast<const R*>(p.sptr);
      else
        sc = *static_cast<const Cx<R>*>(p.sptr);
    } else {
      sc = Cx<R>{(R)p.sre, (R)p.sim};
    }
  }
  for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    const long long i = g / NE;
    const int e = (int)(g - i * NE);
    const long long k = p.gang ? (long long)p.gang[i] : i;
    Cx<R> s = sc;
    if constexpr (SCAL == SC_FIELD) {
      if constexpr (SREAL) {
        const R* q = (p.s.mode == OM_PTR) ? static_cast<const R*>(p.s.ptrs[k]) : static_cast<const R*>(p.s.base) + k;
        s.re = *q;
      } else {
        s = *rec_ptr<R>(p.s, k, 1);
      }
    }
    const Cx<R> b = rec_ptr<R>(p.b, k, NE)[perm_elem<PERM, NE>(e)];
    Cx<R> c{R(0), R(0)};
    if constexpr (TWO) c = rec_ptr<R>(p.c, k, NE)[e];
    Cx<R>* out = static_cast<Cx<R>*>(p.out) + k * NE + e;
    const Cx<R> x = load ? *out : Cx<R>{R(0), R(0)};
    *out = ew_apply<R, SHAPE>(p.eqop, x, s, b, c);
  }
}

// Streaming form of the same map when every operand is contiguous and 16-B
// aligned, there is no gang index and no permutation: the records are one
// flat array of n*NE complex numbers, and each thread moves 16-B vectors (two
// F3 / one D3 complex number per vector, two vectors per thread).  A per-site
// scalar field (contiguous) is read for each element's site, element / NE
// (from L1: a site's elements are neighbours).  Element arithmetic is
// ew_apply, so results are identical.
template <typename R, int NE, int SHAPE, int SCAL, bool SREAL>
__global__ void __launch_bounds__(256) ew_flat_kernel(const EwParams p, long long nelem) {
  overlap_begin();
  constexpr bool TWO = SHAPE == EW_PLUS || SHAPE == EW_MINUS || SHAPE >= EW_RT_PLUS;
  constexpr int CPV = 16 / (int)sizeof(Cx<R>);  // complex numbers per 16-B vector
  constexpr int CPT = 2 * CPV;                   // per thread and step
  const bool load = (p.eqop == PEQ || p.eqop == MEQ);
  Cx<R> s{R(0), R(0)};
  if constexpr (SCAL == SC_CONST) {
    if (p.sptr) {
      if constexpr (SREAL)
        s.re = *static_cast<const R*>(p.sptr);
      else
        s = *static_cast<const Cx<R>*>(p.sptr);
    } else {
      s = Cx<R>{(R)p.sre, (R)p.sim};
    }
  }
  const Cx<R>* B = static_cast<const Cx<R>*>(p.b.base);
  const Cx<R>* C = static_cast<const Cx<R>*>(p.c.base);
  Cx<R>* O = static_cast<Cx<R>*>(p.out);
  // the scalar of element q: the constant, or the field at site q / NE
  auto scal_at = [&](long long q) -> Cx<R> {
    if constexpr (SCAL == SC_FIELD) {
      const long long site = q / NE;
      if constexpr (SREAL)
        return Cx<R>{static_cast<const R*>(p.s.base)[site], R(0)};
      else
        return static_cast<const Cx<R>*>(p.s.base)[site];
    } else {
      return s;
    }
  };
  // With a complex scalar field the loads are issued together (ld_here): left to the
  // compiler, which takes 32 registers where __ldg took 40, they come late.  Without
  // one it does better itself.  (us: QLA_F3_D_vpeq_C_times_D on 666,666 sites __ldg
  // 27, plain loads 37, so 25, on 2.8 M 126 / 161 / 124; QLA_D3_D_veq_conj_D on
  // 333,333 plain loads 19, so 21.)
  constexpr bool HERE = SCAL == SC_FIELD && !SREAL;
  auto load2 = [](const double2* q) { return HERE ? ld_here(q) : ld_in(q); };
  auto load4 = [](const float4* q) { return HERE ? ld_here(q) : ld_in(q); };
  const long long nvec = nelem / CPT;
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < nvec;
       v += (long long)gridDim.x * blockDim.x) {
    const long long g0 = v * CPT;
    Cx<R> b[CPT], c[CPT], x[CPT];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const long long q = g0 + h * CPV;
      if constexpr (sizeof(R) == 4) {
        const float4 u = load4(reinterpret_cast<const float4*>(B + q));
        b[2 * h] = Cx<R>{u.x, u.y};
        b[2 * h + 1] = Cx<R>{u.z, u.w};
        if constexpr (TWO) {
          const float4 w = load4(reinterpret_cast<const float4*>(C + q));
          c[2 * h] = Cx<R>{w.x, w.y};
          c[2 * h + 1] = Cx<R>{w.z, w.w};
        }
        if (load) {
          const float4 o = *reinterpret_cast<const float4*>(O + q);
          x[2 * h] = Cx<R>{o.x, o.y};
          x[2 * h + 1] = Cx<R>{o.z, o.w};
        }
      } else {
        const double2 u = load2(reinterpret_cast<const double2*>(B + q));
        b[h] = Cx<R>{u.x, u.y};
        if constexpr (TWO) {
          const double2 w = load2(reinterpret_cast<const double2*>(C + q));
          c[h] = Cx<R>{w.x, w.y};
        }
        if (load) {
          const double2 o = *reinterpret_cast<const double2*>(O + q);
          x[h] = Cx<R>{o.x, o.y};
        }
      }
    }
    Cx<R> y[CPT];
#pragma unroll
    for (int j = 0; j < CPT; j++)
      y[j] = ew_apply<R, SHAPE>(p.eqop, load ? x[j] : Cx<R>{R(0), R(0)}, scal_at(g0 + j), b[j], c[j]);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const long long q = g0 + h * CPV;
      if constexpr (sizeof(R) == 4)
        *reinterpret_cast<float4*>(O + q) = make_float4(y[2 * h].re, y[2 * h].im, y[2 * h + 1].re, y[2 * h + 1].im);
      else
        *reinterpret_cast<double2*>(O + q) = make_double2(y[h].re, y[h].im);
    }
  }
  // tail: the last nelem % CPT numbers, one per thread of the first block
  const long long t0 = nvec * CPT;
  if (blockIdx.x == 0 && t0 + threadIdx.x < nelem) {
    const long long q = t0 + threadIdx.x;
    const Cx<R> x = load ? O[q] : Cx<R>{R(0), R(0)};
    Cx<R> c{R(0), R(0)};
    if constexpr (TWO) c = C[q];
    O[q] = ew_apply<R, SHAPE>(p.eqop, x, scal_at(q), B[q], c);
  }
}

// Adjoint and transposed forms of colour matrices (PERM_M) on the site engine,
// for contiguous 16-B aligned operands: the transposition happens between
// registers, and every record moves once by bulk copies.  (One thread per
// element reads with a stride of a row: QLA_F3_M_veq_Ca_times_Ma on 24^3 x 48
// 19.6 us, 13-15 so.)  in[0] is the scalar field with SC_FIELD, else the matrix.
template <typename R_, int SHAPE, int SCAL, bool SREAL>
struct EwAdjointOp {
  using R = R_;
  static constexpr bool FIELD = SCAL == SC_FIELD;
  static constexpr int NIN = FIELD ? 2 : 1, N0 = FIELD ? 1 : 9, N1 = FIELD ? 9 : 0, N2 = 0, NOUT = 9, NACC = 0;
  template <int NA, int NB>
  __device__ __forceinline__ static void apply(const SiteParams& p, const Cx<R> (&x0)[NA], const Cx<R> (&x1)[NB],
                                               const Cx<R> (&)[1], Cx<R> (&y)[9]) {
    Cx<R> s{R(0), R(0)};
    if constexpr (FIELD) {
      s = x0[0];
    } else if constexpr (SCAL == SC_CONST) {
      if (!p.sptr)
        s = Cx<R>{(R)p.sval, (R)p.sval_im};
      else if constexpr (SREAL)
        s.re = *static_cast<const R*>(p.sptr);
      else
        s = *static_cast<const Cx<R>*>(p.sptr);
    }
#pragma unroll
    for (int e = 0; e < 9; e++) {
      Cx<R> b;
      if constexpr (FIELD)
        b = x1[perm_elem<PERM_M, 9>(e)];
      else
        b = x0[perm_elem<PERM_M, 9>(e)];
      y[e] = ew_apply<R, SHAPE>(p.eqop, y[e], s, b, Cx<R>{R(0), R(0)});
    }
  }
  template <int NA, int NB>
  __device__ static void accum(const SiteParams&, const Cx<R> (&)[NA], const Cx<R> (&)[NB], const Cx<R> (&)[1],
                               double*) {}
  __device__ static void finish(const SiteParams&, const double*) {}
};

// Fields of fewer sites than this stay with one thread per element: the tiles'
// pipeline takes longer to fill than such a field to move (us, per element / tiles:
// QLA_F3_M_veq_Ca_times_Ma on 3,000 sites 3.5 / 4.1, on 30,000 4.6 / 4.7, on 666,666 22
// / 14; M_veq_V_times_Va on 10,000 3.7 / 4.5, on 30,000 4.5 / 4.2).
inline bool engine_pays(int n) { return n > 128LL * device_sm_count(); }

// host side: SCAL_ARG is a pointer to the constant (host or device memory)
// for SC_CONST, ignored otherwise
template <typename R, int NE, int SHAPE, int PERM, int SCAL, bool SREAL>
inline void api_ew(const char* kid, void* r, const void* scal, Opnd s, Opnd b, Opnd c, const int* gang, int n,
                   int eqop) {
  constexpr bool TWO = SHAPE == EW_PLUS || SHAPE == EW_MINUS || SHAPE >= EW_RT_PLUS;
  if (n <= 0) return;
  if (!r || !opnd_ok(b) || (TWO && !opnd_ok(c)) || (SCAL == SC_CONST && !scal) || (SCAL == SC_FIELD && !opnd_ok(s))) {
    set_error(QLAGPU_ERR_NULLPTR, kid, "NULL argument");
    return;
  }
  EwParams p;
  std::memset(&p, 0, sizeof(p));
  p.out = r;
  p.b = b;
  p.c = c;
  p.s = s;
  p.gang = gang;
  p.n = n;
  p.eqop = eqop;
  if constexpr (SCAL == SC_CONST) {
    if (is_device_ptr(scal)) {
      p.sptr = scal;
    } else if constexpr (SREAL) {
      p.sre = (double)*static_cast<const R*>(scal);
    } else {
      p.sre = (double)static_cast<const Cx<R>*>(scal)->re;
      p.sim = (double)static_cast<const Cx<R>*>(scal)->im;
    }
  }
  if constexpr (PERM == PERM_M && NE == 9 && !TWO && !(SCAL == SC_FIELD && SREAL)) {
    if (gang == nullptr && engine_pays(n) && b.mode == OM_CONTIG && aligned16(r) && aligned16(b.base) &&
        (SCAL != SC_FIELD || (s.mode == OM_CONTIG && aligned16(s.base)))) {
      SiteParams q = make_params(n, eqop);
      q.in[0] = SCAL == SC_FIELD ? s : b;
      if (SCAL == SC_FIELD) q.in[1] = b;
      q.out = r;
      q.sptr = p.sptr;
      q.sval = p.sre;
      q.sval_im = p.sim;
      SiteLauncher<EwAdjointOp<R, SHAPE, SCAL, SREAL>>::run(q, kid);
      return;
    }
  }
  const long long total = (long long)n * NE;
  const long long cap = (long long)device_sm_count() * 16;
  const bool flat = PERM == PERM_ID && (SCAL != SC_FIELD || s.mode == OM_CONTIG) && gang == nullptr &&
                    b.mode == OM_CONTIG &&
                    (reinterpret_cast<uintptr_t>(b.base) & 15u) == 0 && (reinterpret_cast<uintptr_t>(r) & 15u) == 0 &&
                    (!TWO || (c.mode == OM_CONTIG && (reinterpret_cast<uintptr_t>(c.base) & 15u) == 0));
  if (flat) {
    constexpr int CPT = 2 * (16 / (int)sizeof(Cx<R>));
    long long grid = (total / CPT + 255) / 256;
    if (grid > cap) grid = cap;
    launch_kernel(ew_flat_kernel<R, NE, SHAPE, SCAL, SREAL>, (unsigned)(grid < 1 ? 1 : grid), 256, 0, current_stream(), p, total);
  } else {
    long long grid = (total + 255) / 256;
    if (grid > cap) grid = cap;
    launch_kernel(ew_kernel<R, NE, SHAPE, PERM, SCAL, SREAL>, (unsigned)(grid < 1 ? 1 : grid), 256, 0, current_stream(), p);
  }
  check_launch(kid);
}

// ---------------------------------------------------------------------------
// outer product M (eqop) a b^+ of two ColorVectors: on the site engine where the
// operands are contiguous and 16-B aligned (every record is moved once, by bulk
// copies; one thread per element, whose factors come from two other records,
// took 20.9 us for M_veq_V_times_Va on 24^3 x 48, so 13.0), else one thread
// per element
template <typename R_>
struct OuterOp {
  using R = R_;
  static constexpr int NIN = 2, N0 = 3, N1 = 3, N2 = 0, NOUT = 9, NACC = 0;
  __device__ __forceinline__ static void apply(const SiteParams& p, const Cx<R> (&a)[3], const Cx<R> (&b)[3],
                                               const Cx<R> (&)[1], Cx<R> (&y)[9]) {
    // c_(eqop)_c_times_ca(r, a, b): the scalar slot carries a
#pragma unroll
    for (int e = 0; e < 9; e++) y[e] = ew_apply<R, EW_CTA>(p.eqop, y[e], a[e / 3], b[e % 3], Cx<R>{R(0), R(0)});
  }
  __device__ static void accum(const SiteParams&, const Cx<R> (&)[3], const Cx<R> (&)[3], const Cx<R> (&)[1],
                               double*) {}
  __device__ static void finish(const SiteParams&, const double*) {}
};

template <typename R>
__global__ void __launch_bounds__(256) outer_kernel(const EwParams p) {
  overlap_begin();
  const long long total = p.n * 9;
  const bool load = (p.eqop == PEQ || p.eqop == MEQ);
  for (long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    const long long i = g / 9;
    const int e = (int)(g - i * 9);
    const long long k = p.gang ? (long long)p.gang[i] : i;
    const Cx<R> a = rec_ptr<R>(p.b, k, 3)[e / 3];
    const Cx<R> b = rec_ptr<R>(p.c, k, 3)[e % 3];
    Cx<R>* out = static_cast<Cx<R>*>(p.out) + k * 9 + e;
    const Cx<R> x = load ? *out : Cx<R>{R(0), R(0)};
    *out = ew_apply<R, EW_CTA>(p.eqop, x, a, b, Cx<R>{R(0), R(0)});
  }
}

template <typename R>
inline void api_outer(const char* kid, void* r, Opnd a, Opnd b, const int* gang, int n, int eqop) {
  if (n <= 0) return;
  if (!r || !opnd_ok(a) || !opnd_ok(b)) {
    set_error(QLAGPU_ERR_NULLPTR, kid, "NULL argument");
    return;
  }
  if (gang == nullptr && engine_pays(n) && a.mode == OM_CONTIG && b.mode == OM_CONTIG && aligned16(r) &&
      aligned16(a.base) && aligned16(b.base)) {
    api_map<OuterOp<R>>(kid, r, a, b, gang, n, eqop);
    return;
  }
  EwParams p;
  std::memset(&p, 0, sizeof(p));
  p.out = r;
  p.b = a;
  p.c = b;
  p.gang = gang;
  p.n = n;
  p.eqop = eqop;
  long long grid = ((long long)n * 9 + 255) / 256;
  const long long cap = (long long)device_sm_count() * 16;
  if (grid > cap) grid = cap;
  launch_kernel(outer_kernel<R>, (unsigned)(grid < 1 ? 1 : grid), 256, 0, current_stream(), p);
  check_launch(kid);
}

// ---------------------------------------------------------------------------
// site-local dot products and norms (field outputs), one thread per site
enum LdKind : int { LD_DOT = 0, LD_DOT_AA = 1, LD_ADOT = 2, LD_REDOT = 3, LD_NORM2 = 4 };
// LD_DOT    x += conj(a_e) b_e                 (X_dot_X)
// LD_DOT_AA x += conj(a_e) conj(b_perm(e))     (M_dot_Ma, P_dot_Pa)
// LD_ADOT   x += a_perm(e) b_e                 (Ma_dot_M, Pa_dot_P)
// LD_REDOT  x += Re(conj(a_e) b_e)             (re_X_dot_X)
// LD_NORM2  x += |a_e|^2                       (norm2_X)

// one term of the accumulation
template <typename R, int KIND>
__device__ __forceinline__ void ldot_term(Cx<R> ua, Cx<R> vb, double& xr, double& xi) {
  const double ur = ua.re, ui = ua.im, vr = vb.re, vi = vb.im;
  if constexpr (KIND == LD_DOT || KIND == LD_REDOT || KIND == LD_NORM2) {
    xr = __dadd_rn(xr, __dadd_rn(__dmul_rn(ur, vr), __dmul_rn(ui, vi)));
    if constexpr (KIND == LD_DOT) xi = __dadd_rn(xi, __dsub_rn(__dmul_rn(ur, vi), __dmul_rn(ui, vr)));
  } else if constexpr (KIND == LD_DOT_AA) {
    xr = __dadd_rn(xr, __dsub_rn(__dmul_rn(ur, vr), __dmul_rn(ui, vi)));
    xi = __dadd_rn(xi, __dsub_rn(__dmul_rn(-ur, vi), __dmul_rn(ui, vr)));
  } else {
    xr = __dadd_rn(xr, __dsub_rn(__dmul_rn(ur, vr), __dmul_rn(ui, vi)));
    xi = __dadd_rn(xi, __dadd_rn(__dmul_rn(ur, vi), __dmul_rn(ui, vr)));
  }
}
// the accumulation of one site: x over the elements e in order, from the
// records a and b (any memory space) of ne numbers; blk: row length of the
// permuted source
template <typename R, int KIND>
__device__ __forceinline__ void ldot_site(const Cx<R>* a, const Cx<R>* b, int ne, int blk, double& xr, double& xi) {
  xr = 0.0;
  xi = 0.0;
  if constexpr (KIND == LD_ADOT || KIND == LD_DOT_AA) {
    for (int x = 0; x < blk; x++)
#pragma unroll 3
      for (int y = 0; y < blk; y++) {
        const int e = x * blk + y, pe = y * blk + x;
        ldot_term<R, KIND>(a[KIND == LD_ADOT ? pe : e], b[KIND == LD_DOT_AA ? pe : e], xr, xi);
      }
  } else {
#pragma unroll 4
    for (int e = 0; e < ne; e++) ldot_term<R, KIND>(a[e], b[e], xr, xi);
  }
}
// The same for records read where they lie in global memory, where it matters
// how many loads of a thread are in flight and how many threads share the L1.
// Measured, us, ldot_site / so: the record length NE known at compile time, D3
// re_M_dot_pM on 1.39 M sites 143 / 104, F3 re_D_dot_pD on 2.8 M 207 / 179 (but F3
// norm2_P on 333,333 gang sites 342 / 382, F3 Ma_dot_M on 1.39 M 92 / 111: those stay
// with ldot_site); N colours not unrolled by hand, DN re_D_dot_D nc = 4 on 390,625 gang
// sites 111 / 104, M_dot_Ma 110 / 98 (but FN norm2_pD nc = 4 on 375,000 48 / 51).
template <typename R, int KIND, int NE>
__device__ __forceinline__ void ldot_scattered(const Cx<R>* a, const Cx<R>* b, int ne, int blk, double& xr,
                                               double& xi) {
  constexpr bool permuted = KIND == LD_ADOT || KIND == LD_DOT_AA;
  if constexpr (NE == 1 || (NE > 0 && !permuted && (KIND != LD_NORM2 || sizeof(R) == 8))) {
    xr = 0.0;
    xi = 0.0;
#pragma unroll 4
    for (int e = 0; e < NE; e++) ldot_term<R, KIND>(a[e], b[e], xr, xi);
  } else if (NE == 0 && (permuted ? sizeof(R) == 8 : KIND != LD_NORM2)) {
    const int rows = permuted ? blk : 1, cols = permuted ? blk : ne;
    xr = 0.0;
    xi = 0.0;
    for (int x = 0; x < rows; x++)
      for (int y = 0; y < cols; y++) {
        const int e = x * cols + y, pe = permuted ? y * blk + x : e;
        ldot_term<R, KIND>(a[KIND == LD_ADOT ? pe : e], b[KIND == LD_DOT_AA ? pe : e], xr, xi);
      }
  } else {
    ldot_site<R, KIND>(a, b, ne, blk, xr, xi);
  }
}

template <typename R, int KIND>
__device__ __forceinline__ void ldot_store(void* out, long long k, int eqop, double xr, double xi) {
  if constexpr (KIND >= LD_REDOT) {
    R* q = static_cast<R*>(out) + k;
    switch (eqop) {
      case EQ: *q = (R)xr; break;
      case EQM: *q = (R)(-xr); break;
      case PEQ: *q = (R)__dadd_rn((double)*q, xr); break;
      default: *q = (R)__dsub_rn((double)*q, xr); break;
    }
  } else {
    Cx<R>* q = static_cast<Cx<R>*>(out) + k;
    const Cx<R> t{(R)xr, (R)xi};
    switch (eqop) {
      case EQ: *q = t; break;
      case EQM: *q = Cx<R>{-t.re, -t.im}; break;
      case PEQ: *q = Cx<R>{radd(q->re, t.re), radd(q->im, t.im)}; break;
      default: *q = Cx<R>{rsub(q->re, t.re), rsub(q->im, t.im)}; break;
    }
  }
}

// one thread per site, records read where they are (gang or pointer forms)
template <typename R, int KIND, int NE>
__global__ void __launch_bounds__(256) ldot_kernel(const EwParams p, int ne, int blk) {
  overlap_begin();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < p.n;
       i += (long long)gridDim.x * blockDim.x) {
    const long long k = p.gang ? (long long)p.gang[i] : i;
    const Cx<R>* a = rec_ptr<R>(p.b, k, ne);
    const Cx<R>* b = (KIND == LD_NORM2) ? a : rec_ptr<R>(p.c, k, ne);
    double xr, xi;
    ldot_scattered<R, KIND, NE>(a, b, ne, blk, xr, xi);
    ldot_store<R, KIND>(p.out, k, p.eqop, xr, xi);
  }
}

// Contiguous operands without a gang index: a warp takes 32 sites.
// Their records come into the warp's shared-memory slots with bulk copies
// (8-B cp.async where a base is not 16-B aligned, and in partial tiles of records
// below 512 B; of P records those took longer than all the full tiles: D3 re_P_dot_P
// on 3,000 sites 24.6 us, 7.0 with a bulk copy per lane), each lane then sums its site in the reference's order from there, and the 32
// results leave as one coalesced store.  The per-site FP64 chain is short
// beside the copies of the SM's other warps, so the kernel runs at the rate of
// the copies; a block-wide tile with a barrier between copying and summing
// left three of four warps idle while it summed P records.  Where all eight
// lanes of a phase would meet on one bank (records of a multiple of 128 B) the
// slots are padded by 16 B: long records (P) then come one bulk copy per lane,
// short ones in 16-B pieces, consecutive lanes taking consecutive pieces.  The
// record length is an argument: the fixed and the N-colour libraries share the
// kernel.  Measured (before / after, us): QLA_F3_C_veq_D_dot_D on 24^3 x 48
// 29.1 / 22.1, R_veq_norm2_P on an eighth of it 30.7 / 24.5;
// QLA_FN_C_veq_D_dot_D at nc = 4 on 20^3 x 40 82 / 17.1.
__host__ __device__ inline unsigned ldot_slot(unsigned rb) { return (rb % 128u == 0u) ? rb + 16u : rb; }
template <typename R, int KIND>
__global__ void __launch_bounds__(128) ldot_tile_kernel(const EwParams p, int ne, int blk, int bulk, unsigned* err) {
  overlap_begin();
  extern __shared__ __align__(128) unsigned char ldsm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  constexpr int NOP = KIND == LD_NORM2 ? 1 : 2;
  const unsigned rb = (unsigned)ne * (unsigned)sizeof(Cx<R>), sb = ldot_slot(rb);
  unsigned char* mine = ldsm + (size_t)warp * (128u + NOP * 32u * sb);
  uint64_t* bar = reinterpret_cast<uint64_t*>(mine);
  unsigned char* slot[2] = {mine + 128, mine + 128 + (NOP - 1) * 32u * sb};
  const char* base[2] = {static_cast<const char*>(p.b.base), static_cast<const char*>(p.c.base)};
  if (lane == 0) {
    mbar_init(bar, 1);
    mbar_init_fence();
  }
  __syncwarp();
  // short padded records: 32 / per records at a time, a 16-B piece per lane
  const unsigned per = rb / 16u;
  const bool pieces = sb != rb && per <= 32u;
  const unsigned r0 = pieces ? lane / per : 0u, pc = pieces ? lane % per : 0u, rstep = pieces ? 32u / per : 1u;
  const unsigned rend = r0 < rstep ? 32u : 0u;
  const long long i0 = ((long long)blockIdx.x * nw + warp) * 32;
  if (i0 >= p.n) return;
  const int nv = p.n - i0 < 32 ? (int)(p.n - i0) : 32;
  const bool tail = nv < 32 && rb % 16u == 0u && rb >= 512u;  // one bulk copy per lane and operand
  if (bulk && (nv == 32 || tail)) {
    if (pieces && nv == 32) {
#pragma unroll
      for (int j = 0; j < NOP; j++) {
        const char* src = base[j] + i0 * rb + pc * 16u;
        for (unsigned r = r0; r < rend; r += rstep) cp_async_16(slot[j] + r * sb + pc * 16u, src + r * rb);
      }
      cp_async_wait_all();
      __syncwarp();
    } else {
      if (lane == 0) mbar_arrive_expect_tx(bar, NOP * (unsigned)nv * rb);
      __syncwarp();
#pragma unroll
      for (int j = 0; j < NOP; j++) {
        const char* src = base[j] + i0 * rb;
        if (sb != rb || tail) {
          if (lane < nv) bulk_g2s(slot[j] + lane * sb, src + lane * rb, rb, bar, policy_evict_first());
        } else if (lane == 0) {
          bulk_g2s(slot[j], src, 32u * rb, bar, policy_evict_first());
        }
      }
      const bool ok = mbar_wait_bounded(bar, 0u, err);
      if (!__all_sync(0xffffffffu, ok)) {
        mbar_wait_bounded(bar, 0u, err, 200000000ull);  // drain before the slots are released
        return;
      }
    }
  } else {
    // a partial tile of short records, or a base off a 16-B boundary: 8-B copies, or
    // 4-B ones (QLA_F_Complex is declared 8-B aligned, but a caller's array of two
    // floats per number need not be)
    const bool by8 = ((reinterpret_cast<uintptr_t>(base[0]) | reinterpret_cast<uintptr_t>(base[NOP - 1])) & 7u) == 0;
    const unsigned w = by8 ? 8u : 4u, pw = rb / w, total = (unsigned)nv * pw;
#pragma unroll
    for (int j = 0; j < NOP; j++)
      for (unsigned q = lane; q < total; q += 32u) {
        unsigned char* dst = slot[j] + (q / pw) * sb + (q % pw) * w;
        const char* src = base[j] + i0 * rb + q * w;
        if (by8)
          cp_async_8(dst, src);
        else
          cp_async_4(dst, src);
      }
    cp_async_wait_all();
    __syncwarp();
  }
  if (lane < nv) {
    double xr, xi;
    const Cx<R>* a = reinterpret_cast<const Cx<R>*>(slot[0] + lane * sb);
    const Cx<R>* b = reinterpret_cast<const Cx<R>*>(slot[NOP - 1] + lane * sb);
    if constexpr (KIND == LD_ADOT || KIND == LD_DOT_AA) {
      ldot_site<R, KIND>(a, b, ne, blk, xr, xi);
    } else if (rb % 16u == 0u) {  // the same terms in the same order, 16 B per load
      xr = 0.0;
      xi = 0.0;
      constexpr int CPV = 16 / (int)sizeof(Cx<R>);
#pragma unroll 3
      for (int v = 0; v < ne / CPV; v++) {
        Cx<R> ua[CPV], vb[CPV];
        load_rec<R, CPV>(ua, a + v * CPV);
        if constexpr (KIND != LD_NORM2) load_rec<R, CPV>(vb, b + v * CPV);
#pragma unroll
        for (int h = 0; h < CPV; h++) ldot_term<R, KIND>(ua[h], KIND == LD_NORM2 ? ua[h] : vb[h], xr, xi);
      }
    } else {
      ldot_site<R, KIND>(a, b, ne, blk, xr, xi);
    }
    ldot_store<R, KIND>(p.out, i0 + lane, p.eqop, xr, xi);
  }
}

// ne complex numbers per record (NE: the same, 0 where it is not known at compile
// time), blk: row length of a permuted source
template <typename R, int KIND, int NE>
inline void run_ldot(const char* kid, int ne, int blk, void* r, Opnd a, Opnd b, const int* gang, int n, int eqop) {
  EwParams p;
  std::memset(&p, 0, sizeof(p));
  p.out = r;
  p.b = a;
  p.c = b;
  p.gang = gang;
  p.n = n;
  p.eqop = eqop;
  constexpr int NOP = KIND == LD_NORM2 ? 1 : 2;
  const unsigned rb = (unsigned)ne * (unsigned)sizeof(Cx<R>);
  const size_t warp_bytes = 128u + NOP * 32u * (size_t)ldot_slot(rb);
  const int sms = device_sm_count();
  // Records that neighbouring lanes read from the same lines need no staging: up to
  // 24 B always, up to 48 B in small fields, where the copies' latency counts; in double
  // 48 B always, and norms of 32 B.  Measured, us, tiles / one site per thread: F norm2_C on
  // 666,666 sites 5.6 / 4.2, F3 norm2_V 6.4 / 3.7, FN norm2_V nc = 2 on 1.5 M 11.6 / 6.1,
  // on 30,000 4.6 / 3.5, DN norm2_V nc = 2 on 750,000 6.8 / 5.5, D3 V_dot_V on 333,333 7.6 /
  // 5.3, on 30,000 4.4 / 3.5; but FN H_dot_H nc = 2 (32 B) on 1.5 M 17 / 27, DN V_dot_V
  // nc = 2 (32 B) on 750,000 9.1 / 9.9, F3 norm2_H (48 B) on 666,666 7.1 / 7.5.
  const bool near = rb <= 24u || (rb <= 48u && n <= 65536) ||
                    (sizeof(R) == 8 && (rb == 48u || (KIND == LD_NORM2 && rb <= 32u)));
  // (records too long for one warp's slots -- P of many colours -- go direct)
  if (gang == nullptr && a.mode == OM_CONTIG && (KIND == LD_NORM2 || b.mode == OM_CONTIG) &&
      !near && warp_bytes <= 200u * 1024u) {
    int nw = 4;
    while (nw > 1 && nw * warp_bytes > 56u * 1024u) nw /= 2;
    const size_t smem = (size_t)nw * warp_bytes;
    const void* fn = reinterpret_cast<const void*>(&ldot_tile_kernel<R, KIND>);
    launch_smem_limit(fn, 227 * 1024);
    // one tile per warp: the copies of the blocks that follow fill the SM while
    // the present ones sum (persistent warps of two or three tiles each ended
    // unevenly: norm2_D 20 us, 13 so)
    const long long grid = ((long long)n + 32 * nw - 1) / (32 * nw);
    const int bulk = aligned16(a.base) && (KIND == LD_NORM2 || aligned16(b.base)) ? 1 : 0;
    launch_kernel(ldot_tile_kernel<R, KIND>, (unsigned)grid, 32 * nw, smem, current_stream(), p, ne, blk, bulk, device_error_word());
  } else {
    long long grid = ((long long)n + 255) / 256;
    if (grid > (long long)sms * 16) grid = (long long)sms * 16;
    launch_kernel(ldot_kernel<R, KIND, NE>, (unsigned)(grid < 1 ? 1 : grid), 256, 0, current_stream(), p, ne, blk);
  }
  check_launch(kid);
}

template <typename R, int NE, int KIND, int PERM>
inline void api_ldot(const char* kid, void* r, Opnd a, Opnd b, const int* gang, int n, int eqop) {
  if (n <= 0) return;
  if (!r || !opnd_ok(a) || (KIND != LD_NORM2 && !opnd_ok(b))) {
    set_error(QLAGPU_ERR_NULLPTR, kid, "NULL argument");
    return;
  }
  run_ldot<R, KIND, NE>(kid, NE, PERM == PERM_P ? 12 : PERM == PERM_M ? 3 : 1, r, a, b, gang, n, eqop);
}

}  // namespace qlab
