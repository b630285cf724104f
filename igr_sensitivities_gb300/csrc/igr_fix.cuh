// Line contractions with the LGL differentiation matrix in 64-bit block fixed
// point: the integer pipes do what the FP64 pipe is too slow for.
//
// Why: GB300 issues one FP64 warp instruction per 64 cycles and SM
// sub-partition (DADD: 76), while its integer multiply-adds (32 x 32 + 64 bit,
// about 5 cycles) and logic / shifts (2 cycles) run on other pipes at the same
// time. A P3 line (4 nodes, 14 FP64 instructions) takes 1067 cycles per warp on
// the FP64 pipe; in fixed point it takes 398, and four independent FP64
// instructions per line hide in those (412 together; measured with 16 warps
// per SM). P4 lines: 1673 against 547.
//
// Representation: the values of one line share the exponent e of their largest
// member and become integers |X| < 2^62, split as X = h 2^32 + 2 l with |h| <=
// 2^30 and a balanced l (|l| <= 2^30); the matrix is scaled by a power of two so
// that no row or column has an absolute sum above 0.7, and stored the same way.
// A product then takes three 32 x 32 -> 64 bit multiply-adds (h h, h l, l h),
// whose sums over at most five terms stay below 2^63:
//   H = sum h_D h_X,  M = sum (h_D l_X + l_D h_X),  G = H + M / 2^31.
// The low x low products and the truncation of the line's values are a few units
// of 2^-61 of the line's scale, and one rounding to nearest ends the sum: over
// random lines the results are off by 3.6e-17 rms of |D||x| where the FP64 chain
// is off by 4.8e-17. A whole SIP line (flux, transposed contraction, mass and
// face terms) has 0.2 to 0.85 times the chain's rms error (tests/test_fixed_point.py).
// No step has a mean error (ties and inexact shifts go to the odd neighbour, low
// words are balanced): a mean of half a unit, invisible in any field, made
// dJ/dalpha, a sum over the mesh, the stages and the iterations with a cancellation
// of 1e3 to 1e6, 2 to 60 times less exact than the FP64 chain's
// (tests/test_gpu_long_double.py). The cycles above were measured before that; it
// costs 8% of k2_apply and k2_apply_rev.
//
// Lines that hold infinities, NaN or values beyond 2^1007, and lines of nothing
// but subnormal-range values (below 2^-894), take the FP64 chain, as before. A
// line of zeros gives zeros, a negated line the negated result to the bit (but for a
// tie of 32 low bits).
// Lines in which an interior node leads too far take the chain for the rows that
// leave it out (fix::leads).
#pragma once
#include <cmath>

#ifdef __CUDACC__
#include <cuda_runtime.h>
#endif

namespace igrgpu {

constexpr int FIX_MAXNP = 5;

// A matrix as integers: A[i][k] = (h 2^32 + 2 l) 2^(s - 63).
struct FixMat {
  int h[FIX_MAXNP][FIX_MAXNP], l[FIX_MAXNP][FIX_MAXNP];
  int s;
};

// The FixMat of the leading np x np block of A: scaled by 2^-s so that no row or column has an absolute sum above 0.7
// (with h < 2^31 and |l| <= 2^30 this keeps M below 2^63 over five terms), rounded at 2^-63.
inline FixMat make_fix(const double A[FIX_MAXNP][FIX_MAXNP], int np) {
  FixMat F = {};
  double most = 0.0;
  for (int i = 0; i < np; ++i) {
    double r = 0.0, c = 0.0;
    for (int k = 0; k < np; ++k) { r += std::fabs(A[i][k]); c += std::fabs(A[k][i]); }
    most = std::fmax(most, std::fmax(r, c));
  }
  while (F.s < 64 && 0.7 * std::ldexp(1.0, F.s) < most) ++F.s;
  const double unit = std::ldexp(1.0, 63 - F.s);
  for (int i = 0; i < np; ++i)
    for (int k = 0; k < np; ++k) {
      const long long f = std::llrint(A[i][k] * unit);
      const long long h = (f + (1LL << 31)) >> 32;
      F.h[i][k] = (int)h;
      F.l[i][k] = (int)((f - h * (1LL << 32)) / 2);
    }
  return F;
}

namespace fix {

constexpr int E_MIN = 128, E_MAX = 2030;  // biased exponents the integer path takes
constexpr int E_FLUX = 96;                // and the least of a flux

// One instruction each on the GPU; the C forms serve host builds of this header (the unit test).
__device__ __forceinline__ long long mad(int a, int b, long long c) {
#ifdef __CUDA_ARCH__
  long long r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
#else
  return (long long)a * b + c;
#endif
}
// a >> s, 0 for s > 63 (PTX clamps the shift amount; C leaves it undefined)
__device__ __forceinline__ unsigned long long shr(unsigned long long a, unsigned s) {
#ifdef __CUDA_ARCH__
  unsigned long long r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(a), "r"(s));
  return r;
#else
  return s > 63 ? 0 : a >> s;
#endif
}
// 1 where a / 2^s is inexact, else 0; lo is a's low word, which stands for all that a shift beyond 32 bits drops
__device__ __forceinline__ unsigned inexact(unsigned lo, unsigned s) {
#ifdef __CUDA_ARCH__
  unsigned mask;
  asm("bmsk.clamp.b32 %0, 0, %1;" : "=r"(mask) : "r"(s));  // the low s bits
  return min(lo & mask, 1u);
#else
  return s != 0 && lo << (s > 32 ? 0 : 32 - s) != 0;
#endif
}
__device__ __forceinline__ int abs_hi(double v) { return __double2hiint(v) & 0x7fffffff; }

// |v| 2^(53 + PRE) / 2^(e - 1022), truncated or (ODD) to the odd neighbour; e is a biased exponent >= v's
template <int PRE, bool ODD = false>
__device__ __forceinline__ unsigned long long magnitude(double v, int e) {
  const unsigned hi = __double2hiint(v), lo = __double2loint(v);
  const unsigned m = (hi & 0xfffffu) | 0x100000u;
  const unsigned long long t = ((unsigned long long)__funnelshift_l(lo, m, PRE) << 32) | (lo << PRE);
  const unsigned s = e - ((hi & 0x7fffffffu) >> 20);
  return shr(t, s) | (ODD ? inexact((unsigned)t, s) : 0);
}

// A product drops l l of its two factors. One of them always has a balanced l (|l| <= 2^30, no mean): a mean would add up over the
// nodes and iterations behind a sum such as dJ/dalpha. The last bit of an odd t goes to the odd neighbour, like sar's (even():
// t is even, or a magnitude whose last bits are zero but for values far below the line's largest).
struct Limb { int h, l; };
__device__ __forceinline__ Limb even(long long t) { return {(int)((t + (1LL << 31)) >> 32), (int)(unsigned)t >> 1}; }
__device__ __forceinline__ Limb balanced(long long t) {
  const Limb x = even(t);
  return {x.h, x.l | ((int)(unsigned)t & 1)};
}
// v 2^62 / 2^(e - 1022) as h 2^32 + 2 l, l balanced
__device__ __forceinline__ Limb limbs(double v, int e) {
  const Limb t = even((long long)magnitude<9>(v, e));
  const int sg = (__double2hiint(v) >> 31) | 1;
  return {t.h * sg, t.l * sg};
}
// v 2^63 / 2^(e - 1022) as h 2^32 + 2 l, l of v's sign
__device__ __forceinline__ Limb factor(double v, int e) {
  const unsigned long long t = magnitude<10>(v, e);
  const int sg = (__double2hiint(v) >> 31) | 1;
  return {(int)(t >> 32) * sg, (int)((unsigned)t >> 1) * sg};
}
// a + v, v in units of 2^(53 + PRE) / 2^(e - 1022), an inexact v to the odd neighbour (see sar)
template <int PRE>
__device__ __forceinline__ long long add(long long a, double v, int e) {
  const long long s = __double2hiint(v) >> 31;
  return a + ((long long)magnitude<PRE, true>(v, e) ^ s) - s;
}

// G 2^(e - 1082) rounded to nearest, ties to even, |G| < 2^62
__device__ __forceinline__ double to_double(long long G, int e) {
  const long long sg = G >> 63;
  const unsigned long long a = (unsigned long long)((G ^ sg) - sg);
  const unsigned mh = (unsigned)(a >> 32);
  const bool z = mh == 0;
  const unsigned m = z ? (unsigned)a : mh;
  int lz = __clz(m);
  lz = z ? lz + 32 : lz;
  unsigned long long t = a << (lz - 1);  // leading bit 62
  t += 0x1ff + ((unsigned)(t >> 10) & 1);
  unsigned hi = (unsigned)(t >> 42) + (unsigned)((e + 3 - lz) << 20);  // the implicit bit adds one to the exponent
  hi |= (unsigned)(sg & 0x80000000);
  return __hiloint2double(m ? hi : 0, (unsigned)(t >> 10));
}

template <int NP>
__device__ __forceinline__ constexpr bool skip(int i, int k) { return i == k && i > 0 && i < NP - 1; }

// P1 lines stay on the FP64 chain: it is four instructions with the exact factors +-1/2, no slower than the integers
// (256 cycles) and as exact as it can be.
template <int NP>
constexpr bool F64_LINE = NP <= 2;

// FP64 needed: a value out of range, or a line of tiny values that are not all zero
template <int NP>
__device__ __forceinline__ bool out_of_range(int m, const double* v) {
  if (F64_LINE<NP>) return true;
  if ((unsigned)(m - (E_MIN << 20)) < (unsigned)((E_MAX - E_MIN) << 20)) return false;
  if (m >= (E_MAX << 20)) return true;
  unsigned any = 0;
#pragma unroll
  for (int k = 0; k < NP; ++k) any |= (unsigned)abs_hi(v[k]) | (unsigned)__double2loint(v[k]);
  return any != 0;
}
template <int NP>
__device__ __forceinline__ int max_hi(const double* v) {
  int m = abs_hi(v[0]);
#pragma unroll
  for (int k = 1; k < NP; ++k) m = max(m, abs_hi(v[k]));
  return m;
}

// A row of D or D^T leaves out its own interior node. Where that node exceeds all others by too much, units that go by the
// line's largest value are too coarse for that row on its own, and the FP64 chain runs. Up to these bounds (differences of high
// words: a factor of about 2 or 3 for rows of D, 8 for D itself unscaled and for D^T) the integer row's rms error is at most the chain's;
// at 2^4 a row of D has two to three times the chain's, and it doubles with every further power of two
// (tests/fixed_point_forms.cpp, leading).
template <int NP>
constexpr int LEAD = NP == 3 ? 1 << 20 : 3 << 19;
constexpr int LEAD_T = 3 << 20;
template <int NP, int BY>
__device__ __forceinline__ bool leads(const double* v) {
  int big = abs_hi(v[1]), next = max(abs_hi(v[0]), abs_hi(v[NP - 1]));
#pragma unroll
  for (int k = 2; k < NP - 1; ++k) {
    const int a = abs_hi(v[k]);
    next = max(next, min(big, a));
    big = max(big, a);
  }
  return big - next > BY;
}

constexpr long long HALF = 1LL << 31;  // M / 2^31 is added as 2 (M >> 32): rounded to nearest by this

// One sum of a line: coefficient (h, l)[k] by index function cf(k) -> Limb, over the terms keep(k) lets through
template <int NP, class CF, class KEEP>
__device__ __forceinline__ long long line_sum(const Limb* x, CF cf, KEEP keep, long long acc) {
  // P2's matrix has few bits: one in 32 of its M is a tie. The line's first value says which way these go, by its last bit
  // and its sign (so that the negated line gives the negated sum).
  long long H = acc, M = NP == 3 ? HALF - 1 + ((x[0].h ^ (x[0].h >> 31)) & 1) : HALF;
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    if (!keep(k)) continue;
    const Limb c = cf(k);
    H = mad(c.h, x[k].h, H);
    M = mad(c.h, x[k].l, M);
    M = mad(c.l, x[k].h, M);
  }
  return mad((int)(M >> 32), 2, H);
}

// acc + G c / 2^64 for |G| < 2^62 and c of 63 bits
__device__ __forceinline__ long long times(long long G, Limb c, long long acc = 0) {
  const Limb g = balanced(G);
  const long long M = mad(g.l, c.h, mad(g.h, c.l, HALF));
  return mad((int)(M >> 32), 2, mad(g.h, c.h, acc));
}

}  // namespace fix

// A factor every sum of a line is multiplied by, prepared once per thread.
struct FixScale {
  double d;
  fix::Limb m;  // d = (m.h 2^32 + 2 m.l) 2^(e - 1085)
  int e;
};
__device__ __forceinline__ FixScale fix_scale(double d) {
  FixScale s;
  s.d = d;
  s.e = fix::abs_hi(d) >> 20;
  s.m = fix::factor(d, s.e);
  return s;
}

// out[i] = acc[i] + c sum_k A[i][k] v[k] (T: A[k][i]) for every node of a line, rounded once. acc[i] is read only where
// has(i) (else 0), c only if SCALED (else 1). A is the FP64 matrix of F; its zero interior diagonal is skipped where
// SKIP is set. The scaled sum is the integer product of G and the factor, four more multiply-adds per node against an
// FP64 multiply's 64 cycles; a scaled line's units are 2^-60 of its scale, 2^-61 otherwise.
template <int NP, bool T, bool SKIP, bool SCALED, class MAT, class HAS>
__device__ __forceinline__ void line_op(const FixMat& F, const MAT& A, const FixScale* c, const double* v,
                                        const double* acc, HAS has, double* out) {
  const int m = fix::max_hi<NP>(v);
  int ma = 0;
#pragma unroll
  for (int i = 0; i < NP; ++i) if (has(i)) ma = max(ma, fix::abs_hi(acc[i]));
  // exponent of the sums above that of the line: |sum| < 2^(e + up - 1022)
  const int up = F.s + (SCALED ? c->e - 1022 : 0);
  const int mm = max(m, ma);
  bool slow = fix::F64_LINE<NP> || (SCALED && (unsigned)(c->e - 1022 + 256) > 512u);
  if ((unsigned)(mm - (fix::E_MIN << 20)) >= (unsigned)((fix::E_MAX - fix::E_MIN) << 20)) {
    unsigned any = 0;
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      any |= (unsigned)fix::abs_hi(v[k]) | (unsigned)__double2loint(v[k]);
      if (has(k)) any |= (unsigned)fix::abs_hi(acc[k]) | (unsigned)__double2loint(acc[k]);
    }
    slow |= any != 0;
  }
  const int e = max(max(m >> 20, (ma >> 20) - up), fix::E_MIN);
  if (SCALED) slow |= (unsigned)(e + up - 64) >= (unsigned)(fix::E_MAX - 64);
  auto row_fp64 = [&](int i, double s) {
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      if (SKIP && fix::skip<NP>(i, k)) continue;
      s = fma(T ? A[k][i] : A[i][k], v[k], s);
    }
    return s;
  };
  if (slow) {
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const double s = row_fp64(i, (has(i) && !SCALED) ? acc[i] : 0.0);
      out[i] = SCALED ? (has(i) ? fma(c->d, s, acc[i]) : c->d * s) : s;
    }
    return;
  }
  fix::Limb x[NP];
#pragma unroll
  for (int k = 0; k < NP; ++k) x[k] = fix::limbs(v[k], e);
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    const long long A0 = has(i) ? fix::add<SCALED ? 7 : 8>(0, acc[i], e + up) : 0;
    long long G = fix::line_sum<NP>(
        x, [&](int k) { return fix::Limb{T ? F.h[k][i] : F.h[i][k], T ? F.l[k][i] : F.l[i][k]}; },
        [&](int k) { return !(SKIP && fix::skip<NP>(i, k)); }, SCALED ? 0 : A0);
    if (SCALED) G = fix::times(G, c->m, A0);
    out[i] = fix::to_double(G, e + up - (SCALED ? 0 : 1));
  }
  if (fix::leads<NP, T ? fix::LEAD_T : fix::LEAD<NP>>(v)) {
#pragma unroll
    for (int i = 1; i < NP - 1; ++i) {
      if (fix::abs_hi(v[i]) != m) continue;
      const double s = row_fp64(i, 0.0), a = has(i) ? acc[i] : 0.0;
      out[i] = SCALED ? fma(c->d, s, a) : s + a;
    }
  }
}

// out[i] = sum_k D[i][k] v[k]: the reference derivative of a line at its nodes
template <int NP, class BASIS>
__device__ __forceinline__ void line_rows(const BASIS& B, const double* v, double* out) {
  line_op<NP, false, true, false>(B.fD, B.D, nullptr, v, nullptr, [](int) { return false; }, out);
}
// out[i] = c sum_k D[i][k] v[k]
template <int NP, class BASIS>
__device__ __forceinline__ void line_rows(const BASIS& B, const FixScale& c, const double* v, double* out) {
  line_op<NP, false, true, true>(B.fD, B.D, &c, v, nullptr, [](int) { return false; }, out);
}
// out[i] = acc[i] + c sum_k D[i][k] v[k]
template <int NP, class BASIS>
__device__ __forceinline__ void line_rows_acc(const BASIS& B, const FixScale& c, const double* v, const double* acc,
                                              double* out) {
  line_op<NP, false, true, true>(B.fD, B.D, &c, v, acc, [](int) { return true; }, out);
}
// ---------------------------------------------------------------------------
// A line of the SIP operator without leaving the integers: fluxes k (D x) and
// their transposed contraction, so that neither the derivatives nor the fluxes
// are rounded to doubles and taken apart again (a conversion costs 13
// instructions in, 22 out, the products and sums 4 multiply-adds each).
// ---------------------------------------------------------------------------

// The fluxes of a line: k[i] (D x)[i] = P[i] 2^(e - 1084), |P| < 2^62, and at the two end nodes as doubles. Lines outside the
// integer path's range (see line_op) hold the doubles' bits in P (slow).
template <int NP>
struct FixFlux {
  long long P[NP];
  int e;  // 0 for a line of zeros
  bool slow;
  double t0, tL;
};

namespace fix {
// v = (h 2^32 + 2 l) 2^(e - 1085), e its biased exponent (v normal)
__device__ __forceinline__ Limb mantissa(double v) {
  const unsigned hi = __double2hiint(v), lo = __double2loint(v);
  const int sg = ((int)hi >> 31) | 1;
  return {(int)__funnelshift_l(lo, (hi & 0xfffffu) | 0x100000u, 10) * sg, (int)((lo << 9) & 0x7fffffffu) * sg};
}
// a / 2^s, an inexact result rounded to its odd neighbour: as a floor it would be low by half a unit on average, which adds up
// over the nodes and iterations behind a sum such as dJ/dalpha (2 to 60 times the FP64 chain's error there).
__device__ __forceinline__ long long sar(long long a, unsigned s) {
#ifdef __CUDA_ARCH__
  long long r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(a), "r"(s));
#else
  const long long r = a >> (s > 63 ? 63 : s);
#endif
  return r | inexact((unsigned)a, s);
}
__device__ __forceinline__ bool zero(double v) { return (((unsigned)abs_hi(v)) | (unsigned)__double2loint(v)) == 0; }
// k is a coefficient the integer path takes: nonzero, finite, of moderate exponent
__device__ __forceinline__ bool plain_coef(int k_hi) { return (unsigned)(k_hi - (523 << 20)) < (unsigned)(1000 << 20); }
}  // namespace fix

// The flux at one end of a line; k is the coefficient there. It depends on nothing else, so that both sides of a face hold
// the same bits.
template <int NP, class BASIS>
__device__ __forceinline__ double flux_end(const BASIS& B, bool last, const double* x, double k) {
  const int m = fix::max_hi<NP>(x), ke = fix::abs_hi(k);
  const int ex = max(m >> 20, fix::E_MIN), e = ex + B.fD.s - 1022 + (ke >> 20);
  if (fix::out_of_range<NP>(m, x) || !fix::plain_coef(ke) || (unsigned)(e - fix::E_FLUX) >= (unsigned)(fix::E_MAX - fix::E_FLUX)) {
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < NP; ++j) s = fma(last ? B.D[NP - 1][j] : B.D[0][j], x[j], s);
    return s * k;
  }
  fix::Limb X[NP];
#pragma unroll
  for (int j = 0; j < NP; ++j) X[j] = fix::limbs(x[j], ex);
  const long long G = fix::line_sum<NP>(
      X, [&](int j) { return fix::Limb{last ? B.fD.h[NP - 1][j] : B.fD.h[0][j], last ? B.fD.l[NP - 1][j] : B.fD.l[0][j]}; },
      [](int) { return true; }, 0);
  return fix::to_double(fix::times(G, fix::mantissa(k)), e);
}

// ROWS: the fluxes serve by themselves (products). The operator's sums need no such care with x: each of them holds a flux of
// another node, whose FP64 form carries the rounding of a leading x too (measured at factors up to 2^12: 0.5 to 0.6 of the
// chain's error); a leading coefficient matters from 2^4 on.
template <int NP, bool ROWS = false, class BASIS>
__device__ __forceinline__ void flux_line(const BASIS& B, const double* x, const double* k, FixFlux<NP>& f) {
  const int m = fix::max_hi<NP>(x);
  int ke[NP], km = 0, kn = 0x7fffffff;
  bool ok = true;
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    ke[i] = fix::abs_hi(k[i]);
    ok &= fix::plain_coef(ke[i]);
    km = max(km, ke[i]);
    kn = min(kn, ke[i]);
  }
  const int ex = max(m >> 20, fix::E_MIN);
  const int eg = ex + B.fD.s - 1022;  // P_i before alignment has exponent eg + ke_i
  // Every P_i, and the line's after its shift by up to 30 below, stays where to_double's exponent cannot pass below zero.
  f.slow = fix::out_of_range<NP>(m, x) || !ok || eg + (kn >> 20) < fix::E_FLUX || eg + (km >> 20) >= fix::E_MAX ||
           (ROWS && fix::leads<NP, fix::LEAD<NP>>(x)) || (km - kn > (4 << 20) && fix::leads<NP, 4 << 20>(k));
  if (f.slow) {
    f.e = 0;
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      double g = 0.0;
#pragma unroll
      for (int j = 0; j < NP; ++j) if (!fix::skip<NP>(i, j)) g = fma(B.D[i][j], x[j], g);
      f.P[i] = __double_as_longlong(g * k[i]);
    }
    f.t0 = flux_end<NP>(B, false, x, k[0]);
    f.tL = flux_end<NP>(B, true, x, k[NP - 1]);
    return;
  }
  f.e = m == 0 ? 0 : eg + (km >> 20);
  fix::Limb X[NP];
#pragma unroll
  for (int i = 0; i < NP; ++i) X[i] = fix::limbs(x[i], ex);
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    const long long G = fix::line_sum<NP>(
        X, [&](int j) { return fix::Limb{B.fD.h[i][j], B.fD.l[i][j]}; }, [&](int j) { return !fix::skip<NP>(i, j); }, 0);
    if (i > 0 && i < NP - 1) {  // k in units of the line's largest: 63 bits, exact down to 2^-10 of it
      f.P[i] = fix::times(G, fix::factor(k[i], km >> 20));
      continue;
    }
    const long long P = fix::times(G, fix::mantissa(k[i]));
    (i == 0 ? f.t0 : f.tL) = fix::to_double(P, eg + (ke[i] >> 20));
    f.P[i] = fix::sar(P, (km >> 20) - (ke[i] >> 20));
  }
  // A smooth line's fluxes are far below what its values allow: shifted up to use their bits, so that the units of the
  // sums that follow go by the fluxes, as an FP64 sum's roundings do.
  unsigned any = 0;
#pragma unroll
  for (int i = 0; i < NP; ++i) { const int h = (int)(f.P[i] >> 32); any |= h ^ (h >> 31); }
  const int z = __clz(any) - 2;  // to |P| < 2^62
#pragma unroll
  for (int i = 0; i < NP; ++i) f.P[i] = (long long)((unsigned long long)f.P[i] << z);
  if (m != 0) f.e += 2 - z;
}

// Sums in units of 2^59 / 2^(e - 1022); e < 0: the bits of doubles (FP64 lines).
template <int NP>
struct FixSums { long long G[NP]; int e; };

// D^T (P + u0 at node 0 + uL at node NP-1) in units of at least exponent `need`, the largest exponent of what the
// caller adds; all_zero: the caller adds zeros only. False (nothing formed) where the FP64 chain has to run.
template <int NP, class BASIS>
__device__ __forceinline__ bool div_line(const BASIS& B, const FixFlux<NP>& f, double u0, double uL, int need, bool all_zero,
                                         FixSums<NP>& r) {
  const int mu = max(fix::abs_hi(u0), fix::abs_hi(uL)) >> 20;
  const int sd = B.fD.s;
  int e = max(max(f.e, mu) + sd, need);
  if (f.slow || e >= fix::E_MAX) return false;
  if (e < 192) {
    if (f.e != 0 || !fix::zero(u0) || !fix::zero(uL) || !all_zero) return false;
    e = 192;
  }
  r.e = e;
  fix::Limb S[NP];
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    long long v = fix::sar(f.P[i], e - sd - f.e + 3);
    if (i == 0) v = fix::add<6>(v, u0, e - sd);
    if (i == NP - 1) v = fix::add<6>(v, uL, e - sd);
    S[i] = fix::even(2 * v);
  }
#pragma unroll
  for (int k = 0; k < NP; ++k)
    r.G[k] = fix::line_sum<NP>(
        S, [&](int i) { return fix::Limb{B.fD.h[i][k], B.fD.l[i][k]}; }, [&](int i) { return !fix::skip<NP>(i, k); }, 0);
  return true;
}

// The same in FP64: acc[k] + sum_i D[i][k] (flux_i + u at the ends)
template <int NP, class BASIS>
__device__ __forceinline__ void div_line_fp64(const BASIS& B, const FixFlux<NP>& f, double u0, double uL, double* acc) {
  double s[NP];
#pragma unroll
  for (int i = 0; i < NP; ++i) s[i] = f.slow ? __longlong_as_double(f.P[i]) : fix::to_double(f.P[i], f.e - 2);
  s[0] += u0;
  s[NP - 1] += uL;
#pragma unroll
  for (int k = 0; k < NP; ++k)
#pragma unroll
    for (int i = 0; i < NP; ++i) if (!fix::skip<NP>(i, k)) acc[k] = fma(B.D[i][k], s[i], acc[k]);
}

// A row's sums kept between the phases: units as FixSums, e < 0: doubles.
template <int NP, class BASIS>
__device__ __forceinline__ void row_sums(const BASIS& B, const FixFlux<NP>& f, double u0, double uL, double a0, double aL,
                                         FixSums<NP>& r) {
  const int need = max(fix::abs_hi(a0), fix::abs_hi(aL)) >> 20;
  if (div_line<NP>(B, f, u0, uL, need, fix::zero(a0) && fix::zero(aL), r)) {
    r.G[0] = fix::add<6>(r.G[0], a0, r.e);
    r.G[NP - 1] = fix::add<6>(r.G[NP - 1], aL, r.e);
    return;
  }
  double acc[NP];
#pragma unroll
  for (int k = 0; k < NP; ++k) acc[k] = k == 0 ? a0 : (k == NP - 1 ? aL : 0.0);
  div_line_fp64<NP>(B, f, u0, uL, acc);
  r.e = -1;
#pragma unroll
  for (int k = 0; k < NP; ++k) r.G[k] = __double_as_longlong(acc[k]);
}

// Derivatives of a line: (D v)[i] = G[i] 2^(e - 1084), |G| < 2^62 and shifted up to use these bits; e = 0: a line of zeros; slow: the
// bits of doubles.
template <int NP>
struct FixDeriv { long long G[NP]; int e; bool slow; };

template <int NP, class BASIS>
__device__ __forceinline__ void deriv_line(const BASIS& B, const double* v, FixDeriv<NP>& d) {
  const int m = fix::max_hi<NP>(v);
  d.slow = fix::out_of_range<NP>(m, v) || fix::leads<NP, fix::LEAD_T>(v);
  d.e = 0;
  if (d.slow) {
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      double g = 0.0;
#pragma unroll
      for (int j = 0; j < NP; ++j) if (!fix::skip<NP>(i, j)) g = fma(B.D[i][j], v[j], g);
      d.G[i] = __double_as_longlong(g);
    }
    return;
  }
  const int ex = max(m >> 20, fix::E_MIN);
  fix::Limb X[NP];
#pragma unroll
  for (int i = 0; i < NP; ++i) X[i] = fix::limbs(v[i], ex);
  unsigned any = 0;
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    d.G[i] = fix::line_sum<NP>(
        X, [&](int j) { return fix::Limb{B.fD.h[i][j], B.fD.l[i][j]}; }, [&](int j) { return !fix::skip<NP>(i, j); }, 0);
    const int h = (int)(d.G[i] >> 32);
    any |= h ^ (h >> 31);
  }
  const int z = __clz(any) - 2;
#pragma unroll
  for (int i = 0; i < NP; ++i) d.G[i] = (long long)((unsigned long long)d.G[i] << z);
  if (m != 0) d.e = ex + B.fD.s + 1 - z;
}
template <int NP>
__device__ __forceinline__ double deriv_at(const FixDeriv<NP>& d, int i) {
  return d.slow ? __longlong_as_double(d.G[i]) : fix::to_double(d.G[i], d.e - 2);
}
template <int NP>
__device__ __forceinline__ double flux_at(const FixFlux<NP>& f, int i) {
  return f.slow ? __longlong_as_double(f.P[i]) : fix::to_double(f.P[i], f.e - 2);
}

// The products flux_i (D v)_i, with z0 and zL added at the end nodes, in units of 2^60 / 2^(r.e - 1022) (r.e < 0: the
// bits of doubles). They go by the line's largest flux and derivative and are not aligned to the operator's sums: exact by the
// line's norm (0.1 to 0.9 of the FP64 chain's rms error), not for a node far below it in both factors.
template <int NP>
__device__ __forceinline__ bool product_line(const FixFlux<NP>& f, const FixDeriv<NP>& d, double z0, double zL,
                                             FixSums<NP>& r) {
  const int mz = max(fix::abs_hi(z0), fix::abs_hi(zL)) >> 20;
  const bool none = f.e == 0 || d.e == 0;
  const int ep = none ? 0 : f.e + d.e - 1022;
  int e = max(ep, mz);
  if (f.slow || d.slow || e >= fix::E_MAX || (!none && ep < 64)) return false;
  if (e < 128) {
    if (!none || !fix::zero(z0) || !fix::zero(zL)) return false;
    e = 128;
  }
  r.e = e;
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    const fix::Limb p = fix::balanced(f.P[i]), g = fix::balanced(d.G[i]);
    const long long M = fix::mad(p.h, g.l, fix::mad(p.l, g.h, fix::HALF));
    long long v = fix::sar(fix::mad((int)(M >> 32), 2, fix::mad(p.h, g.h, 0)), e - ep);
    if (i == 0) v = fix::add<7>(v, z0, e);
    if (i == NP - 1) v = fix::add<7>(v, zL, e);
    r.G[i] = v;
  }
  return true;
}
template <int NP>
__device__ __forceinline__ void row_products(const FixFlux<NP>& f, const FixDeriv<NP>& d, double z0, double zL,
                                             FixSums<NP>& r) {
  if (product_line<NP>(f, d, z0, zL, r)) return;
  r.e = -1;
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    double v = flux_at<NP>(f, i) * deriv_at<NP>(d, i);
    if (i == 0) v += z0;
    if (i == NP - 1) v += zL;
    r.G[i] = __double_as_longlong(v);
  }
}
// acc + sg (row + column) at one node, rounded once: r and c are sums of a row and a column in units of
// 2^U / 2^(e - 1022) (e < 0: the bits of doubles).
template <int U>
__device__ __forceinline__ double node_total(long long r, int er, long long c, int ec, double acc, int sg) {
  const int e = max(max(er, ec), fix::abs_hi(acc) >> 20);
  if (er >= 0 && ec >= 0 && e >= 128 && e < fix::E_MAX) {
    const long long v = fix::sar(r, e - er) + fix::sar(c, e - ec);
    return fix::to_double(fix::add<U - 53>(sg > 0 ? v : -v, acc, e), e + 60 - U);
  }
  const double x = er < 0 ? __longlong_as_double(r) : (er < 64 ? 0.0 : fix::to_double(r, er + 60 - U));
  const double y = ec < 0 ? __longlong_as_double(c) : (ec < 64 ? 0.0 : fix::to_double(c, ec + 60 - U));
  return sg > 0 ? acc + (x + y) : acc - (x + y);
}

// c v in units of 2^62 / 2^(e - 1022), e = exponent of v + that of c - 1022 (v normal, c.e of FixScale)
__device__ __forceinline__ long long weighted(double v, const FixScale& c) {
  const fix::Limb x = fix::mantissa(v);
  // plus the mean of the dropped product of the low words, both of their factor's sign
  const long long M = fix::mad(x.h, c.m.l, fix::mad(x.l, c.m.h, fix::HALF + (x.h < 0 ? -(c.m.l >> 1) : c.m.l >> 1)));
  return fix::mad((int)(M >> 32), 2, fix::mad(x.h, c.m.h, 0));
}
// a qa + b qb + row + column at one node (units of 2^60; see node_total), rounded once; 0 < a, b <= 1
__device__ __forceinline__ double node_blend(long long r, int er, long long c, int ec, double qa, const FixScale& a, double qb,
                                             const FixScale& b) {
  const int xa = fix::abs_hi(qa) >> 20, xb = fix::abs_hi(qb) >> 20;
  const int e = max(max(er, ec), max(xa, xb));
  if (er >= 0 && ec >= 0 && e >= 128 && e < fix::E_MAX) {
    long long v = fix::sar(r, e - er) + fix::sar(c, e - ec);
    v += fix::sar(weighted(qa, a), e - (xa + a.e - 1022) + 2) + fix::sar(weighted(qb, b), e - (xb + b.e - 1022) + 2);
    return fix::to_double(v, e);
  }
  return node_total<60>(r, er, c, ec, fma(b.d, qb, a.d * qa), 1);
}

// ---------------------------------------------------------------------------
// A scaled line derivative (or its transpose, T) kept as integers, c (D v), with row_add_ends' terms at its end nodes,
// in units of 2^60 / 2^(e - 1022); r.e < 0: the bits of doubles (FP64 lines). node_total and node_blend end the sums.
// ---------------------------------------------------------------------------
// rows: the sums serve by themselves, not as a small addition to the node's value (see fix::leads)
template <int NP, bool T, class BASIS>
__device__ __forceinline__ bool scaled_line(const BASIS& B, const FixScale& c, const double* v, bool rows, FixSums<NP>& r) {
  const int m = fix::max_hi<NP>(v);
  if (fix::out_of_range<NP>(m, v) || (rows && fix::leads<NP, T ? fix::LEAD_T : fix::LEAD<NP>>(v)) || (unsigned)(c.e - 1022 + 256) > 512u) return false;
  const int ex = max(m >> 20, fix::E_MIN), e = ex + B.fD.s + c.e - 1022;
  if ((unsigned)(e - 64) >= (unsigned)(fix::E_MAX - 64)) return false;
  fix::Limb X[NP];
#pragma unroll
  for (int k = 0; k < NP; ++k) X[k] = fix::limbs(v[k], ex);
#pragma unroll
  for (int i = 0; i < NP; ++i)
    r.G[i] = fix::times(fix::line_sum<NP>(
                            X, [&](int k) { return fix::Limb{T ? B.fD.h[k][i] : B.fD.h[i][k], T ? B.fD.l[k][i] : B.fD.l[i][k]}; },
                            [&](int k) { return !fix::skip<NP>(i, k); }, 0), c.m);
  r.e = m == 0 ? 0 : e;
  return true;
}
template <int NP, bool T, class BASIS>
__device__ __forceinline__ void scaled_line_fp64(const BASIS& B, const FixScale& c, const double* v, double* out) {
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < NP; ++k) if (!fix::skip<NP>(i, k)) s = fma(T ? B.D[k][i] : B.D[i][k], v[k], s);
    out[i] = c.d * s;
  }
}
template <int NP, bool T, class BASIS>
__device__ __forceinline__ void row_scaled(const BASIS& B, const FixScale& c, const double* v, FixSums<NP>& r, bool rows = true) {
  if (scaled_line<NP, T>(B, c, v, rows, r)) return;
  double s[NP];
  scaled_line_fp64<NP, T>(B, c, v, s);
  r.e = -1;
#pragma unroll
  for (int i = 0; i < NP; ++i) r.G[i] = __double_as_longlong(s[i]);
}
// value i of such sums
template <int NP>
__device__ __forceinline__ double sums_at(const FixSums<NP>& r, int i) {
  return r.e < 0 ? __longlong_as_double(r.G[i]) : fix::to_double(r.G[i], r.e);
}
template <int NP>
__device__ __forceinline__ void row_add_ends(FixSums<NP>& r, double a0, double aL) {
  const int ma = max(fix::abs_hi(a0), fix::abs_hi(aL)) >> 20;
  const int e = max(r.e, ma);
  if (r.e >= 0 && (e == 0 || e >= 128) && e < fix::E_MAX) {  // e = 0: zeros
    const int sh = e - r.e;
#pragma unroll
    for (int i = 0; i < NP; ++i) r.G[i] = fix::sar(r.G[i], sh);
    r.e = e;
    if (e != 0) {
      r.G[0] = fix::add<7>(r.G[0], a0, e);
      r.G[NP - 1] = fix::add<7>(r.G[NP - 1], aL, e);
      return;
    }
    if (fix::zero(a0) && fix::zero(aL)) return;
    r.e = 64;  // subnormals: below
  }
  double s[NP];
#pragma unroll
  for (int i = 0; i < NP; ++i) s[i] = sums_at<NP>(r, i);
  s[0] += a0;
  s[NP - 1] += aL;
  r.e = -1;
#pragma unroll
  for (int i = 0; i < NP; ++i) r.G[i] = __double_as_longlong(s[i]);
}
}  // namespace igrgpu
