// Host build of the fixed-point line contractions (csrc/igr_fix.cuh) for
// tests/test_fixed_point.py: random and edge-case lines against long double.
// Prints one line "name ok|BAD worst" per case; worst is the error over the bound.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <initializer_list>
#include <limits>

#define __device__
#define __forceinline__ inline
static int __double2hiint(double v) { uint64_t b; std::memcpy(&b, &v, 8); return (int)(b >> 32); }
static int __double2loint(double v) { uint64_t b; std::memcpy(&b, &v, 8); return (int)b; }
static double __hiloint2double(int h, int l) {
  const uint64_t b = ((uint64_t)(uint32_t)h << 32) | (uint32_t)l;
  double v; std::memcpy(&v, &b, 8); return v;
}
static long long __double_as_longlong(double v) { long long b; std::memcpy(&b, &v, 8); return b; }
static double __longlong_as_double(long long b) { double v; std::memcpy(&v, &b, 8); return v; }
static unsigned __funnelshift_l(unsigned lo, unsigned hi, unsigned s) { return (unsigned)((((uint64_t)hi << 32) | lo) << s >> 32); }
static int __clz(unsigned m) { return m ? __builtin_clz(m) : 32; }
static int max(int a, int b) { return a > b ? a : b; }
static int min(int a, int b) { return a < b ? a : b; }
#include "../igr_sensitivities_gb300/csrc/igr_fix.cuh"
using namespace igrgpu;

struct Basis { double D[FIX_MAXNP][FIX_MAXNP]; FixMat fD; };

static Basis make(int np) {
  const double a = std::sqrt(0.2), b = std::sqrt(3.0 / 7.0);
  const double x[6][5] = {{0}, {0}, {-1, 1}, {-1, 0, 1}, {-1, -a, a, 1}, {-1, -b, 0, b, 1}};
  Basis B = {};
  double lam[5];
  for (int j = 0; j < np; ++j) {
    lam[j] = 1;
    for (int i = 0; i < np; ++i) if (i != j) lam[j] *= x[np][j] - x[np][i];
    lam[j] = 1 / lam[j];
  }
  for (int j = 0; j < np; ++j)
    for (int i = 0; i < np; ++i)
      if (i != j) { B.D[i][j] = (lam[j] / lam[i]) / (x[np][i] - x[np][j]); B.D[i][i] -= B.D[i][j]; }
  B.fD = make_fix(B.D, np);
  return B;
}

static uint64_t rs = 88172645463325252ull;
static double uni() { rs ^= rs << 13; rs ^= rs >> 7; rs ^= rs << 17; return (double)(rs >> 11) / 9007199254740992.0; }

static double value(int kind) {
  const double u = 2 * uni() - 1;
  switch (kind) {
    case 0: return u;
    case 1: return 1 + 1e-6 * u;                              // cancelling derivative
    case 2: return u * std::ldexp(1.0, (int)(80 * uni()) - 40);  // wide range within a line
    case 3: return uni() < 0.5 ? 0.0 : u;
    case 4: return std::ldexp(u, -880);                       // near the lower end of the range
    case 5: return std::ldexp(u, 1000);                       // near the upper end
    case 6: return -0.0;
    case 7: return std::ldexp(u, -1040);                      // subnormal: the FP64 chain
    default: return u * 1e307;                                // overflows or nearly so: the FP64 chain
  }
}

template <int NP> static int run() {
  const Basis B = make(NP);
  int bad = 0;
  // T: transposed; S: scaled; acc: 0 none, 1 the end nodes, 2 all
  auto check = [&](const char* name, bool T, bool S, int acc) {
    for (int kind = 0; kind <= 8; ++kind) {
      double worst = 0;
      bool ok = true;
      for (int it = 0; it < 3000; ++it) {
        double v[NP], ac[NP], out[NP];
        for (int k = 0; k < NP; ++k) v[k] = value(kind);
        const double big = std::ldexp(1.0, (int)(40 * uni()) - 20);  // accumulands above and below the line
        for (int k = 0; k < NP; ++k) ac[k] = kind == 6 ? 0.0 : value(kind == 2 ? 0 : kind) * (kind == 4 || kind >= 5 ? 1.0 : big);
        const double c = S ? (uni() < 0.5 ? -1 : 1) * std::ldexp(1 + uni(), (int)(24 * uni()) - 8) : 1.0;
        const FixScale f = fix_scale(c);
        auto has = [&](int k) { return acc == 2 || (acc == 1 && (k == 0 || k == NP - 1)); };
        if (!T && !S) line_rows<NP>(B, v, out);
        else if (!T && S && !acc) line_rows<NP>(B, f, v, out);
        else if (!T && S) line_rows_acc<NP>(B, f, v, ac, out);
        else if (S) line_op<NP, true, true, true>(B.fD, B.D, &f, v, ac, has, out);
        else line_op<NP, true, true, false>(B.fD, B.D, nullptr, v, ac, has, out);
        // the largest the sum's exponent can be, by the line and by the accumulands
        long double top = 0;
        for (int k = 0; k < NP; ++k) top = fmaxl(top, fabsl((long double)v[k]));
        top *= std::ldexp(fabs(c), B.fD.s);
        for (int k = 0; k < NP; ++k) if (has(k)) top = fmaxl(top, fabsl((long double)ac[k]));
        for (int i = 0; i < NP; ++i) {
          long double s = 0;
          for (int k = 0; k < NP; ++k)
            if (!fix::skip<NP>(i, k)) s += (long double)(T ? B.D[k][i] : B.D[i][k]) * v[k];
          s = s * c + (has(i) ? (long double)ac[i] : 0.0L);
          // one rounding of the result, and 2^-55 of the line's scale: five truncations of 2^-60 at a factor and a
          // scale within [1, 2) of their powers of two, and the same for the FP64 chain's five roundings of 2^-53
          const bool fp = NP == 2 || kind >= 7 || (S && kind == 5);  // the FP64 chain runs (scaled sums beyond 2^1007 too)
          if (kind == 7) {  // the FP64 chain itself, bit for bit
            double f64 = (!S && has(i)) ? ac[i] : 0.0;
            for (int k = 0; k < NP; ++k)
              if (!fix::skip<NP>(i, k)) f64 = std::fma(T ? B.D[k][i] : B.D[i][k], v[k], f64);
            if (S) f64 = has(i) ? std::fma(c, f64, ac[i]) : c * f64;
            ok &= out[i] == f64;
            continue;
          }
          const long double bound = fabsl(s) * 1.2e-16L + top * (fp ? 8e-16L : 2.8e-17L) + 1e-322L;
          if (fabsl(s) > 1.7e308L || !std::isfinite(out[i])) { ok &= !std::isfinite(out[i]) == (fabsl(s) > 1.7e308L) || fp; continue; }
          if (top == 0 && out[i] != 0) ok = false;
          worst = fmax(worst, (double)(fabsl(out[i] - s) / bound));
        }
      }
      ok &= worst <= 1;
      bad += !ok;
      std::printf("NP%d %s kind%d %s %.3f\n", NP, name, kind, ok ? "ok" : "BAD", worst);
    }
  };
  check("rows", false, false, 0);
  check("rows_scaled", false, true, 0);
  check("rows_scaled_acc", false, true, 2);
  check("cols_scaled", true, true, 0);
  check("cols_acc_ends", true, false, 1);
  check("cols_acc", true, false, 2);
  // fluxes k (D x) and column sums acc +- (R + D^T (flux + u) + a)
  // kinds 9..12: smooth lines 1 + d (polynomial) of ever smaller variation, with the mass and row terms of such a field
  for (int kind = 0; kind <= 12; ++kind) {
    double wf = 0, ws = 0, sum_i = 0, sum_f = 0;
    bool ok = true;
    for (int it = 0; it < 4000; ++it) {
      double x[NP], k[NP], acc[NP], out[NP], row[NP], y[NP];
      long long R[NP];
      int er[NP];
      const bool far = NP == 2 || kind == 7 || kind == 8;  // the FP64 chain
      for (int i = 0; i < NP; ++i) {
        x[i] = value(kind);
        k[i] = (0.01 + uni()) * 1e-4;
        acc[i] = kind == 6 ? 0.0 : value(kind == 2 ? 0 : kind) * 1e-3;
        row[i] = kind == 6 ? 0.0 : value(kind == 2 ? 0 : kind) * 1e-3;
      }
      double u0 = value(kind) * 1e-3, uL = value(kind) * 1e-2, a0 = value(kind) * 1e-3, aL = value(kind) * 1e-4;
      if (kind >= 9) {
        const double d = std::pow(100.0, 9 - kind), c1 = 2 * uni() - 1, c2 = 2 * uni() - 1, c3 = 2 * uni() - 1, r = 0.3 * (2 * uni() - 1);
        for (int i = 0; i < NP; ++i) {
          const double s = 2.0 * i / (NP - 1) - 1;
          x[i] = 1 + d * s * (c1 + s * (c2 + s * c3));
          k[i] = 1e-4 / (1 + r * s);
          acc[i] = x[i] * k[i] / 12;
          row[i] = d * k[i] * (2 * uni() - 1);
        }
        u0 = d * 1e-6 * (2 * uni() - 1); uL = d * 1e-6 * (2 * uni() - 1); a0 = d * 1e-4 * (2 * uni() - 1); aL = d * 1e-4 * (2 * uni() - 1);
      }
      FixFlux<NP> f;
      flux_line<NP>(B, x, k, f);
      long double top = 0, F[NP], xm = 0, km = 0;
      for (int i = 0; i < NP; ++i) { xm = fmaxl(xm, fabsl((long double)x[i])); km = fmaxl(km, fabsl((long double)k[i])); }
      for (int i = 0; i < NP; ++i) {
        long double g = 0;
        for (int j = 0; j < NP; ++j) if (!fix::skip<NP>(i, j)) g += (long double)B.D[i][j] * x[j];
        F[i] = g * k[i];
      }
      const long double rel = far ? 8e-16L : 2.8e-17L;  // as above; tiny: the subnormals' quantum through D and k
      const long double tiny = 1e-321L;
      const long double b0 = fabsl(F[0]) * 1.2e-16L + xm * ldexpl(1, B.fD.s) * k[0] * rel + tiny;
      const long double bL = fabsl(F[NP - 1]) * 1.2e-16L + xm * ldexpl(1, B.fD.s) * k[NP - 1] * rel + tiny;
      if (!(fabsl(F[0]) > 1e300L) && !(fabsl(F[NP - 1]) > 1e300L) && kind != 8) {
        wf = fmax(wf, (double)fmaxl(fabsl(f.t0 - F[0]) / b0, fabsl(f.tL - F[NP - 1]) / bL));
        const double h0 = flux_end<NP>(B, false, x, k[0]), hL = flux_end<NP>(B, true, x, k[NP - 1]);
        ok &= std::memcmp(&h0, &f.t0, 8) == 0 && std::memcmp(&hL, &f.tL, 8) == 0;
      }
      // the rows' parts come from rows of their own
      for (int i = 0; i < NP; ++i) {
        FixFlux<NP> z;
        double zx[NP] = {}, zk[NP];
        for (int j = 0; j < NP; ++j) zk[j] = 1e-4;
        flux_line<NP>(B, zx, zk, z);
        FixSums<NP> r;
        row_sums<NP>(B, z, 0.0, 0.0, row[i], 0.0, r);
        R[i] = r.G[0];
        er[i] = r.e;
      }
      const int sg = uni() < 0.5 ? 1 : -1;
      FixSums<NP> col;
      row_sums<NP>(B, f, u0, uL, a0, aL, col);
      for (int i = 0; i < NP; ++i) out[i] = node_total<59>(R[i], er[i], col.G[i], col.e, acc[i], sg);
      // the same in FP64, in the order of a chain of multiply-adds
      double c64[NP], s64[NP];
      for (int i = 0; i < NP; ++i) {
        double g = 0;
        for (int j = 0; j < NP; ++j) if (!fix::skip<NP>(i, j)) g = std::fma(B.D[i][j], x[j], g);
        s64[i] = g * k[i];
      }
      s64[0] += u0;
      s64[NP - 1] += uL;
      for (int i = 0; i < NP; ++i) {
        c64[i] = row[i];
        if (i == 0) c64[i] += a0;
        if (i == NP - 1) c64[i] += aL;
        for (int j = 0; j < NP; ++j) if (!fix::skip<NP>(i, j)) c64[i] = std::fma(B.D[j][i], s64[j], c64[i]);
        c64[i] = acc[i] + sg * c64[i];
      }
      top = xm * ldexpl(1, 2 * B.fD.s) * km + ldexpl(1, B.fD.s) * fmaxl(fabsl((long double)u0), fabsl((long double)uL));
      for (int i = 0; i < NP; ++i) top = fmaxl(fmaxl(top, fabsl((long double)acc[i])), fabsl((long double)row[i]));
      top = fmaxl(fmaxl(top, fabsl((long double)a0)), fabsl((long double)aL));
      for (int i = 0; i < NP; ++i) {
        long double s = row[i] + (i == 0 ? a0 : 0.0) + (i == NP - 1 ? aL : 0.0);
        for (int j = 0; j < NP; ++j)
          if (!fix::skip<NP>(i, j)) s += (long double)B.D[j][i] * (F[j] + (j == 0 ? u0 : 0.0) + (j == NP - 1 ? uL : 0.0));
        s = acc[i] + sg * s;
        if (kind == 8) continue;
        if (top == 0) { ok &= out[i] == 0; continue; }
        const long double ei = (out[i] - s) / top, ef = (c64[i] - s) / top;
        sum_i += (double)(ei * ei);
        sum_f += (double)(ef * ef);
      }
    }
    // no less exact than the FP64 chain; near and beyond the range's ends (4, 7, 8) and on P1 lines the chain itself runs
    ws = sum_f > 0 && NP > 2 && kind != 4 && kind != 7 ? std::sqrt(sum_i / sum_f) : 0;
    ok &= wf <= 1 && ws <= 1;
    bad += !ok;
    std::printf("NP%d sip kind%d %s %.3f %.3f\n", NP, kind, ok ? "ok" : "BAD", wf, ws);
  }
  // products flux_i (D v)_i summed over a row part, end terms and what is there already; kinds as above
  for (int kind = 0; kind <= 12; ++kind) {
    double sum_i = 0, sum_f = 0;
    bool ok = true;
    for (int it = 0; it < 4000; ++it) {
      double x[NP], v[NP], k[NP], acc[NP], out[NP], row[NP];
      long long R[NP];
      int er[NP];
      const double d = kind >= 9 ? std::pow(100.0, 9 - kind) : 1;
      const double c1 = 2 * uni() - 1, c2 = 2 * uni() - 1, c3 = 2 * uni() - 1;
      for (int i = 0; i < NP; ++i) {
        const double s = 2.0 * i / (NP - 1) - 1;
        x[i] = kind >= 9 ? 1 + d * s * (c1 + s * (c2 + s * c3)) : value(kind);
        v[i] = kind >= 9 ? 2 - d * s * (c3 + s * (c1 + s * c2)) : value(kind == 5 ? 0 : kind);
        k[i] = (0.5 + uni()) * 1e-4;
        const double w = kind >= 9 ? d * d * 1e-4 : (kind == 6 ? 0 : (kind == 5 ? 1e290 : (kind == 4 || kind == 7 ? 0 : 1e-4)));
        acc[i] = w * (2 * uni() - 1);
        row[i] = w * (2 * uni() - 1);
      }
      const double z0 = row[0] * 0.3, zL = row[0] * 0.2;
      FixFlux<NP> f, zf;
      FixDeriv<NP> dv, zd;
      flux_line<NP>(B, x, k, f);
      deriv_line<NP>(B, v, dv);
      double zeros[NP] = {};
      flux_line<NP>(B, zeros, k, zf);
      deriv_line<NP>(B, zeros, zd);
      for (int i = 0; i < NP; ++i) {
        FixSums<NP> r;
        row_products<NP>(zf, zd, row[i], 0.0, r);
        R[i] = r.G[0];
        er[i] = r.e;
      }
      const int sg = uni() < 0.5 ? 1 : -1;
      FixSums<NP> col;
      row_products<NP>(f, dv, z0, zL, col);
      for (int i = 0; i < NP; ++i) out[i] = node_total<60>(R[i], er[i], col.G[i], col.e, acc[i], sg);
      if (kind == 8) continue;
      long double top = 0, S[NP];
      double c64[NP];
      for (int i = 0; i < NP; ++i) {
        long double gx = 0, gv = 0;
        double hx = 0, hv = 0;
        for (int j = 0; j < NP; ++j)
          if (!fix::skip<NP>(i, j)) {
            gx += (long double)B.D[i][j] * x[j]; gv += (long double)B.D[i][j] * v[j];
            hx = std::fma(B.D[i][j], x[j], hx); hv = std::fma(B.D[i][j], v[j], hv);
          }
        S[i] = gx * k[i] * gv + (i == 0 ? z0 : 0.0) + (i == NP - 1 ? zL : 0.0) + row[i];
        S[i] = acc[i] + sg * S[i];
        double h = k[i] * hx * hv;
        if (i == 0) h += z0;
        if (i == NP - 1) h += zL;
        c64[i] = acc[i] + sg * (h + row[i]);
        top = fmaxl(top, fmaxl(fabsl((long double)acc[i]), fmaxl(fabsl((long double)row[i]), fabsl(gx * k[i] * gv))));
      }
      for (int i = 0; i < NP; ++i) {
        if (top < 1e-300L) { ok &= kind == 4 || kind == 7 || out[i] == 0; continue; }
        const long double ei = (out[i] - S[i]) / top, ef = (c64[i] - S[i]) / top;
        sum_i += (double)(ei * ei);
        sum_f += (double)(ef * ef);
      }
    }
    const double ratio = sum_f > 0 && NP > 2 && kind != 4 && kind != 7 ? std::sqrt(sum_i / sum_f) : 0;
    ok &= ratio <= 1;
    bad += !ok;
    std::printf("NP%d products kind%d %s %.3f\n", NP, kind, ok ? "ok" : "BAD", ratio);
  }
  // a qa + b qb + row + column at a node, against long double and against the FP64 form of the weights
  {
    double sum_i = 0, sum_f = 0;
    bool ok = true;
    for (int it = 0; it < 20000; ++it) {
      const double ws[3][2] = {{0.25, 0.75}, {2.0 / 3, 1.0 / 3}, {1.0, 0.5}};
      const FixScale a = fix_scale(ws[it % 3][0]), b = fix_scale(ws[it % 3][1]);
      double qa = 1 + 0.3 * (2 * uni() - 1), qb = qa * (1 + 1e-2 * uni());
      if (it % 5 == 1) qa = 0.0;
      if (it % 5 == 2) qb = -qb;
      if (it % 5 == 3) { qa *= 1e-9; qb *= 1e-9; }
      double x[NP], y[NP], k[NP], zero[NP] = {};
      for (int i = 0; i < NP; ++i) { x[i] = 1e-3 * (2 * uni() - 1); y[i] = 1e-3 * (2 * uni() - 1); k[i] = 1; }
      FixSums<NP> r, c;
      const FixScale one = fix_scale(1.0);
      row_scaled<NP, false>(B, one, x, r);
      row_scaled<NP, false>(B, one, y, c);
      long double R = 0, C = 0;
      for (int j = 0; j < NP; ++j) { R += (long double)B.D[0][j] * x[j]; C += (long double)B.D[0][j] * y[j]; }
      const double got = node_blend(r.G[0], r.e, c.G[0], c.e, qa, a, qb, b);
      const long double want = (long double)a.d * qa + (long double)b.d * qb + R + C;
      const double f64 = std::fma(b.d, qb, a.d * qa) + ((double)R + (double)C);
      sum_i += (double)((got - want) * (got - want));
      sum_f += (double)((f64 - want) * (f64 - want));
    }
    if (NP > 2) ok = sum_i <= sum_f;
    bad += !ok;
    std::printf("NP%d blend 0 %s %.3f\n", NP, ok ? "ok" : "BAD", std::sqrt(sum_i / sum_f));
  }
  // infinities and NaN come out as not finite wherever the FP64 chain has them
  const double inf = std::numeric_limits<double>::infinity();
  for (double x : {inf, -inf, std::numeric_limits<double>::quiet_NaN()})
    for (int at = 0; at < NP; ++at) {
      double v[NP], ac[NP], out[NP];
      for (int k = 0; k < NP; ++k) { v[k] = 0.5 + k; ac[k] = 1; }
      v[at] = x;
      bool ok = true;
      line_rows<NP>(B, v, out);
      for (int i = 0; i < NP; ++i) ok &= std::isfinite(out[i]) == fix::skip<NP>(i, at);
      line_op<NP, true, true, false>(B.fD, B.D, nullptr, v, ac, [](int) { return true; }, out);
      for (int i = 0; i < NP; ++i) ok &= std::isfinite(out[i]) == fix::skip<NP>(i, at);
      v[at] = 0.25; ac[at] = x;
      line_op<NP, true, true, false>(B.fD, B.D, nullptr, v, ac, [](int) { return true; }, out);
      for (int i = 0; i < NP; ++i) ok &= std::isfinite(out[i]) == (i != at);
      bad += !ok;
      std::printf("NP%d nonfinite%d %s 0\n", NP, at, ok ? "ok" : "BAD");
    }
  return bad;
}

int main() { return run<2>() + run<3>() + run<4>() + run<5>() ? 1 : 0; }
