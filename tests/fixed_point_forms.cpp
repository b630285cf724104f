// Host checks of csrc/igr_fix.cuh beyond fixed_point_check.cpp (whose host forms of the intrinsics and basis it uses), for
// tests/test_fixed_point_forms.py: one check per name, run as "fixed_point_forms NAME". Prints "name NP ok|BAD worst".
#define main fixed_point_main
#include "fixed_point_check.cpp"
#undef main
#include <type_traits>

static int report(const char* name, int np, bool ok, double worst) {
  std::printf("%s NP%d %s %.3g\n", name, np, ok ? "ok" : "BAD", worst);
  return !ok;
}

// Fluxes near the lower end of the range with coefficients apart by up to 2^40, half of the lines cancelling: the end fluxes
// and the operator's sums stay with the FP64 chain, to its own rounding errors (five of 2^-53 of the line's scale, twice) and
// the subnormals' quantum.
template <int NP> static int flux_range() {
  const Basis B = make(NP);
  double worst = 0;
  for (int it = 0; it < 40000; ++it) {
    double x[NP], k[NP], s64[NP], top = 0;
    const int ex = -894 + (int)(30 * uni()), ek = -110 + (int)(90 * uni());
    const bool level = uni() < 0.5;
    for (int i = 0; i < NP; ++i) {
      x[i] = std::ldexp(level ? 1.1 : 1 + uni(), ex);
      k[i] = std::ldexp(1 + uni(), ek + (int)(40 * uni()));
    }
    const double scale = std::ldexp(1.0, ex + 1 + B.fD.s);
    FixFlux<NP> f;
    flux_line<NP>(B, x, k, f);
    for (int i = 0; i < NP; ++i) {
      double g = 0;
      for (int j = 0; j < NP; ++j) if (!fix::skip<NP>(i, j)) g = std::fma(B.D[i][j], x[j], g);
      s64[i] = g * k[i];
      top = std::fmax(top, scale * k[i]);
    }
    for (int i = 0; i < NP; i += NP - 1) {
      const double t = i == 0 ? f.t0 : f.tL, h = flux_end<NP>(B, i != 0, x, k[i]);
      worst = std::fmax(worst, std::fmax(std::fabs(t - s64[i]), std::fabs(h - s64[i])) / (scale * k[i] * 1e-15 + 1e-321));
    }
    FixSums<NP> r;
    row_sums<NP>(B, f, 0.0, 0.0, 0.0, 0.0, r);
    for (int j = 0; j < NP; ++j) {
      double g = 0;
      for (int i = 0; i < NP; ++i) if (!fix::skip<NP>(i, j)) g = std::fma(B.D[i][j], s64[i], g);
      const double y = node_total<59>(r.G[j], r.e, 0, 0, 0.0, 1);
      worst = std::fmax(worst, std::fabs(y - g) / (std::ldexp(top, B.fD.s) * 4e-15 + 1e-320));
    }
  }
  return report("flux_range", NP, worst <= 1, worst);
}

// The matrices of the kernels' forms: D, D with the own side's share of the face corrections, W2 = w D^2 elementwise.
struct Full { double D[FIX_MAXNP][FIX_MAXNP], Dr[FIX_MAXNP][FIX_MAXNP], W2[FIX_MAXNP][FIX_MAXNP]; FixMat fD, fDr, fW2; };
static Full full(int np) {
  const Basis B = make(np);
  const double w[6][5] = {{0}, {0}, {1, 1}, {1. / 3, 4. / 3, 1. / 3}, {1. / 6, 5. / 6, 5. / 6, 1. / 6}, {.1, 49. / 90, 32. / 45, 49. / 90, .1}};
  Full F = {};
  std::memcpy(F.D, B.D, sizeof(F.D));
  std::memcpy(F.Dr, B.D, sizeof(F.D));
  F.Dr[0][0] += 0.5 / w[np][0];
  F.Dr[np - 1][np - 1] -= 0.5 / w[np][np - 1];
  for (int i = 0; i < np; ++i) for (int k = 0; k < np; ++k) F.W2[i][k] = w[np][i] * (B.D[i][k] * B.D[i][k]);
  F.fD = make_fix(F.D, np); F.fDr = make_fix(F.Dr, np); F.fW2 = make_fix(F.W2, np);
  return F;
}

// One interior value (or coefficient) larger than the others by 2^g: its own row, which leaves it out, is as exact relative to
// its own terms as the FP64 chain's, in rms over random lines.
template <int NP> static int leading() {
  if (NP == 2) return 0;
  const Full B = full(NP);
  int bad = 0;
  const char* forms[] = {"rows", "cols", "w2_cols", "w2_rows", "dr_cols", "scaled", "deriv", "flux", "div", "div_coef"};
  for (int form = 0; form < 10; ++form)
    for (int g8 = 0; g8 <= 160; g8 += g8 < 32 ? 2 : 16) {
      double si = 0, sf = 0;
      for (int it = 0; it < 20000; ++it) {
        const int at = 1 + (int)(uni() * (NP - 2));
        double v[NP], k[NP], out[NP];
        for (int i = 0; i < NP; ++i) { v[i] = (uni() < 0.5 ? -1 : 1) * (1 + uni()); k[i] = 1e-4 * (1 + uni()); }
        const double s = std::exp2(g8 / 8.0);
        (form == 9 ? k : v)[at] *= s;
        const FixScale c = fix_scale((1 + uni()) * 8);
        const bool T = form == 1 || form == 2 || form >= 4 && form != 6 && form != 7;
        const double (*A)[FIX_MAXNP] = form == 4 ? B.Dr : (form == 2 || form == 3 ? B.W2 : B.D);
        auto none = [](int) { return false; };
        FixSums<NP> r;
        if (form == 0) line_op<NP, false, true, true>(B.fD, B.D, &c, v, nullptr, none, out);
        if (form == 1) line_op<NP, true, true, true>(B.fD, B.D, &c, v, nullptr, none, out);
        if (form == 2) line_op<NP, true, false, true>(B.fW2, B.W2, &c, v, nullptr, none, out);
        if (form == 3) line_op<NP, false, false, true>(B.fW2, B.W2, &c, v, nullptr, none, out);
        if (form == 4) line_op<NP, true, true, true>(B.fDr, B.Dr, &c, v, nullptr, none, out);
        if (form == 5) { row_scaled<NP, true>(B, c, v, r); for (int i = 0; i < NP; ++i) out[i] = sums_at<NP>(r, i); }
        if (form == 6) { FixDeriv<NP> d; deriv_line<NP>(B, v, d); for (int i = 0; i < NP; ++i) out[i] = deriv_at<NP>(d, i); }
        if (form >= 7) {
          FixFlux<NP> f;
          if (form == 7) flux_line<NP, true>(B, v, k, f);
          else flux_line<NP>(B, v, k, f);
          for (int i = 0; i < NP; ++i) out[i] = flux_at<NP>(f, i);
          if (form >= 8) {
            row_sums<NP>(B, f, 0.0, 0.0, 0.0, 0.0, r);
            for (int i = 0; i < NP; ++i) out[i] = node_total<59>(r.G[i], r.e, 0, 0, 0.0, 1);
          }
        }
        long double ref = 0, mag = 0;
        double f64 = 0;
        if (form < 8) {
          for (int j = 0; j < NP; ++j) {
            if (j == at) continue;
            const double a = T ? A[j][at] : A[at][j];
            ref += (long double)a * v[j]; mag += fabsl((long double)a * v[j]); f64 = std::fma(a, v[j], f64);
          }
          const double cc = form == 7 ? k[at] : (form == 6 ? 1.0 : c.d);
          ref *= cc; mag *= cc; f64 *= cc;
        } else {
          for (int i = 0; i < NP; ++i) {
            if (i == at) continue;
            long double G = 0, H = 0;
            double h = 0;
            for (int j = 0; j < NP; ++j) {
              if (fix::skip<NP>(i, j)) continue;
              G += (long double)B.D[i][j] * v[j]; H += fabsl((long double)B.D[i][j] * v[j]); h = std::fma(B.D[i][j], v[j], h);
            }
            ref += B.D[i][at] * (G * k[i]); mag += fabs(B.D[i][at]) * (H * k[i]); f64 = std::fma(B.D[i][at], h * k[i], f64);
          }
        }
        const long double ei = (out[at] - ref) / mag, ef = (f64 - ref) / mag;
        si += (double)(ei * ei); sf += (double)(ef * ef);
      }
      const double ratio = std::sqrt(si / sf);
      char name[64];
      std::snprintf(name, sizeof(name), "leading %s 2^%.2f", forms[form], g8 / 8.0);
      bad += report(name, NP, ratio <= 1.001, ratio);  // 1 where the chain runs or both round once, the same sums
    }
  return bad;
}

// No result is high or low on average: the mean error over random lines stays within five standard errors of zero.
template <int NP> static int mean() {
  if (NP == 2) return 0;
  const Full B = full(NP);
  int bad = 0;
  const int n = 200000;
  const char* forms[] = {"conversion", "scaled", "deriv", "flux", "operator", "products", "stage"};
  for (int kind = 0; kind < 3; ++kind) {  // both signs; positive; a slope with noise, v against x
    long double s1[7] = {}, s2[7] = {};
    for (int it = 0; it < n; ++it) {
      double x[NP], v[NP], k[NP], out[NP];
      for (int i = 0; i < NP; ++i) {
        const double s = 2.0 * i / (NP - 1) - 1, u = uni();
        x[i] = kind == 0 ? 2 * u - 1 : (kind == 1 ? 1 + u : 1 + 0.3 * s + 1e-3 * u);
        v[i] = kind == 0 ? 2 * uni() - 1 : (kind == 1 ? 1 + uni() : -0.7 * x[i] + 1e-3 * uni());
        k[i] = 1e-4 * (1 + 0.3 * uni());
      }
      const int at = it % NP, other = (at + 1) % NP;
      auto contract = [&](bool T, int i, const long double* a) {
        long double r = 0;
        for (int j = 0; j < NP; ++j) if (!fix::skip<NP>(i, j)) r += (long double)(T ? B.D[j][i] : B.D[i][j]) * a[j];
        return r;
      };
      long double X[NP], V[NP], P[NP];
      for (int i = 0; i < NP; ++i) { X[i] = x[i]; V[i] = v[i]; }
      for (int i = 0; i < NP; ++i) P[i] = contract(false, i, X) * k[i];
      const FixScale c = fix_scale(3.7 + uni());
      FixFlux<NP> f;
      FixDeriv<NP> d;
      FixSums<NP> y, z, q;
      line_op<NP, true, true, true>(B.fD, B.D, &c, v, nullptr, [](int) { return false; }, out);
      flux_line<NP>(B, x, k, f);
      deriv_line<NP>(B, v, d);
      row_sums<NP>(B, f, 0.0, 0.0, 0.0, 0.0, y);
      row_products<NP>(f, d, 0.0, 0.0, z);
      row_scaled<NP, false>(B, c, v, q);
      const double m = 1e-5 * (1 + uni()) * x[at], zs = 1e-4 * (2 * uni() - 1), qa = 100 + uni(), qb = 100 + uni();
      const FixScale wa = fix_scale(0.25), wb = fix_scale(0.75);
      const long long G = (long long)rs >> (2 + it % 9);
      const long double e[7] = {
          fix::to_double(G, 1082) - (long double)G,
          out[at] - contract(true, at, V) * c.d,
          deriv_at<NP>(d, at) - contract(false, at, V),
          flux_at<NP>(f, at) - P[at],
          node_total<59>(y.G[at], y.e, y.G[other], y.e, m, 1) - (contract(true, at, P) + contract(true, other, P) + m),
          node_total<60>(z.G[at], z.e, z.G[other], z.e, zs, -1) - (zs - P[at] * contract(false, at, V) - P[other] * contract(false, other, V)),
          node_blend(q.G[at], q.e, q.G[other], q.e, qa, wa, qb, wb) -
              (0.25L * qa + 0.75L * qb + c.d * (contract(false, at, V) + contract(false, other, V)))};
      for (int j = 0; j < 7; ++j) { s1[j] += e[j]; s2[j] += e[j] * e[j]; }
    }
    for (int j = 0; j < 7; ++j) {
      const double sigma = s2[j] > 0 ? (double)(fabsl(s1[j]) / std::sqrt((double)s2[j])) : 0;
      char name[64];
      std::snprintf(name, sizeof(name), "mean %s kind%d", forms[j], kind);
      bad += report(name, NP, sigma <= 5, sigma);
    }
  }
  return bad;
}

// Both sides of a face hold the same end flux, whatever the other coefficients of either line are.
template <int NP> static int face_sides() {
  const Basis B = make(NP);
  int differ = 0;
  for (int it = 0; it < 20000; ++it) {
    double x[NP], k[NP];
    for (int i = 0; i < NP; ++i) { x[i] = (2 * uni() - 1) * std::ldexp(1.0, it % 3 == 0 ? (int)(12 * uni()) : 0); k[i] = 1e-4 * (1 + uni()); }
    k[it % NP] *= it % 2 ? std::ldexp(1.0, (int)(1200 * uni()) - 600) : 0.0;
    FixFlux<NP> f;
    flux_line<NP>(B, x, k, f);
    const double h0 = flux_end<NP>(B, false, x, k[0]), hL = flux_end<NP>(B, true, x, k[NP - 1]);
    differ += std::memcmp(&h0, &f.t0, 8) != 0 || std::memcmp(&hL, &f.tL, 8) != 0;
  }
  return report("face_sides", NP, differ == 0, differ);
}

// The forms that the kernels use, over the kinds of lines of fixed_point_check.cpp: scaled sums with the matrices Dr and W2 and
// with end terms, against long double. The rms error is at most the FP64 chain's, with three standard errors of it (both may
// end in one rounding of the same size); single errors stay below 8e-16 of the largest term, also where the chain runs.
template <int NP> static int forms() {
  const Full B = full(NP);
  int bad = 0;
  const char* names[] = {"dr_cols_ends", "w2_cols_ends", "w2_rows_ends", "stage_line", "transposes"};
  for (int form = 0; form < 5; ++form)
    for (int kind = 0; kind <= 8; ++kind) {
      double si = 0, sf = 0, worst = 0;
      bool ok = true;
      for (int it = 0; it < 4000; ++it) {
        double v[NP], out[NP];
        for (int i = 0; i < NP; ++i) v[i] = value(kind);
        const double big = std::ldexp(1.0, (int)(40 * uni()) - 20);
        const double a0 = kind == 6 ? 0.0 : value(kind) * (kind < 4 ? big : 1), aL = kind == 6 ? 0.0 : value(kind) * (kind < 4 ? big : 1);
        const FixScale c = fix_scale((uni() < 0.5 ? -1 : 1) * std::ldexp(1 + uni(), (int)(8 * uni()) - 8));
        const bool T = form == 0 || form == 1 || form == 4;
        const FixMat& F = form == 0 ? B.fDr : (form < 3 ? B.fW2 : B.fD);
        const double (*A)[FIX_MAXNP] = form == 0 ? B.Dr : (form < 3 ? B.W2 : B.D);
        auto ends = [](int k) { return k == 0 || k == NP - 1; };
        double acc[NP] = {};
        acc[0] = form == 4 ? 0.0 : a0;
        acc[NP - 1] = form == 4 ? 0.0 : aL;
        FixSums<NP> r;
        if (form == 0) line_op<NP, true, true, true>(F, A, &c, v, acc, ends, out);
        if (form == 1) line_op<NP, true, false, true>(F, A, &c, v, acc, ends, out);
        if (form == 2) line_op<NP, false, false, true>(F, A, &c, v, acc, ends, out);
        if (form == 3) { row_scaled<NP, false>(B, c, v, r); row_add_ends<NP>(r, a0, aL); }
        if (form == 4) row_scaled<NP, true>(B, c, v, r);
        if (form >= 3) for (int i = 0; i < NP; ++i) out[i] = node_total<60>(r.G[i], r.e, 0, 0, 0.0, 1);
        long double top = std::fmax(std::fabs(acc[0]), std::fabs(acc[NP - 1]));
        for (int i = 0; i < NP; ++i) top = fmaxl(top, ldexpl(fabsl((long double)v[i] * c.d), F.s));
        for (int i = 0; i < NP; ++i) {
          long double s = 0;
          double f64 = 0;
          for (int k = 0; k < NP; ++k) {
            if ((form == 0 || form >= 3) && fix::skip<NP>(i, k)) continue;
            const double m = T ? A[k][i] : A[i][k];
            s += (long double)m * v[k];
            f64 = std::fma(m, v[k], f64);
          }
          s = s * c.d + acc[i];
          f64 = std::fma(c.d, f64, acc[i]);
          if (!std::isfinite(f64) || fabsl(s) > 1.7e308L || top > 1e307L) continue;
          if (top == 0) { ok &= out[i] == 0; continue; }
          const long double ei = (out[i] - s) / top, ef = (f64 - s) / top;
          worst = std::fmax(worst, (double)(fabsl(out[i] - s) / (top * 8e-16L + 1e-321L)));
          si += (double)(ei * ei); sf += (double)(ef * ef);
        }
      }
      const double ratio = NP > 2 && kind < 7 && kind != 4 && sf > 0 ? std::sqrt(si / sf) : 0;
      char name[64];
      std::snprintf(name, sizeof(name), "forms %s kind%d", names[form], kind);
      bad += report(name, NP, ok && worst <= 1 && ratio <= 1 + 3 / std::sqrt(4000.0 * NP), std::fmax(worst, ratio));
    }
  return bad;
}

// Infinities and NaN come out as not finite wherever the FP64 chain has them, in the same forms and in the operator's lines.
template <int NP> static int nonfinite() {
  const Full B = full(NP);
  int wrong = 0;
  const double inf = std::numeric_limits<double>::infinity();
  for (double bad : {inf, -inf, std::numeric_limits<double>::quiet_NaN()})
    for (int at = 0; at < NP + 2; ++at) {  // NP, NP + 1: an end term
      double v[NP], k[NP], acc[NP] = {}, out[NP];
      for (int i = 0; i < NP; ++i) { v[i] = 0.5 + i; k[i] = 1e-4 * (1 + i); }
      acc[0] = 0.25; acc[NP - 1] = -0.5;
      if (at < NP) v[at] = bad;
      else acc[at == NP ? 0 : NP - 1] = bad;
      const FixScale c = fix_scale(-1.5);
      auto ends = [](int i) { return i == 0 || i == NP - 1; };
      auto chain = [&](const double (*A)[FIX_MAXNP], bool T, bool skip, int i) {
        double s = 0;
        for (int j = 0; j < NP; ++j) if (!(skip && fix::skip<NP>(i, j))) s = std::fma(T ? A[j][i] : A[i][j], v[j], s);
        return std::fma(c.d, s, acc[i]);
      };
      line_op<NP, true, true, true>(B.fDr, B.Dr, &c, v, acc, ends, out);
      for (int i = 0; i < NP; ++i) wrong += std::isfinite(out[i]) != std::isfinite(chain(B.Dr, true, true, i));
      line_op<NP, true, false, true>(B.fW2, B.W2, &c, v, acc, ends, out);
      for (int i = 0; i < NP; ++i) wrong += std::isfinite(out[i]) != std::isfinite(chain(B.W2, true, false, i));
      FixSums<NP> r;
      row_scaled<NP, false>(B, c, v, r);
      row_add_ends<NP>(r, acc[0], acc[NP - 1]);
      for (int i = 0; i < NP; ++i)
        wrong += std::isfinite(node_total<60>(r.G[i], r.e, 0, 0, 1.0, 1)) != std::isfinite(chain(B.D, false, true, i));
      FixFlux<NP> f;
      FixDeriv<NP> d;
      flux_line<NP>(B, v, k, f);
      deriv_line<NP>(B, v, d);
      row_products<NP>(f, d, 0.0, 0.0, r);
      for (int i = 0; i < NP; ++i) {
        const bool fine = at >= NP || fix::skip<NP>(i, at);
        wrong += std::isfinite(deriv_at<NP>(d, i)) != fine;
        wrong += std::isfinite(flux_at<NP>(f, i)) != fine;
        wrong += std::isfinite(node_total<60>(r.G[i], r.e, 0, 0, 1.0, -1)) != fine;
      }
    }
  return report("nonfinite", NP, wrong == 0, wrong);
}

// A negated operand gives the negated result to the bit.
template <int NP> static int odd() {
  const Basis B = make(NP);
  int differ = 0;
  for (int it = 0; it < 40000; ++it) {
    double x[NP], y[NP], k[NP], v[NP], a[NP], b[NP];
    const double m = 1e-5 * uni(), wide = it % 2 ? 20 : 0;
    for (int i = 0; i < NP; ++i) {
      x[i] = (2 * uni() - 1) * std::ldexp(1.0, (int)(wide * uni()));
      y[i] = -x[i];
      k[i] = 1e-4 * (1 + uni());
      v[i] = 2 * uni() - 1;
    }
    const FixScale c = fix_scale(1 + uni());
    FixFlux<NP> f, g;
    FixDeriv<NP> d;
    FixSums<NP> r, s;
    line_rows<NP>(B, c, x, a);
    line_rows<NP>(B, c, y, b);
    for (int i = 0; i < NP; ++i) differ += a[i] != -b[i];
    flux_line<NP>(B, x, k, f);
    flux_line<NP>(B, y, k, g);
    deriv_line<NP>(B, v, d);
    differ += (f.t0 != -g.t0) + (f.tL != -g.tL);
    auto compare = [&](auto units) {
      constexpr int U = decltype(units)::value;
      for (int i = 0; i < NP; ++i) {
        const int j = (i + 1) % NP;
        differ += node_total<U>(r.G[i], r.e, r.G[j], r.e, m, 1) != -node_total<U>(s.G[i], s.e, s.G[j], s.e, -m, 1);
      }
    };
    row_sums<NP>(B, f, m, -m, x[0] * m, m, r);
    row_sums<NP>(B, g, -m, m, y[0] * m, -m, s);
    compare(std::integral_constant<int, 59>());
    row_products<NP>(f, d, m, x[0] * m, r);
    row_products<NP>(g, d, -m, y[0] * m, s);
    compare(std::integral_constant<int, 60>());
    row_scaled<NP, true>(B, c, x, r);
    row_add_ends<NP>(r, m, x[0] * m);
    row_scaled<NP, true>(B, c, y, s);
    row_add_ends<NP>(s, -m, y[0] * m);
    compare(std::integral_constant<int, 60>());
  }
  return report("odd", NP, differ == 0, differ);
}

template <int NP> static int run_one(const char* name) {
  if (!std::strcmp(name, "flux_range")) return flux_range<NP>();
  if (!std::strcmp(name, "leading")) return leading<NP>();
  if (!std::strcmp(name, "mean")) return mean<NP>();
  if (!std::strcmp(name, "odd")) return odd<NP>();
  if (!std::strcmp(name, "face_sides")) return face_sides<NP>();
  if (!std::strcmp(name, "forms")) return forms<NP>();
  if (!std::strcmp(name, "nonfinite")) return nonfinite<NP>();
  return 1;
}

int main(int, char** v) {
  return run_one<2>(v[1]) + run_one<3>(v[1]) + run_one<4>(v[1]) + run_one<5>(v[1]) ? 1 : 0;
}
