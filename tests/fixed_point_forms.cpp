// Host checks of csrc/igr_fix.cuh beyond fixed_point_check.cpp (whose host forms of the intrinsics and basis it uses), for
// tests/test_fixed_point_forms.py: one check per name, run as "fixed_point_forms NAME". Prints "name NP ok|BAD worst".
#define main fixed_point_main
#include "fixed_point_check.cpp"
#undef main

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

template <int NP> static int run_one(const char* name) {
  if (!std::strcmp(name, "flux_range")) return flux_range<NP>();
  return 1;
}

int main(int, char** v) {
  return run_one<2>(v[1]) + run_one<3>(v[1]) + run_one<4>(v[1]) + run_one<5>(v[1]) ? 1 : 0;
}
