// The oracle's templates in long double, for tests/test_gpu_long_double.py: how far results of the discretisation are from
// its exact evaluation (the same double constants, basis and inputs). Every ld_ function returns relative errors in the
// 2-norm of the values it is given.
#include <cmath>
namespace igr {
inline long double value(long double x) { return x; }  // seen by the oracle's templates
}
#include "../oracle/igr2d_adjoint.hpp"

namespace igr {
// forward-mode dual numbers over long double
#ifndef DIRECTIONS
#define DIRECTIONS 2
#endif
constexpr int ND = 2 + DIRECTIONS;
struct Dl {
  long double v, d[ND];
  Dl() : v(0) { for (auto& x : d) x = 0; }
  Dl(double x) : v(x) { for (auto& y : d) y = 0; }  // NOLINT
};
inline Dl map(long double v, const Dl& a, long double fa) { Dl r; r.v = v; for (int k = 0; k < ND; ++k) r.d[k] = fa * a.d[k]; return r; }
inline Dl map(long double v, const Dl& a, long double fa, const Dl& b, long double fb) {
  Dl r; r.v = v; for (int k = 0; k < ND; ++k) r.d[k] = fa * a.d[k] + fb * b.d[k]; return r;
}
inline Dl operator+(const Dl& a, const Dl& b) { return map(a.v + b.v, a, 1, b, 1); }
inline Dl operator-(const Dl& a, const Dl& b) { return map(a.v - b.v, a, 1, b, -1); }
inline Dl operator*(const Dl& a, const Dl& b) { return map(a.v * b.v, a, b.v, b, a.v); }
inline Dl operator/(const Dl& a, const Dl& b) { const long double q = a.v / b.v; return map(q, a, 1 / b.v, b, -q / b.v); }
inline Dl operator-(const Dl& a) { return map(-a.v, a, -1); }
inline Dl operator+(const Dl& a, double b) { return map(a.v + b, a, 1); }
inline Dl operator+(double a, const Dl& b) { return map(a + b.v, b, 1); }
inline Dl operator-(const Dl& a, double b) { return map(a.v - b, a, 1); }
inline Dl operator-(double a, const Dl& b) { return map(a - b.v, b, -1); }
inline Dl operator*(const Dl& a, double b) { return map(a.v * b, a, b); }
inline Dl operator*(double a, const Dl& b) { return map(a * b.v, b, a); }
inline Dl operator/(const Dl& a, double b) { return map(a.v / b, a, 1 / (long double)b); }
inline Dl operator/(double a, const Dl& b) { const long double q = a / b.v; return map(q, b, -q / b.v); }
inline Dl& operator+=(Dl& a, const Dl& b) { return a = a + b; }
inline Dl sqrt(const Dl& a) { const long double s = std::sqrt(a.v); return map(s, a, 0.5L / s); }
inline Dl abs(const Dl& a) { return std::signbit(a.v) ? -a : a; }
inline long double value(const Dl& x) { return x.v; }
inline bool operator>(const Dl& a, double b) { return a.v > b; }
inline bool operator<(const Dl& a, double b) { return a.v < b; }
}  // namespace igr
using namespace igr;
using LD = long double;

namespace {
Grid2D grid(int p, const double* xi, const double* w, const double* D, int nex, int ney, double lx, double ly) {
  return Grid2D(basis_from_arrays(p, xi, w, D), make_mesh2d(nex, ney, lx, ly));
}
std::vector<LD> wide(const double* a, size_t n) { return std::vector<LD>(a, a + n); }
double err(const double* y, const std::vector<LD>& ref) {
  LD e = 0, s = 0;
  for (size_t k = 0; k < ref.size(); ++k) { e += (y[k] - ref[k]) * (y[k] - ref[k]); s += ref[k] * ref[k]; }
  return (double)std::sqrt(e / s);
}
}  // namespace

#define GRID int p, const double *xi, const double *w, const double *D, int nex, int ney, double lx, double ly
#define MAKE const Grid2D G = grid(p, xi, w, D, nex, ney, lx, ly); const size_t N = G.N

extern "C" {
// ncand candidates y[c N ..] for A x -> out[c]
void ld_apply(GRID, double alpha, const double* x, const double* rho, int ncand, const double* y, double* out) {
  MAKE;
  std::vector<LD> r(N), X = wide(x, N), R = wide(rho, N);
  apply_sip<LD>(G, r.data(), X.data(), R.data(), (LD)alpha);
  for (int c = 0; c < ncand; ++c) out[c] = err(y + c * N, r);
}
// candidates for (Sigma, dmx, dmy, drho, dE), five fields each, of a right-hand side from the warm start sig -> out[5 c + f]
void ld_rhs(GRID, double gamma, double alpha, int n_iter, int solver, const double* q, const double* sig, int ncand,
            const double* y, double* out) {
  MAKE;
  std::vector<LD> Q = wide(q, 4 * N), S = wide(sig, N);
  const LD* qc[4] = {&Q[0], &Q[N], &Q[2 * N], &Q[3 * N]};
  Work2D<LD> W;
  W.alloc(N);
  igr_euler_rhs<LD>(G, qc, S.data(), (LD)gamma, (LD)alpha, n_iter, solver, W);
  for (int c = 0; c < ncand; ++c)
    for (int f = 0; f < 5; ++f) out[5 * c + f] = err(y + (5 * c + f) * N, f == 0 ? S : W.dq[f - 1]);
}
// J, dJ/dgamma, dJ/dalpha and ND - 2 directional derivatives along dir[k 4N ..] after n_steps -> out[2 k], as pairs of
// doubles (value, remainder), k = 0 .. ND; and the final state -> state[4 N]
void ld_gradient(GRID, double gamma, double alpha, int n_steps, double dt, int n_iter, int solver, int obj, const double* prm,
                 const double* q0, const double* dir, double* out) {
  MAKE;
  std::vector<Dl> q[4];
  for (int v = 0; v < 4; ++v) {
    q[v].resize(N);
    for (size_t n = 0; n < N; ++n) {
      q[v][n].v = q0[v * N + n];
      for (int k = 2; k < ND; ++k) q[v][n].d[k] = dir[(k - 2) * 4 * N + v * N + n];
    }
  }
  Dl* qp[4] = {q[0].data(), q[1].data(), q[2].data(), q[3].data()};
  Dl g(gamma), al(alpha);
  g.d[0] = 1;
  al.d[1] = 1;
  const Dl J = objective_run<Dl>(G, obj, qp, n_steps, dt, g, al, n_iter, solver, prm);
  for (int k = 0; k <= ND; ++k) {
    const LD x = k == 0 ? J.v : J.d[k - 1];
    out[2 * k] = (double)x;
    out[2 * k + 1] = (double)(x - out[2 * k]);
  }
}
}
