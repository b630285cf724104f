// 2D tangent (forward sensitivity) kernels: run_sensitivity of
// IGR_adjoints_2d/sensitivity.jl:353-413.
//
// Per RK stage the tangent needs, besides the primal stage:
//   k2_sens_rhs      the tangent elliptic source b_s (form 2,
//                    compute_sensitivity_elliptic_rhs!, sensitivity.jl:236-292),
//                    solved with the primal stage's operator (same rho, alpha)
//                    by the ordinary solver kernels;
//   k2_sens_hyp_rk   the tangent DG right-hand side
//                    (compute_sensitivity_hyperbolic_rhs!, sensitivity.jl:131-215)
//                    fused with the SSP-RK3 stage combination of the tangent.
// The tangent LLF flux uses the primal wave speed (sensitivity_llf_flux_x/_y,
// sensitivity.jl:85-118: no d lambda term); it is read from the face-node wave
// speeds the primal k2_hyp_rk of the same stage wrote.
// k2_sens_hyp_rk is the primal stage with other physics (dg_stage: rows and
// columns side by side); k2_sens_rhs runs rows, then columns, on one thread per
// element line.
#pragma once
#include "igr2d_kernels.cuh"

namespace igrgpu {

// ---------------------------------------------------------------------------
// Tangent elliptic source, form 2 (sensitivity.jl:236-292). Per node, with
// u = mu/rho, s_u = (zeta - u sigma)/rho (tangent velocity), r_s = sigma/rho:
//   Rp = alpha (div u^2 + ux_x^2 + 2 ux_y uy_x + uy_y^2)
//   Rs = alpha (2 div u div s_u + 2 (ux_x sx_x + ux_y sy_x + uy_x sx_y + uy_y sy_y))
//   b  = w_i w_j Jx Jy (Rs + r_s Rp - alpha (d_x r_s d_x Sigma + d_y r_s d_y Sigma) / rho)
// ---------------------------------------------------------------------------
struct SensRhsArgs2D {
  const Tile2D* tiles; const Inst2D* inst; BasisDev B;
  const double *q[3], *invr, *S;   // mu_x, mu_y, rho of the stage; 1/rho; solved Sigma
  const double *s[3];              // zeta_x, zeta_y, sigma (tangent of mu_x, mu_y, rho)
  double* b_out;
};

// What bounds it: FP64 issue; the twelve line derivatives are integer work in rolled loops over the fields. With
// k2_sens_hyp_rk 393 us per launch on average with FP64 contractions, 189 us now (122 and 279 us, 2 x 256^2 P3).
template <int NP>
__global__ void __launch_bounds__(Tiling2D<NP>::NT) k2_sens_rhs(SensRhsArgs2D a) {
  using TL = Tiling2D<NP>;
  constexpr int TE = TL::TE, NN = TL::NN;
  constexpr int NQ = 6;  // u_x, u_y, s_x, s_y, Sigma, sigma/rho
  __shared__ double s_v[NQ][TE][NN];   // the fields, then their y derivatives
  __shared__ double s_dx[NQ][TE][NN];  // x derivatives
  const Tile2D tl = a.tiles[blockIdx.x];
  const Inst2D I = a.inst[tl.inst];
  chained_start();
  const ElemView vr = elem_view<NP>(tl, I, 0), vc = elem_view<NP>(tl, I, 1);
  const BasisDev& B = a.B;
  if (vr.valid) {
    const int t = vr.t, e = vr.e;
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const long long n = vr.base + t * NP + i;
      const int nd = t * NP + i;
      const double ir = a.invr[n];
      const double ux = a.q[0][n] * ir, uy = a.q[1][n] * ir, sr = a.s[2][n];
      s_v[0][e][nd] = ux; s_v[1][e][nd] = uy;
      s_v[2][e][nd] = (a.s[0][n] - ux * sr) * ir;
      s_v[3][e][nd] = (a.s[1][n] - uy * sr) * ir;
      s_v[4][e][nd] = a.S[n];
      s_v[5][e][nd] = sr * ir;
    }
    const FixScale sc = fix_scale(I.ijx);
#pragma unroll 1
    for (int c = 0; c < NQ; ++c) {
      double v[NP], d[NP];
#pragma unroll
      for (int i = 0; i < NP; ++i) v[i] = s_v[c][e][t * NP + i];
      line_rows<NP>(B, sc, v, d);
#pragma unroll
      for (int i = 0; i < NP; ++i) s_dx[c][e][t * NP + i] = d[i];
    }
  }
  __syncthreads();
  if (!vc.valid) return;
  const int t = vc.t, e = vc.e;
  double so[NP];  // sigma / rho
#pragma unroll
  for (int l = 0; l < NP; ++l) so[l] = s_v[5][e][l * NP + t];
  const FixScale sc = fix_scale(I.ijy);
#pragma unroll 1
  for (int c = 0; c < NQ; ++c) {  // in place: the column is the thread's own from here on
    double v[NP], d[NP];
#pragma unroll
    for (int l = 0; l < NP; ++l) v[l] = s_v[c][e][l * NP + t];
    line_rows<NP>(B, sc, v, d);
#pragma unroll
    for (int l = 0; l < NP; ++l) s_v[c][e][l * NP + t] = d[l];
  }
  const double wa = B.w[t] * (I.jx * I.jy) * I.alpha;
#pragma unroll
  for (int l = 0; l < NP; ++l) {
    const int nd = l * NP + t;
    const long long n = vc.base + nd;
    const double uxx = s_dx[0][e][nd], uyx = s_dx[1][e][nd], sxx = s_dx[2][e][nd], syx = s_dx[3][e][nd];
    const double Sx = s_dx[4][e][nd], dxs = s_dx[5][e][nd];
    const double uxy = s_v[0][e][nd], uyy = s_v[1][e][nd], sxy = s_v[2][e][nd], syy = s_v[3][e][nd];
    const double Sy = s_v[4][e][nd], dys = s_v[5][e][nd];
    const double divu = uxx + uyy, divs = sxx + syy;
    // Rp / alpha and Rs / (2 alpha)
    const double Rp = fma(divu, divu, fma(uxx, uxx, fma(uyy, uyy, 2.0 * uxy * uyx)));
    const double Rs = fma(divu, divs, fma(uxx, sxx, fma(uyy, syy, fma(uxy, syx, uyx * sxy))));
    const double b = fma(so[l], Rp, fma(2.0, Rs, -(fma(dxs, Sx, dys * Sy) * a.invr[n])));
    a.b_out[n] = (wa * B.w[l]) * b;
  }
}

// ---------------------------------------------------------------------------
// Tangent fluxes at one node (sensitivity_flux_x/_y, sensitivity.jl:43-76):
//   Phi = (gamma-1) (eta - sigma |u|^2/2 - rho u . s_u)  [+ s_gamma rho e]
//   P~  = Phi + varsigma
//   fx  = (zx ux + mx sux + P~, zx uy + mx suy, zx, (eta + P~) ux + (E + P + Sigma) sux)
//   fy  = (zx uy + mx suy, zy uy + my suy + P~, zy, (eta + P~) uy + (E + P + Sigma) suy)
// The s_gamma term (direct dP/dgamma source, zero in the reference's 2D
// package) follows the 1D package (IGR_adjoints_1d/sensitivity.jl:36-41).
// ---------------------------------------------------------------------------
struct SensNode { double fx[4], fy[4]; };

__device__ __forceinline__ SensNode sens_phys(double g, double sg, double mx, double my, double r, double E, double S,
                                              double ir, double zx, double zy, double sr, double et, double vs) {
  SensNode o;
  const double ux = mx * ir, uy = my * ir;
  const double sux = (zx - ux * sr) * ir, suy = (zy - uy * sr) * ir;
  const double u2h = 0.5 * fma(ux, ux, uy * uy);
  const double P = (g - 1.0) * (E - r * u2h);
  double Phi = (g - 1.0) * (et - sr * u2h - r * fma(ux, sux, uy * suy));
  if (sg != 0.0) Phi = fma(sg, r * (E * ir - u2h), Phi);
  const double Pt = Phi + vs;
  const double etp = et + Pt, eps = E + P + S;
  const double f1 = fma(zx, uy, mx * suy);
  o.fx[0] = fma(zx, ux, fma(mx, sux, Pt)); o.fx[1] = f1; o.fx[2] = zx; o.fx[3] = fma(etp, ux, eps * sux);
  o.fy[0] = f1; o.fy[1] = fma(zy, uy, fma(my, suy, Pt)); o.fy[2] = zy; o.fy[3] = fma(etp, uy, eps * suy);
  return o;
}

struct SensHypArgs2D {
  const Tile2D* tiles; const Inst2D* inst; BasisDev B;
  const double *q[4], *invr, *S;   // primal stage input and its Sigma
  const double *s[4], *vs;         // tangent stage input and varsigma
  const double *sn[4];             // tangent at the step start (stages 2 and 3)
  const double *ws_x, *ws_y;       // primal |u_n| + c at x-face / y-face nodes of this stage
  double c0, c1, c2, s_gamma;
  double *so[4];                   // tangent stage output (may alias sn: pointwise)
  double *k_out[4];                // optional: raw tangent RHS
  int* status;
};

// The tangent fluxes, lifted with the primal wave speeds.
struct TangentStage {
  const SensHypArgs2D& a;
  double g;
  __device__ __forceinline__ FluxNode at(long long n) const {
    FluxNode f;
#pragma unroll
    for (int v = 0; v < 4; ++v) f.q[v] = a.s[v][n];
    const SensNode p = sens_phys(g, a.s_gamma, a.q[0][n], a.q[1][n], a.q[2][n], a.q[3][n], a.S[n], a.invr[n], f.q[0], f.q[1],
                                 f.q[2], f.q[3], a.vs[n]);
    f.fx0 = p.fx[0]; f.f1 = p.fx[1]; f.fx3 = p.fx[3]; f.fy1 = p.fy[1]; f.fy3 = p.fy[3];
    return f;
  }
  __device__ __forceinline__ double speed(int dir, long long n, double, double, bool) const {
    return dir == 0 ? a.ws_x[n] : a.ws_y[n];
  }
  __device__ __forceinline__ double qn(int v, long long n) const { return a.sn[v][n]; }
  __device__ __forceinline__ void put(int v, long long n, double x) const {
    if (a.k_out[v]) a.k_out[v][n] = x;
    if (a.so[v]) a.so[v][n] = x;
    if (a.status && nonfinite_bits(x)) flag_nonfinite(a.status);
  }
};

template <int NP>
__global__ void __launch_bounds__(2 * Tiling2D<NP>::NH) k2_sens_hyp_rk(SensHypArgs2D a) {
  __shared__ StageSmem<NP, false> sm;
  const Tile2D tl = a.tiles[blockIdx.x];
  const Inst2D I = a.inst[tl.inst];
  chained_start();
  dg_stage<NP, false>(TangentStage{a, I.gamma}, a.B, tl, I, a.c0, a.c1, a.c2, a.k_out[0] != nullptr, sm);
}

}  // namespace igrgpu
