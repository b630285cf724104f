// 2D continuous adjoint (optimise-then-discretise, conservative Pi form,
// IGR_adjoints_2d/adjoint_pde.jl:41-611) on the forward kernels' tiling.
//
// Backward in time the adjoint a = (a_mux, a_muy, a_rho, a_E) advances by
//   d_tau a = +div F_dag(q, a) - S_loc(q) a + S_Sigma(q, Pi),
// with the primal q and Sigma frozen at the stored snapshot for all three
// stages of a step. Everything that depends on the snapshot alone is computed
// once per step (k2_pde_prep): the ten local-source coefficients (the
// pointwise q-derivatives of div F, :138-217), the nodal velocity gradients,
// grad(Sigma)/rho and R_tr of the nonlocal source (:381-466), 1/rho and the
// LLF wave speeds. Each stage then runs
//   k2_pde_b   (alpha > 0)  b = alpha w_i w_j Jx Jy (div a_mu + grad a_E . u)  (:337-364, :490-493)
//   Pi solve   (alpha > 0)  the forward's SIP operator and solver kernels, warm start = previous Pi
//   k2_pde_rk               adjoint DG operator + sources + SSP-RK3 combination
// so a stage reads the adjoint once and writes it once, like the forward.
#pragma once
#include "igr2d_kernels.cuh"

namespace igrgpu {

// Local-source coefficients per node: S_loc = C a with
//   S_mux = a_mux C0 + a_muy C1 + a_E C2,  S_muy = a_mux C3 + a_muy C4 + a_E C5,
//   S_rho = a_mux C6 + a_muy C7 + a_E C8,  S_E = a_E C9.
constexpr int PDE_SRC = 10;
// Nonlocal-source primal fields per node: d_x u_x, d_x u_y, d_y u_x, d_y u_y
// (of the nodal velocity), d_x Sigma / rho, d_y Sigma / rho, R_tr.
constexpr int PDE_NL = 7;

struct PdePrepArgs2D {
  const Tile2D* tiles; const Inst2D* inst; BasisDev B;
  const double *q[4], *S;
  double* invr;            // 1 / rho
  double* src[PDE_SRC];
  double* nl[PDE_NL];      // nullptr entries: not needed (alpha = 0)
  double *ws_x, *ws_y;     // |u_x| + c, |u_y| + c
};

// What bounds it: FP64 issue (the source coefficients); the fourteen line derivatives are integer work in rolled loops.
template <int NP>
__global__ void __launch_bounds__(Tiling2D<NP>::NT) k2_pde_prep(PdePrepArgs2D a) {
  using TL = Tiling2D<NP>;
  constexpr int TE = TL::TE, NN = TL::NN;
  // mux, muy, rho, E, Sigma, u_x, u_y: x-derivatives (physical); the fields, then their y-derivatives; 1/rho
  __shared__ double s_dx[7][TE][NN], s_dy[7][TE][NN];
  __shared__ double s_ir[TE][NN];
  const Tile2D tl = a.tiles[blockIdx.x];
  const Inst2D I = a.inst[tl.inst];
  chained_start();
  const ElemView vr = elem_view<NP>(tl, I, 0), vc = elem_view<NP>(tl, I, 1);
  const BasisDev& B = a.B;
  const int nf = a.nl[0] ? 7 : 5;  // the velocity gradients serve the nonlocal source only
  if (vr.valid) {
    const int t = vr.t, e = vr.e;
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const long long n = vr.base + t * NP + i;
      const int nd = t * NP + i;
      const double mx = a.q[0][n], my = a.q[1][n], r = a.q[2][n], ir = 1.0 / r;
      s_ir[e][nd] = ir;
      s_dy[0][e][nd] = mx; s_dy[1][e][nd] = my; s_dy[2][e][nd] = r; s_dy[3][e][nd] = a.q[3][n]; s_dy[4][e][nd] = a.S[n];
      s_dy[5][e][nd] = mx * ir; s_dy[6][e][nd] = my * ir;
    }
    const FixScale sc = fix_scale(I.ijx);
#pragma unroll 1
    for (int v = 0; v < nf; ++v) {
      double f[NP], d[NP];
#pragma unroll
      for (int i = 0; i < NP; ++i) f[i] = s_dy[v][e][t * NP + i];
      line_rows<NP>(B, sc, f, d);
#pragma unroll
      for (int i = 0; i < NP; ++i) s_dx[v][e][t * NP + i] = d[i];
    }
  }
  __syncthreads();
  if (!vc.valid) return;
  const int t = vc.t, e = vc.e;
  double f0[NP], f1[NP], f3[NP], f4[NP], u0[NP], u1[NP];
#pragma unroll
  for (int l = 0; l < NP; ++l) {
    const int nd = l * NP + t;
    f0[l] = s_dy[0][e][nd]; f1[l] = s_dy[1][e][nd]; f3[l] = s_dy[3][e][nd]; f4[l] = s_dy[4][e][nd];
    u0[l] = s_dy[5][e][nd]; u1[l] = s_dy[6][e][nd];
  }
  const FixScale sc = fix_scale(I.ijy);
#pragma unroll 1
  for (int v = 0; v < nf; ++v) {  // in place: the column is the thread's own from here on
    double f[NP], d[NP];
#pragma unroll
    for (int l = 0; l < NP; ++l) f[l] = s_dy[v][e][l * NP + t];
    line_rows<NP>(B, sc, f, d);
#pragma unroll
    for (int l = 0; l < NP; ++l) s_dy[v][e][l * NP + t] = d[l];
  }
  const double g = I.gamma, gm = g - 1.0;
#pragma unroll
  for (int l = 0; l < NP; ++l) {
    const long long n = vc.base + l * NP + t;
    const int nd = l * NP + t;
    const double mxx = s_dx[0][e][nd], myx = s_dx[1][e][nd], rx = s_dx[2][e][nd], Ex = s_dx[3][e][nd], Sx = s_dx[4][e][nd];
    const double mxy = s_dy[0][e][nd], myy = s_dy[1][e][nd], ry = s_dy[2][e][nd], Ey = s_dy[3][e][nd], Sy = s_dy[4][e][nd];
    const double mx = f0[l], my = f1[l], en = f3[l], Sg = f4[l];
    const double ir = s_ir[e][nd], ir2 = ir * ir, ir3 = ir2 * ir;
    const double ux = u0[l], uy = u1[l];
    // quotient-rule velocity gradients of the local source (adjoint_pde.jl:163-164)
    const double uxx = (mxx - ux * rx) * ir, uyy = (myy - uy * ry) * ir;
    const double m2 = fma(mx, mx, my * my);
    const double P = gm * (en - m2 * (0.5 * ir));
    const double Hb = en + P + Sg;
    const double Pr = gm * fma(ux, ux, uy * uy) * 0.5;
    const double mdx = fma(mx, mxx, my * myx), mdy = fma(mx, mxy, my * myy);
    const double Pbx = fma(gm, Ex - mdx * ir + m2 * rx * (0.5 * ir2), Sx);
    const double Pby = fma(gm, Ey - mdy * ir + m2 * ry * (0.5 * ir2), Sy);
    const double dPx_dmx = gm * (mx * rx * ir2 - mxx * ir);
    const double dPx_dmy = gm * (my * rx * ir2 - myx * ir);
    const double dPx_dr = gm * (mdx * ir2 - m2 * rx * ir3);
    const double dPy_dmx = gm * (mx * ry * ir2 - mxy * ir);
    const double dPy_dmy = gm * (my * ry * ir2 - myy * ir);
    const double dPy_dr = gm * (mdy * ir2 - m2 * ry * ir3);
    const double HEx = Ex + Pbx, HEy = Ey + Pby;
    const double c0 = mxx * ir + uxx - mx * rx * ir2 + dPx_dmx + uyy;                                   // dmx/dmx
    const double c3 = dPx_dmy + mxy * ir - mx * ry * ir2;                                              // dmx/dmy
    const double c6 = -mxx * ux * ir + mx * (ux * rx * ir2 - uxx * ir) + dPx_dr - mxy * uy * ir +
                      mx * (uy * ry * ir2 - uyy * ir);                                                 // dmx/drho
    const double c1 = myx * ir - my * rx * ir2 + dPy_dmx;                                              // dmy/dmx
    const double c4 = uxx + myy * ir + uyy - my * ry * ir2 + dPy_dmy;                                  // dmy/dmy
    const double c7 = -myx * ux * ir + my * (ux * rx * ir2 - uxx * ir) - myy * uy * ir +
                      my * (uy * ry * ir2 - uyy * ir) + dPy_dr;                                        // dmy/drho
    const double c2 = dPx_dmx * ux + HEx * ir - gm * ux * uxx - Hb * rx * ir2 + dPy_dmx * uy - gm * ux * uyy;  // dE/dmx
    const double c5 = dPx_dmy * ux - gm * uy * uxx + dPy_dmy * uy + HEy * ir - gm * uy * uyy - Hb * ry * ir2;  // dE/dmy
    const double c8 = dPx_dr * ux - HEx * ux * ir + Pr * uxx + Hb * (ux * rx * ir2 - uxx * ir) + dPy_dr * uy -
                      HEy * uy * ir + Pr * uyy + Hb * (uy * ry * ir2 - uyy * ir);                      // dE/drho
    const double c9 = g * (uxx + uyy);                                                                 // dE/dE
    a.src[0][n] = c0; a.src[1][n] = c1; a.src[2][n] = c2; a.src[3][n] = c3; a.src[4][n] = c4;
    a.src[5][n] = c5; a.src[6][n] = c6; a.src[7][n] = c7; a.src[8][n] = c8; a.src[9][n] = c9;
    a.invr[n] = ir;
    const double cs = sqrt(g * P * ir);
    a.ws_x[n] = fabs(ux) + cs;
    a.ws_y[n] = fabs(uy) + cs;
    if (a.nl[0]) {
      // nodal-velocity gradients (adjoint_pde.jl:391-404)
      const double nxx = s_dx[5][e][nd], nyx = s_dx[6][e][nd];
      const double nxy = s_dy[5][e][nd], nyy = s_dy[6][e][nd];
      const double dv = nxx + nyy;
      double R = fma(dv, dv, nxx * nxx);
      R = fma(2.0 * nxy, nyx, R);
      R = fma(nyy, nyy, R);
      a.nl[0][n] = nxx; a.nl[1][n] = nyx; a.nl[2][n] = nxy; a.nl[3][n] = nyy;
      a.nl[4][n] = Sx * ir; a.nl[5][n] = Sy * ir; a.nl[6][n] = R;
    }
  }
}

// b = alpha w_i w_j Jx Jy (d_x a_mux + d_y a_muy + u_x d_x a_E + u_y d_y a_E)
struct PdeBArgs2D {
  const Tile2D* tiles; const Inst2D* inst; BasisDev B;
  const double *a[4], *mx, *my, *invr;
  double* b;
};

template <int NP>
__global__ void __launch_bounds__(Tiling2D<NP>::NT) k2_pde_b(PdeBArgs2D a) {
  using TL = Tiling2D<NP>;
  constexpr int TE = TL::TE, NN = TL::NN;
  __shared__ double s_d[2][TE][NN];  // d_x a_mux, d_x a_E
  const Tile2D tl = a.tiles[blockIdx.x];
  const Inst2D I = a.inst[tl.inst];
  chained_start();
  const ElemView vr = elem_view<NP>(tl, I, 0), vc = elem_view<NP>(tl, I, 1);
  const BasisDev& B = a.B;
  if (vr.valid) {
    const int t = vr.t, e = vr.e;
    double am[NP], aE[NP], d[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) { const long long n = vr.base + t * NP + i; am[i] = a.a[0][n]; aE[i] = a.a[3][n]; }
    const FixScale sc = fix_scale(I.ijx);
    line_rows<NP>(B, sc, am, d);
#pragma unroll
    for (int i = 0; i < NP; ++i) s_d[0][e][t * NP + i] = d[i];
    line_rows<NP>(B, sc, aE, d);
#pragma unroll
    for (int i = 0; i < NP; ++i) s_d[1][e][t * NP + i] = d[i];
  }
  __syncthreads();
  if (!vc.valid) return;
  const int t = vc.t, e = vc.e;
  double am[NP], aE[NP], acc[NP], div[NP], aEy[NP];
#pragma unroll
  for (int l = 0; l < NP; ++l) {
    const long long n = vc.base + l * NP + t;
    am[l] = a.a[1][n]; aE[l] = a.a[3][n]; acc[l] = s_d[0][e][l * NP + t];
  }
  const FixScale sc = fix_scale(I.ijy);
  line_rows_acc<NP>(B, sc, am, acc, div);  // d_x a_mux + d_y a_muy
  line_rows<NP>(B, sc, aE, aEy);
  const double cw = I.alpha * B.w[t] * I.jx * I.jy;
#pragma unroll
  for (int l = 0; l < NP; ++l) {
    const long long n = vc.base + l * NP + t;
    const int nd = l * NP + t;
    const double ir = a.invr[n];
    const double ux = a.mx[n] * ir, uy = a.my[n] * ir;
    const double v = fma(aEy[l], uy, fma(s_d[1][e][nd], ux, div[l]));
    a.b[n] = v * (cw * B.w[l]);
  }
}

// Adjoint DG operator + sources + SSP-RK3 stage:
//   k = +(1/Jx) D fx + (1/Jy) D fy + face terms - C a + S_Sigma,
//   a_out = c0 a^n + c1 a_s + c2 dt k.
struct PdeRkArgs2D {
  const Tile2D* tiles; const Inst2D* inst; BasisDev B;
  const double *q[4], *S, *invr, *ws_x, *ws_y;   // snapshot
  const double* src[PDE_SRC];
  const double* nl[PDE_NL];
  const double* Pi;                              // nullptr: no nonlocal source (alpha = 0)
  const double *a[4];                            // stage input
  const double *an[4];                           // step start (read when c0 != 0)
  double c0, c1, c2;
  double* ao[4];                                 // stage output (may alias an, not a)
  double* k_out[4];                              // optional: the raw operator k
};

// Adjoint flux F_dag in both directions at one node (adjoint_pde.jl:41-80).
struct AdjFlux { double fx[4], fy[4]; };
__device__ __forceinline__ AdjFlux pde_adjoint_flux(double g, double mx, double my, double r, double E, double S,
                                                    double ir, const double a[4]) {
  const double gm = g - 1.0;
  const double ux = mx * ir, uy = my * ir;
  const double P = gm * (E - fma(mx, mx, my * my) * (0.5 * ir));
  const double Hr = (E + P + S) * ir;            // H_bar / rho
  const double Pr = gm * fma(ux, ux, uy * uy) * 0.5;
  const double amu = fma(a[0], ux, a[1] * uy);   // (a_mu . mu) / rho
  const double aEg = a[3] * gm;
  AdjFlux F;
  // x: P_mux = -gm ux, P_muy = -gm uy
  F.fx[0] = fma(a[3], Hr, amu + a[0] * ux - gm * ux * a[0] + a[2]) - aEg * ux * ux;
  F.fx[1] = a[1] * ux - gm * uy * a[0] - aEg * uy * ux;
  F.fx[2] = fma(a[3] * ux, Pr - Hr, Pr * a[0] - ux * amu);
  F.fx[3] = fma(gm, a[0], a[3] * g * ux);
  F.fy[0] = a[0] * uy - gm * ux * a[1] - aEg * ux * uy;
  F.fy[1] = fma(a[3], Hr, amu + a[1] * uy - gm * uy * a[1] + a[2]) - aEg * uy * uy;
  F.fy[2] = fma(a[3] * uy, Pr - Hr, Pr * a[1] - uy * amu);
  F.fy[3] = fma(gm, a[1], a[3] * g * uy);
  return F;
}

// What bounds it: FP64 issue (adjoint fluxes, sources, faces). Volume terms and the nonlocal source's derivatives are
// integer line operations; the faces take f_partner - f_own - lambda (a_L - a_R) (see llf_jump). 8 x 128^2 P3: 793 us with
// FP64 contractions, 544 us with integer ones, 595 us with sums without a mean error and the leading-node checks; k2_pde_prep
// and k2_pde_b together 285, 165 and 170 us per launch on average.
template <int NP>
__global__ void __launch_bounds__(Tiling2D<NP>::NT) k2_pde_rk(PdeRkArgs2D a) {
  using TL = Tiling2D<NP>;
  constexpr int TE = TL::TE, NN = TL::NN, L = TL::L, TX = TL::TX, TY = TL::TY;
  __shared__ double s_fy[4][TE][NN];    // adjoint y fluxes
  __shared__ double s_k[4][TE][NN];     // x fluxes, then the operator's x part
  __shared__ double s_a[4][TE][NN];     // adjoint stage input
  __shared__ double s_w[3][TE][NN];     // nonlocal source: x products, then the x-derivative parts of W_x, W_y, div C
  __shared__ double s_fx[4][TE][NP][2]; // x fluxes at the row ends (left, right)
  __shared__ double s_wx[TE][NP][2];    // wave speeds there
  const Tile2D tl = a.tiles[blockIdx.x];
  const Inst2D I = a.inst[tl.inst];
  chained_start();
  const ElemView vr = elem_view<NP>(tl, I, 0), vc = elem_view<NP>(tl, I, 1);
  const BasisDev& B = a.B;
  const double g = I.gamma;
  const double invJx = I.ijx, invJy = I.ijy;
  const bool nonlocal = a.Pi != nullptr;
  auto ends = [](int k) { return k == 0 || k == L; };
  auto flux = [&](long long n, const double av[4]) {
    return pde_adjoint_flux(g, a.q[0][n], a.q[1][n], a.q[2][n], a.q[3][n], a.S[n], a.invr[n], av);
  };

  // ---- phase 1 (row of vr): adjoint fluxes, x-face data, products of the nonlocal source
  if (vr.valid) {
    const int t = vr.t, e = vr.e;
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const long long n = vr.base + t * NP + i;
      const int nd = t * NP + i;
      const double av[4] = {a.a[0][n], a.a[1][n], a.a[2][n], a.a[3][n]};
      const AdjFlux F = flux(n, av);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        s_k[c][e][nd] = F.fx[c]; s_fy[c][e][nd] = F.fy[c]; s_a[c][e][nd] = av[c];
        if (i == 0 || i == L) s_fx[c][e][t][i == 0 ? 0 : 1] = F.fx[c];
      }
      if (i == 0 || i == L) s_wx[e][t][i == 0 ? 0 : 1] = a.ws_x[n];
      if (nonlocal) {
        const double P = a.Pi[n], nxx = a.nl[0][n], nxy = a.nl[2][n], nyy = a.nl[3][n];
        s_w[0][e][nd] = P * (nxx + nyy + nxx); s_w[1][e][nd] = P * nxy; s_w[2][e][nd] = P * a.nl[4][n];
      }
    }
    if (nonlocal) {
      const FixScale sc = fix_scale(invJx);
#pragma unroll 1
      for (int v = 0; v < 3; ++v) {
        double f[NP], d[NP];
#pragma unroll
        for (int i = 0; i < NP; ++i) f[i] = s_w[v][e][t * NP + i];
        line_rows<NP>(B, sc, f, d);
#pragma unroll
        for (int i = 0; i < NP; ++i) s_w[v][e][t * NP + i] = d[i];
      }
    }
  }
  __syncthreads();
  // ---- phase 2 (row of vr): x volume term and x faces; adjoint LLF (adjoint_pde.jl:89-128) with the
  // forward's face signs flipped (:275-289); the owner computes its side
  if (vr.valid) {
    const int t = vr.t, e = vr.e;
    double pa[2][4], pf[2][4], lam[2];
    const int sf = first_side(vr.ext, TX);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int s = h == 0 ? sf : 1 - sf;
      int it;
      const long long pb = neighbour<NP>(tl, I, vr.ex, vr.ey, s == 0 ? -1 : 1, 0, &it);
      const int nd = t * NP + (s == 0 ? L : 0);
      double av[4], fv[4], ws;
      if (it >= 0) {
#pragma unroll
        for (int c = 0; c < 4; ++c) { av[c] = s_a[c][it][nd]; fv[c] = s_fx[c][it][t][1 - s]; }
        ws = s_wx[it][t][1 - s];
      } else {
        const long long n = pb + nd;
#pragma unroll
        for (int c = 0; c < 4; ++c) av[c] = a.a[c][n];
        const AdjFlux F = flux(n, av);
#pragma unroll
        for (int c = 0; c < 4; ++c) fv[c] = F.fx[c];
        ws = a.ws_x[n];
      }
      const double own = s_wx[e][t][s];
      const double mag = s == 0 ? max_nonneg(own, ws) : max_nonneg(ws, own);
#pragma unroll
      for (int d = 0; d < 2; ++d) {  // register arrays by the run-time side
        if (d != s) continue;
        lam[d] = mag;
#pragma unroll
        for (int c = 0; c < 4; ++c) { pa[d][c] = av[c]; pf[d][c] = fv[c]; }
      }
    }
    // fs - f_own = (f_partner - f_own - lambda (a_L - a_R)) / 2; a_L - a_R = +-(a_partner - a_own)
    const double cf0 = -0.5 * invJx * B.iw0, cfL = 0.5 * invJx * B.iwL;
    const FixScale sc = fix_scale(invJx);
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
      double f[NP], acc[NP], k[NP];
#pragma unroll
      for (int i = 0; i < NP; ++i) f[i] = s_k[c][e][t * NP + i];
      acc[0] = cf0 * llf_jump(pick4(pf[0], c), f[0], -lam[0], pick4(pa[0], c) - s_a[c][e][t * NP]);
      acc[L] = cfL * llf_jump(pick4(pf[1], c), f[L], lam[1], pick4(pa[1], c) - s_a[c][e][t * NP + L]);
      line_op<NP, false, true, true>(B.fD, B.D, &sc, f, acc, ends, k);
#pragma unroll
      for (int i = 0; i < NP; ++i) s_k[c][e][t * NP + i] = k[i];
    }
  }
  __syncthreads();
  if (!vc.valid) return;
  // ---- phase 3 (column of vc): y volume term, y faces, sources, RK combination
  const int t = vc.t, e = vc.e;
  double pa[2][4], pf[2][4], lam[2];
  {
    const int sf = first_side(vc.eyt, TY);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int s = h == 0 ? sf : 1 - sf;
      int it;
      const long long pb = neighbour<NP>(tl, I, vc.ex, vc.ey, 0, s == 0 ? -1 : 1, &it);
      const int nd = (s == 0 ? L : 0) * NP + t;
      double av[4], fv[4];
      if (it >= 0) {
#pragma unroll
        for (int c = 0; c < 4; ++c) { av[c] = s_a[c][it][nd]; fv[c] = s_fy[c][it][nd]; }
      } else {
        const long long n = pb + nd;
#pragma unroll
        for (int c = 0; c < 4; ++c) av[c] = a.a[c][n];
        const AdjFlux F = flux(n, av);
#pragma unroll
        for (int c = 0; c < 4; ++c) fv[c] = F.fy[c];
      }
      const double ws = a.ws_y[pb + nd], own = a.ws_y[vc.base + (s == 0 ? 0 : L) * NP + t];
      const double mag = s == 0 ? max_nonneg(own, ws) : max_nonneg(ws, own);
#pragma unroll
      for (int d = 0; d < 2; ++d) {
        if (d != s) continue;
        lam[d] = mag;
#pragma unroll
        for (int c = 0; c < 4; ++c) { pa[d][c] = av[c]; pf[d][c] = fv[c]; }
      }
    }
  }
  const FixScale sc = fix_scale(invJy);
  // nonlocal source, y parts (adjoint_pde.jl:420-466)
  double Wx[NP], Wy[NP], dC[NP];
  if (nonlocal) {
    double f[3][NP], acc[NP];
#pragma unroll
    for (int l = 0; l < NP; ++l) {
      const long long n = vc.base + l * NP + t;
      const double P = a.Pi[n], nyy = a.nl[3][n];
      f[0][l] = P * a.nl[1][n]; f[1][l] = P * (a.nl[0][n] + nyy + nyy); f[2][l] = P * a.nl[5][n];
    }
#pragma unroll
    for (int l = 0; l < NP; ++l) acc[l] = s_w[0][e][l * NP + t];
    line_rows_acc<NP>(B, sc, f[0], acc, Wx);
#pragma unroll
    for (int l = 0; l < NP; ++l) acc[l] = s_w[1][e][l * NP + t];
    line_rows_acc<NP>(B, sc, f[1], acc, Wy);
#pragma unroll
    for (int l = 0; l < NP; ++l) acc[l] = s_w[2][e][l * NP + t];
    line_rows_acc<NP>(B, sc, f[2], acc, dC);
  }
  // the sources and the x part, summed with the y part
  double kc[4][NP];
#pragma unroll
  for (int l = 0; l < NP; ++l) {
    const long long n = vc.base + l * NP + t;
    const int nd = l * NP + t;
    const double a0 = s_a[0][e][nd], a1 = s_a[1][e][nd], a3 = s_a[3][e][nd];
    // minus the local source
    kc[0][l] = s_k[0][e][nd] - fma(a0, a.src[0][n], fma(a1, a.src[1][n], a3 * a.src[2][n]));
    kc[1][l] = s_k[1][e][nd] - fma(a0, a.src[3][n], fma(a1, a.src[4][n], a3 * a.src[5][n]));
    kc[2][l] = s_k[2][e][nd] - fma(a0, a.src[6][n], fma(a1, a.src[7][n], a3 * a.src[8][n]));
    kc[3][l] = fma(-a3, a.src[9][n], s_k[3][e][nd]);
    if (nonlocal) {
      const double ir = a.invr[n], ir2 = -2.0 * ir;
      kc[0][l] = fma(Wx[l], ir2, kc[0][l]);
      kc[1][l] = fma(Wy[l], ir2, kc[1][l]);
      const double wm = fma(Wx[l], a.q[0][n], Wy[l] * a.q[1][n]);
      kc[2][l] = fma(fma(a.Pi[n], a.nl[6][n], dC[l]) - wm * ir2, ir, kc[2][l]);
    }
  }
  const double cf0 = -0.5 * invJy * B.iw0, cfL = 0.5 * invJy * B.iwL;
  const double c2dt = a.c2 * I.dt;
  const bool with_an = __double_as_longlong(a.c0) != 0;
#pragma unroll 1
  for (int c = 0; c < 4; ++c) {
    double f[NP], acc[NP], k[NP];
#pragma unroll
    for (int l = 0; l < NP; ++l) {
      f[l] = s_fy[c][e][l * NP + t];
      const double r[4] = {kc[0][l], kc[1][l], kc[2][l], kc[3][l]};
      acc[l] = pick4(r, c);
    }
    acc[0] = fma(cf0, llf_jump(pick4(pf[0], c), f[0], -lam[0], pick4(pa[0], c) - s_a[c][e][t]), acc[0]);
    acc[L] = fma(cfL, llf_jump(pick4(pf[1], c), f[L], lam[1], pick4(pa[1], c) - s_a[c][e][L * NP + t]), acc[L]);
    line_rows_acc<NP>(B, sc, f, acc, k);
#pragma unroll
    for (int l = 0; l < NP; ++l) {
      const long long n = vc.base + l * NP + t;
      if (a.k_out[c]) a.k_out[c][n] = k[l];
      double val = fma(c2dt, k[l], a.c1 * s_a[c][e][l * NP + t]);
      if (with_an) val = fma(a.c0, a.an[c][n], val);
      if (a.ao[c]) a.ao[c][n] = val;
    }
  }
}

}  // namespace igrgpu
