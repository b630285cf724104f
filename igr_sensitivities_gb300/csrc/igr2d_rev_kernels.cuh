// 2D discrete-adjoint (reverse-mode) kernels: the transpose of every forward
// kernel in igr2d_kernels.cuh, in the same tile / line-per-thread layout and
// with the same phase-dependent thread mapping (elem_view).
//
// What the reference gets from Enzyme (IGR_adjoints_2d/enzyme_adjoint.jl:270-296)
// is built here by hand, primitive by primitive:
//   k2_hyp_rev    reverse of the LLF/DG hyperbolic RHS and of the SSP-RK3
//                 stage combination; its epilogue starts the reverse of the
//                 fixed-count solver (the last iteration is pointwise);
//   k2_apply_rev  one reverse solver iteration: A u for the residual adjoint u
//                 (A is symmetric, elliptic.jl:30-145) plus the adjoint of the
//                 operator coefficients, d(u^T A(rho, alpha) x_k), against the
//                 taped iterate x_k;
//   k2_setup_rev  reverse of the IGR source (elliptic.jl:159-197) and of
//                 diag(A) (elliptic.jl:205-264), closing d/d rho and d/d alpha.
// Conventions at kinks follow the reference's Float64 Base functions:
// d|u|/du = +1 at u = +0.0, and max(a, b) differentiates into a on ties.
//
// Coefficient adjoints are carried as Z = (1/rho) * d(.)/d(1/rho) so that the
// stored coefficients (all proportional to 1/rho) are reused directly:
// Zm collects the mass part without its coefficient (the sum over the
// solve's reverse applies of +-u x, which k2_setup_rev multiplies by the mass
// coefficient once, instead of every apply), Zs the alpha-proportional
// stiffness/face part; then d/d rho = -Z/rho and d/d alpha = Zs/alpha.
#pragma once
#include "igr2d_kernels.cuh"

namespace igrgpu {

// Reverse of node_phys for both flux directions at one node: fbx, fby are
// the adjoints of the x and y flux components; accumulates into qb[4]
// (mx, my, rho, E) and sets Sb and gb. With u = m / rho, H = (E + P + Sigma) /
// rho, e3 = fbx_3 u_x + fby_3 u_y, pb = fbx_0 + fby_1 + e3 (d/dP_bar) and
// k = -(g-1) pb - T, where T is what the node's wave speeds add to d/dE
// (wavespeed_rev), the flux components and the kinetic part of the pressure
// collect to
//   d/dmx  = u_x (2 fbx_0 + k) + u_y (fbx_1 + fby_0) + fbx_2 + fbx_3 H
//   d/dmy  = u_y (2 fby_1 + k) + u_x (fbx_1 + fby_0) + fby_2 + fby_3 H
//   d/drho = -[u_x^2 (2 fbx_0 + k) / 2 + u_y^2 (2 fby_1 + k) / 2 + u_x u_y (fbx_1 + fby_0) + e3 H]
//   d/dE   = e3 - k.
__device__ __forceinline__ void node_phys_rev(double g, double mx, double my, double E, double S, double ir,
                                              const double fbx[4], const double fby[4], double T, double qb[4], double& Sb,
                                              double& gb) {
  const double ux = mx * ir, uy = my * ir;
  const double gm1 = g - 1.0;
  const double Ek = fma(-0.5, fma(mx, ux, my * uy), E);
  const double H = fma(gm1, Ek, E + S) * ir;
  const double e3 = fma(fbx[3], ux, fby[3] * uy);
  const double pb = fbx[0] + fby[1] + e3;
  const double k = fma(-gm1, pb, -T);
  const double c = fbx[1] + fby[0];
  const double p = ux * fma(2.0, fbx[0], k), q = uy * fma(2.0, fby[1], k), r = c * uy;
  qb[0] = fma(fbx[3], H, qb[0]) + fbx[2] + (p + r);
  qb[1] = fma(c, ux, fma(fby[3], H, qb[1])) + fby[2] + q;
  qb[2] = fma(-ux, fma(0.5, p, r), fma(-uy, 0.5 * q, fma(-e3, H, qb[2])));
  qb[3] += e3 - k;
  Sb = pb;
  gb = pb * Ek;
}

// Reverse of |u_n| + c, c = sqrt(g P / rho), at one node with adjoint wb. With
// Y = wb c / 2 it adds the sign of u_n / rho times wb to the normal momentum,
// -Y / rho - (that) u_n to rho, Y (1/g + 1/(g - 1)) (gs is that factor) to
// d/dgamma, and returns T = (wb / 2c) g (g - 1) / rho, its d/dE: the rest,
// -T u to the momenta and T |u|^2 / 2 to rho, joins node_phys_rev.
__device__ __forceinline__ double wavespeed_rev(double g, double gs, double mn, double ir, double ws, double wb, double& qn,
                                                double& qr, double& gb) {
  const double un = mn * ir;
  const double c = ws - fabs(un);
  const double h = 0.5 * wb, Y = h * c;
  const double t = (signbit(un) ? -wb : wb) * ir;
  gb = fma(Y, gs, gb);
  qn += t;
  qr = fma(-Y, ir, fma(-t, un, qr));
  return (h / c) * ((g * (g - 1.0)) * ir);
}

enum { SREV_NONE = 0, SREV_CHEB = 1, SREV_JACOBI = 2, SREV_PCG = 3 };

// ---------------------------------------------------------------------------
// Reverse of k2_hyp_rk for one stage.
//   forward: q_out = c0 q^n + c1 q_s + c2 dt k(q_s, Sigma)
//   given A = adjoint of q_out:
//     Qn  (+)= c0 A                        (qn_mode: 0 skip, 1 write, 2 add)
//     Qs  (+)= c1 A + H_q^T(c2 dt A)        (qs_add: add instead of write)
//     Sb  (+)= H_S^T(c2 dt A)               (Sb_add)
//     gnode += d/dgamma
// Solver prologue (SREV_CHEB / SREV_JACOBI) with xb = Sb total: produces the
// residual adjoint u = rb_{n-1} for the first k2_apply_rev, initialises the
// adjoint iMb of 1/diag(A) (the forward multiplies by the stored reciprocal),
// and (Chebyshev) the direction adjoint db.
// ---------------------------------------------------------------------------
struct HypRevArgs2D {
  const Tile2D* tiles; const Inst2D* inst; BasisDev B;
  const double *q[4], *invr, *S;     // taped stage input and Sigma_out
  const double *ws_x, *ws_y;         // taped LLF wave speeds at face nodes
  const double *A[4];                // adjoint of the stage output
  double c0, c1, c2;
  double *Qn[4]; int qn_mode;
  double *Qs[4]; int qs_add;
  double *Sb; int Sb_add;
  double *gnode;                     // per-node dJ/dgamma accumulator
  // solver prologue
  int srev;
  const double *cinvM, *r_last;      // taped r_{n-1}
  double *u_out, *db, *iMb;
  double ca, cc, omega;              // Chebyshev a_n, c_n ; Jacobi omega
};

// Rows and columns run side by side, one half of the CTA each; the node work (flux reverse, combination) is spread over
// all threads. What bounds it: FP64 issue. The transposed volume terms run on the integer pipes with the stage
// coefficient and the own side of the face corrections in their matrix; a face takes 5 FP64 instructions per component.
// 8 x 128^2 P3: 680 us with FP64 contractions; 442 with integer ones; 360 with the shorter faces and node reverse; 394 with
// IEEE divides again (pipe 84% busy). 64^2: 40.8, 37.8, and 23.6 in halves.
template <int NP>
__global__ void __launch_bounds__(2 * Tiling2D<NP>::NH) k2_hyp_rev(HypRevArgs2D a) {
  using TL = Tiling2D<NP>;
  constexpr int TE = TL::TE, NN = TL::NN, L = TL::L, TX = TL::TX, NH = TL::NH;
  constexpr int NQ = (TE * NN + 2 * NH - 1) / (2 * NH);  // nodes per thread
  __shared__ double s_A[4][TE][NN];         // adjoint of the stage output; [0] last holds the nodes' d/dgamma
  __shared__ double s_q[4][TE][NN];         // taped stage state
  __shared__ double s_fb[2][4][TE][NN];     // adjoints of the x and y fluxes
  __shared__ double s_qb[2][4][TE][NP][2];  // state adjoints from the faces, at the line ends
  __shared__ double s_w[2][TE][NP][2];      // wave speeds at the line ends
  __shared__ double s_T[2][TE][NP][2];      // what their wave speeds add to d/dE (wavespeed_rev)
  __shared__ double s_g[2][TE][NP];         // the lines' d/dgamma
  const Tile2D tl = a.tiles[blockIdx.x];
  const Inst2D I = a.inst[tl.inst];
  chained_start();
  const BasisDev& B = a.B;
  const double g = I.gamma;
  const double c2dt = a.c2 * I.dt;
  const int dir = threadIdx.x >= NH;  // 0: rows and x faces, 1: columns and y faces
  const ElemView w = elem_view<NP>(tl, I, dir, threadIdx.x - dir * NH);
  const int e = w.e, t = w.t;
  const int st = dir == 0 ? 1 : NP, at = dir == 0 ? t * NP : t;  // node k of the line: at + k st
  const double* ws = dir == 0 ? a.ws_x : a.ws_y;

  // ---- node data into shared memory
  long long node[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const int m = threadIdx.x + q * 2 * NH;
    const int el = m / NN, nd = m % NN, ex = tl.ex0 + el % TX, ey = tl.ey0 + el / TX;
    const bool live = m < TE * NN && ex < I.nex && ey < I.ney;
    const long long n = I.off + (long long)NN * (ex + (long long)I.nex * ey) + nd;
    node[q] = live ? n : -1;
    if (!live) continue;
#pragma unroll
    for (int c = 0; c < 4; ++c) { s_q[c][el][nd] = a.q[c][n]; s_A[c][el][nd] = a.A[c][n]; }
  }
  if (w.valid) {
    s_w[dir][e][t][0] = ws[w.base + at];
    s_w[dir][e][t][1] = ws[w.base + at + L * st];
  }
  __syncthreads();

  // ---- one line of all four components. Its flux adjoints are the transposed volume term of kbar = c2 dt A plus, at the
  // end nodes, the LLF flux's reverse: with x = coefficient of the own correction times kbar / 2 and y the partner's, the
  // own flux gets y - x (-x sits in the matrix, fDr), the own state +-lambda (x + y), and lambda (x + y) dq. The
  // components stay a rolled loop: its body is a few hundred integer instructions.
  if (w.valid) {
    const double ci = c2dt * (dir == 0 ? I.ijx : I.ijy);
    const FixScale sc = fix_scale(-ci);
    long long pn[2];
    int it[2];
    double lam[2], cfo[2], cfp[2], lamb[2];
    bool wins[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int d = s == 0 ? -1 : 1;
      const long long pb = neighbour<NP>(tl, I, w.ex, w.ey, dir == 0 ? d : 0, dir == 0 ? 0 : d, &it[s]);
      pn[s] = pb + at + (s == 0 ? L : 0) * st;
      const double own = s_w[dir][e][t][s], par = it[s] >= 0 ? s_w[dir][it[s] >= 0 ? it[s] : 0][t][1 - s] : ws[pn[s]];
      const double mag = s == 0 ? max_nonneg(own, par) : max_nonneg(par, own);  // max(ws_R, ws_L)
      wins[s] = s == 0 ? gt_nonneg(own, par) : !gt_nonneg(par, own);
      lam[s] = s == 0 ? -mag : mag;
      // correction coefficients: R side (node 0) +invJ/w0, L side (node L) -invJ/wL
      cfo[s] = s == 0 ? 0.5 * ci * B.iw0 : -0.5 * ci * B.iwL;
      cfp[s] = s == 0 ? -0.5 * ci * B.iwL : 0.5 * ci * B.iw0;
      lamb[s] = 0.0;
    }
#pragma unroll 1
    for (int v = 0; v < 4; ++v) {
      double A[NP], acc[NP], fb[NP];
#pragma unroll
      for (int k = 0; k < NP; ++k) A[k] = s_A[v][e][at + k * st];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int nd = at + (s == 0 ? L : 0) * st;
        const double pA = it[s] >= 0 ? s_A[v][it[s] >= 0 ? it[s] : 0][nd] : a.A[v][pn[s]];
        const double pq = it[s] >= 0 ? s_q[v][it[s] >= 0 ? it[s] : 0][nd] : a.q[v][pn[s]];
        const double oq = s_q[v][e][at + (s == 0 ? 0 : L) * st];
        const double y = cfp[s] * pA, h = fma(cfo[s], A[s == 0 ? 0 : L], y);
        acc[s == 0 ? 0 : L] = y;
        s_qb[dir][v][e][t][s] = lam[s] * h;
        lamb[s] = fma(h, s == 0 ? pq - oq : oq - pq, lamb[s]);  // q_L - q_R
      }
      line_op<NP, true, true, true>(B.fDr, B.Dr, &sc, A, acc, [](int k) { return k == 0 || k == L; }, fb);
#pragma unroll
      for (int k = 0; k < NP; ++k) s_fb[dir][v][e][at + k * st] = fb[k];
    }
    // reverse of the wave speed where the own side sets lambda
    double gb = 0.0;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      double T = 0.0;
      if (wins[s]) {
        const int nd = at + (s == 0 ? 0 : L) * st;
        double qn = s_qb[dir][dir][e][t][s], qr = s_qb[dir][2][e][t][s];
        T = wavespeed_rev(g, I.gsum, s_q[dir][e][nd], a.invr[w.base + nd], s_w[dir][e][t][s], lamb[s], qn, qr, gb);
        s_qb[dir][dir][e][t][s] = qn;
        s_qb[dir][2][e][t][s] = qr;
      }
      s_T[dir][e][t][s] = T;
    }
    s_g[dir][e][t] = gb;
  }
  // ---- nodes: merged flux reverse, combination, outputs. What they read is loaded before the barrier and before anything
  // is stored.
  double S[NQ], ir[NQ], Sb[NQ], Qn[NQ][4], Qs[NQ][4], im[NQ], rl[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const long long n = node[q];
    if (n < 0) continue;
    S[q] = a.S[n];
    ir[q] = a.invr[n];
    Sb[q] = a.Sb_add ? a.Sb[n] : 0.0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      Qn[q][c] = a.qn_mode == 2 ? a.Qn[c][n] : 0.0;
      Qs[q][c] = a.qs_add ? a.Qs[c][n] : 0.0;
    }
    if (a.srev != SREV_NONE) {
      im[q] = a.cinvM[n];
      rl[q] = a.r_last[n];
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const long long n = node[q];
    if (n < 0) continue;
    const int m = threadIdx.x + q * 2 * NH;
    const int el = m / NN, nd = m % NN, j = nd / NP, i = nd % NP;
    double fbx[4], fby[4], qq[4], A[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      fbx[c] = s_fb[0][c][el][nd]; fby[c] = s_fb[1][c][el][nd]; A[c] = s_A[c][el][nd];
      qq[c] = (i == 0 || i == L) ? s_qb[0][c][el][j][i == 0 ? 0 : 1] : 0.0;
      if (j == 0 || j == L) qq[c] += s_qb[1][c][el][i][j == 0 ? 0 : 1];
    }
    double T = (i == 0 || i == L) ? s_T[0][el][j][i == 0 ? 0 : 1] : 0.0;
    if (j == 0 || j == L) T += s_T[1][el][i][j == 0 ? 0 : 1];
    double sb, gb;
    node_phys_rev(g, s_q[0][el][nd], s_q[1][el][nd], s_q[3][el][nd], S[q], ir[q], fbx, fby, T, qq, sb, gb);
    s_A[0][el][nd] = gb;  // read by this thread alone so far
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (a.qn_mode == 1) a.Qn[c][n] = a.c0 * A[c];
      else if (a.qn_mode == 2) a.Qn[c][n] = fma(a.c0, A[c], Qn[q][c]);
      const double val = fma(a.c1, A[c], qq[c]);
      a.Qs[c][n] = a.qs_add ? Qs[q][c] + val : val;
    }
    const double Sbt = a.Sb_add ? Sb[q] + sb : sb;
    a.Sb[n] = Sbt;
    if (a.srev == SREV_CHEB) {
      // x_n = x_{n-1} + d_n ; d_n = a_n d_{n-1} + c_n z_n ; z_n = (1/M) r_{n-1}
      const double zb = a.cc * Sbt;
      a.u_out[n] = im[q] * zb;
      a.iMb[n] = zb * rl[q];
      a.db[n] = a.ca * Sbt;
    } else if (a.srev == SREV_JACOBI) {
      // x_n = x_{n-1} + (omega r_{n-1}) (1/M)
      const double tb = a.omega * Sbt;
      a.u_out[n] = tb * im[q];
      a.iMb[n] = tb * rl[q];
    }
  }
  __syncthreads();
  if (dir == 1 && w.valid) {
    double gb = s_g[0][e][t] + s_g[1][e][t];
#pragma unroll
    for (int l = 0; l < NP; ++l) gb += s_A[0][e][l * NP + t];
    a.gnode[w.base + t] += gb;
  }
}

// ---------------------------------------------------------------------------
// One reverse solver iteration m: u = residual adjoint r̄_m, x_m taped.
//   xb -= A u ; bb (+)= u ; Zm/Zs (+)= -(mass / stiffness+face parts of
//   d(u^T A x_m) in Z form); then the solver epilogue builds r̄_{m-1}.
// ---------------------------------------------------------------------------
struct ApplyRevArgs2D {
  const Tile2D* tiles; const Inst2D* inst; BasisDev B;
  const double *u, *xk;               // residual adjoint and taped iterate
  const double *cm, *ckx, *cky, *cpx, *cpy, *cinvM, *invr;
  double *xb, *bb, *Zm, *Zs;
  int first;                          // first reverse apply of this solve: write Zm, Zs (else add)
  int bb_op;                          // bb: 0 untouched, 1 write u, 2 add u
  double zscale;                      // -1 for r = b - A x terms
  // epilogue (when has_next): r̄_{m-1}
  int has_next;
  const double* r_prev;               // taped r_{m-1}
  double *u_out, *db, *iMb;
  double ca, cc, omega;
  // SREV_PCG (reverse of A p_it, second half of the iteration reverse):
  //   u = -(adjoint of A p_it) = alpha_it rb - pApb p_it, formed on load from
  //   (u = rb, xk = p_it); xb = pb: pb += alpha_it xconst + pApb apk + A(adjoint of A p_it);
  //   with has_next, the tile's partial of pb . p_next (betab of the next reverse
  //   iteration) goes to partials[tile] and the instance's last block completes it (isum, mode 2)
  const double *al_it, *papb;  // per-instance alpha_it (tape) and the adjoint of pAp_it
  const double *xconst, *apk, *p_next;
  double* partials;
  InstSum isum;
};

// Partner data across one face for the reverse apply: values of u and x_k, the flux of u at the face node and 1/rho.
struct Partner2 { double u, v, t, ir; };

// Rows and columns run side by side, one half of the CTA each, and the outputs are pointwise over all threads (see
// k2_apply). What bounds it: FP64 issue (60% busy) and the integer ALU (56%). 8 x 128^2 P3, Chebyshev: 226 us with FP64
// contractions; 140 us with integer ones and one thread per pair of lines; in halves, with the pointwise loads ahead of
// its stores, 114 us at seven CTAs per SM (72 registers; 137 us at the 80 the compiler takes); 126 us with sums without a
// mean error and the leading-node checks. 64^2: 18.9, 17.4, 12.4.
template <int NP, int SREV>
__global__ void __launch_bounds__(2 * Tiling2D<NP>::NH, NP == 4 ? 7 : 1) k2_apply_rev(ApplyRevArgs2D a) {
  using TL = Tiling2D<NP>;
  constexpr int TE = TL::TE, NN = TL::NN, SN = TL::SN, L = TL::L, TX = TL::TX, TY = TL::TY, NH = TL::NH;
  constexpr bool PCG = SREV == SREV_PCG;
  constexpr int P2 = pow2_at_least(2 * NH);
  __shared__ __align__(16) double s_u[TE][SN], s_v[TE][SN];
  __shared__ __align__(16) long long s_y[2][TE][SN], s_z[2][TE][SN];  // sums and products of rows and columns (fixed point)
  __shared__ int s_ey[2][TE][NP], s_ez[2][TE][NP];                    // their exponents
  __shared__ double s_t[2][TE][NP][2];                                // end-node fluxes of u
  __shared__ double s_red[PCG ? P2 : 1];
  const Tile2D tl = a.tiles[blockIdx.x];
  const Inst2D I = a.inst[tl.inst];
  chained_start();
  const BasisDev& B = a.B;
  const double hw = B.hw;
  double pal = 0.0, ppb = 0.0;  // PCG: alpha_it and the adjoint of pAp_it
  if (PCG) {
    pal = a.al_it[tl.inst];
    ppb = a.papb[tl.inst];
  }
  // u at node n, given x_k there (PCG forms it from rb and p_it)
  auto ldu = [&](long long n, double xkv) -> double {
    if (PCG) return fma(pal, a.u[n], -ppb * xkv);
    return a.u[n];
  };
  const int dir = threadIdx.x >= NH;  // 0: rows and x faces, 1: columns and y faces
  const ElemView w = elem_view<NP>(tl, I, dir, threadIdx.x - dir * NH);
  const int e = w.e, t = w.t;
  const int st = dir == 0 ? 1 : NP, at = dir == 0 ? t * NP : t;  // node k of the line: at + k st
  const double* ck = dir == 0 ? a.ckx : a.cky;
  // the ends of the line: u, x_k and the stiffness coefficient
  double u0 = 0.0, uL = 0.0, v0 = 0.0, vL = 0.0, k0 = 0.0, kL = 0.0;
  FixFlux<NP> f;
  FixDeriv<NP> d;
  if (w.valid) {
    double u[NP], v[NP], k[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const long long n = w.base + at + i * st;
      v[i] = a.xk[n]; u[i] = ldu(n, v[i]); k[i] = ck[n];
    }
    if (dir == 0) {
#pragma unroll
      for (int i = 0; i < NP; ++i) { s_u[e][at + i] = u[i]; s_v[e][at + i] = v[i]; }
    }
    flux_line<NP, true>(B, u, k, f);
    deriv_line<NP>(B, v, d);
    s_t[dir][e][t][0] = f.t0; s_t[dir][e][t][1] = f.tL;
    u0 = u[0]; uL = u[L]; v0 = v[0]; vL = v[L]; k0 = k[0]; kL = k[L];
  }
  __syncthreads();
  if (w.valid) {
    const double* cp = dir == 0 ? a.cpx : a.cpy;
    auto fetch = [&](int s) {
      Partner2 P;
      int it;
      const int dd = s == 0 ? -1 : 1;
      const long long pb = neighbour<NP>(tl, I, w.ex, w.ey, dir == 0 ? dd : 0, dir == 0 ? 0 : dd, &it);
      const int pn = at + (s == 0 ? L : 0) * st;  // partner face node
      P.ir = a.invr[pb + pn];
      if (it >= 0) {
        P.u = s_u[it][pn]; P.v = s_v[it][pn];
        P.t = s_t[dir][it][t][1 - s];
      } else {
        double p[NP];
        P.v = a.xk[pb + pn];
#pragma unroll
        for (int k = 0; k < NP; ++k) p[k] = ldu(pb + at + k * st, PCG ? a.xk[pb + at + k * st] : 0.0);
        P.u = s == 0 ? p[L] : p[0];
        P.t = flux_end<NP>(B, s == 0, p, ck[pb + pn]);
      }
      return P;
    };
    // One face: own end values (uo, vo, stiffness k, flux t0, derivative of x_k gv, 1/rho io, penalty p), the partner P;
    // s = +1 when the own node is the left side, else -1 (jumps are left minus right). F: the flux terms (consistency +
    // penalty, as added to the left side), us: the symmetry term hw k [u], z: the coefficient adjoint's face terms
    // hw k ([u] gv + gu [x_k]) and, where the own 1/rho sets the penalty, p [u] [x_k].
    auto face = [&](int s, double uo, double vo, double k, double t0, double gv, double io, double p, const Partner2& P,
                    double& F, double& us, double& z) {
      const double ju = s > 0 ? uo - P.u : P.u - uo, jv = s > 0 ? vo - P.v : P.v - vo;
      const double pj = p * ju;
      F = fma(hw, s > 0 ? t0 + P.t : P.t + t0, pj);
      us = hw * k * ju;
      const bool wins = s > 0 ? !gt_nonneg(P.ir, io) : gt_nonneg(io, P.ir);  // the right side wins only when strictly larger
      z = fma(gv, us, jv * fma(hw, t0, wins ? pj : 0.0));
    };
    const int sf = dir == 0 ? first_side(w.ext, TX) : first_side(w.eyt, TY);
    const Partner2 pA = fetch(sf), pB = fetch(1 - sf);
    const Partner2 pl = sf == 0 ? pA : pB, pr = sf == 0 ? pB : pA;
    double Fl, Fr, us0, usL, z0, zL;
    const long long n0 = w.base + at, nL = w.base + at + L * st;
    face(-1, u0, v0, k0, f.t0, deriv_at<NP>(d, 0), a.invr[n0], cp[n0], pl, Fl, us0, z0);
    face(1, uL, vL, kL, f.tL, deriv_at<NP>(d, L), a.invr[nL], cp[nL], pr, Fr, usL, zL);
    FixSums<NP> sums;
    row_products<NP>(f, d, z0, zL, sums);
#pragma unroll
    for (int k = 0; k < NP; ++k) s_z[dir][e][at + k * st] = sums.G[k];
    s_ez[dir][e][t] = sums.e;
    row_sums<NP>(B, f, us0, usL, -Fl, Fr, sums);
#pragma unroll
    for (int k = 0; k < NP; ++k) s_y[dir][e][at + k * st] = sums.G[k];
    s_ey[dir][e][t] = sums.e;
  }
  // ---- pointwise: sums, coefficient adjoints, solver epilogue. Everything is loaded before anything is stored (the
  // compiler has to assume that a store changes what a later load reads), and before the barrier.
  constexpr bool EPI = SREV == SREV_CHEB || SREV == SREV_JACOBI;
  constexpr int NQ = (TE * NN + 2 * NH - 1) / (2 * NH);
  long long node[NQ];
  double acc[NQ], zs[NQ], zm[NQ], bb[NQ], cM[NQ], db[NQ], im[NQ], rp[NQ], iMb[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const int m = threadIdx.x + q * 2 * NH;
    const int el = m / NN, nd = m % NN, ex = tl.ex0 + el % TX, ey = tl.ey0 + el / TX;
    const bool live = m < TE * NN && ex < I.nex && ey < I.ney;
    const long long n = I.off + (long long)NN * (ex + (long long)I.nex * ey) + nd;
    node[q] = live ? n : -1;
    if (!live) continue;
    // xb - cm u (and, for PCG, + alpha_it xconst + pApb apk)
    acc[q] = a.xb[n];
    cM[q] = a.cm[n];
    if (PCG) acc[q] = fma(ppb, a.apk[n], fma(pal, a.xconst[n], acc[q]));
    zs[q] = a.first ? 0.0 : a.Zs[n];
    zm[q] = a.first ? 0.0 : a.Zm[n];
    bb[q] = a.bb_op == 2 ? a.bb[n] : 0.0;
    if (PCG && a.has_next) rp[q] = a.p_next[n];
    if (EPI && a.has_next) {
      im[q] = a.cinvM[n];
      rp[q] = a.r_prev[n];
      iMb[q] = a.iMb[n];
      db[q] = SREV == SREV_CHEB ? a.db[n] : 0.0;
    }
  }
  __syncthreads();
  const int zsg = a.zscale > 0 ? 1 : -1;  // -1 (r = b - A x) or +1 (A p): applied through operand signs, not a multiply
  double part = 0.0;                      // PCG: betab partial of this thread
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const long long n = node[q];
    if (n < 0) continue;
    const int m = threadIdx.x + q * 2 * NH;
    const int el = m / NN, nd = m % NN, j = nd / NP, i = nd % NP;
    const double u = s_u[el][nd], v = s_v[el][nd], uz = zsg > 0 ? u : -u;
    const double xb = node_total<59>(s_y[0][el][nd], s_ey[0][el][j], s_y[1][el][nd], s_ey[1][el][i],
                                     fma(-cM[q], u, acc[q]), -1);
    a.xb[n] = xb;
    a.Zs[n] = node_total<60>(s_z[0][el][nd], s_ez[0][el][j], s_z[1][el][nd], s_ez[1][el][i], zs[q], zsg);
    a.Zm[n] = a.first ? uz * v : fma(uz, v, zm[q]);
    if (a.bb_op == 1) a.bb[n] = u;
    else if (a.bb_op == 2) a.bb[n] = bb[q] + u;
    if (PCG && a.has_next) part = fma(xb, rp[q], part);
    if (SREV == SREV_CHEB && a.has_next) {
      const double dbv = db[q] + xb;
      const double zb = a.cc * dbv;
      a.u_out[n] = im[q] * zb;
      a.iMb[n] = fma(zb, rp[q], iMb[q]);
      a.db[n] = a.ca * dbv;
    } else if (SREV == SREV_JACOBI && a.has_next) {
      const double tb = a.omega * xb;
      a.u_out[n] = tb * im[q];
      a.iMb[n] = fma(tb, rp[q], iMb[q]);
    }
  }
  if (PCG && a.has_next) {
    const double tot = block_sum<P2>(part, s_red);
    inst_sum_last_block(a.isum, tl.inst, I.ntiles, tot, a.partials, blockIdx.x, I.tile0, I.ntiles);
  }
}

// ---------------------------------------------------------------------------
// Reverse of the stage setup: IGR source b and diag(A), plus the conversion of
// the coefficient adjoints (Zm, Zs) into d/d rho and d/d alpha.
//   Qs[mx], Qs[my], Qs[rho] += ...      anode += dJ/dalpha contributions
// ---------------------------------------------------------------------------
struct SetupRevArgs2D {
  const Tile2D* tiles; const Inst2D* inst; BasisDev B;
  const double *mx, *my, *invr;       // taped stage input
  const double *b, *cm, *cM, *cinvM;  // taped source, mass coefficient, diag(A), 1/diag(A)
  const double *bb, *iMb, *Zm, *Zs;   // iMb: adjoint of 1/diag(A)
  double *Qs[3];                      // adjoints of (mx, my, rho) of the stage input
  double *anode;
};

// What bounds it: FP64 issue. All derivatives, transposes and diagonal contractions are integer line operations; the two
// transposes of a node meet as integers. Rows and columns run side by side, between pointwise passes whose loads
// come before any store. 8 x 128^2 P3: 409 us with FP64 contractions, 196 us with integer ones, 167 us in halves, 177 us with sums
// without a mean error and the leading-node checks; 64^2: 22.8, 22.7, 14.9.
template <int NP>
__global__ void __launch_bounds__(2 * Tiling2D<NP>::NH) k2_setup_rev(SetupRevArgs2D a) {
  using TL = Tiling2D<NP>;
  constexpr int TE = TL::TE, NN = TL::NN, SN = TL::SN, L = TL::L, TX = TL::TX, TY = TL::TY, NH = TL::NH;
  constexpr int NQ = (TE * NN + 2 * NH - 1) / (2 * NH);  // nodes per thread
  __shared__ __align__(16) double s_ux[TE][SN], s_uy[TE][SN], s_ir[TE][SN], s_Mb[TE][SN];
  // per direction: derivatives of the velocities, then the adjoints of these, then (integers) their transposes
  __shared__ __align__(16) long long s_dx[2][TE][SN], s_dy[2][TE][SN];
  __shared__ int s_ex[2][TE][NP], s_ey[2][TE][NP];
  __shared__ __align__(16) double s_ib[2][TE][SN];  // d/d(1/rho) from the line's share of diag(A)
  __shared__ double s_m0[NN];                       // w_i w_j Jx Jy
  // per face node of a side: alpha eta w J / d (penalty) and the self terms' -+alpha D_ee w J / J' (x: left, right; y: bottom, top)
  __shared__ double s_p[2][NP], s_s[2][2][NP];
  const Tile2D tl = a.tiles[blockIdx.x];
  const Inst2D I = a.inst[tl.inst];
  chained_start();
  const BasisDev& B = a.B;
  const double invJx = I.ijx, invJy = I.ijy;
  const double alpha = I.alpha;
  if (alpha <= 0.0) return;
  // the thread's nodes: node(m) or -1; m = el NN + nd
  auto node = [&](int m) -> long long {
    const int el = m / NN, nd = m % NN, ex = tl.ex0 + el % TX, ey = tl.ey0 + el / TX;
    return m < TE * NN && ex < I.nex && ey < I.ney ? I.off + (long long)NN * (ex + (long long)I.nex * ey) + nd : -1;
  };
  auto mbar = [&](double iMb, double im) { return -(iMb * im) * im; };  // d/dM = -d/d(1/M) / M^2
  // ---- pointwise: velocities, 1/rho, adjoint of diag(A)
  double bb[NQ];
  {
    double ir[NQ], mx[NQ], my[NQ], im[NQ], imb[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const long long n = node(threadIdx.x + q * 2 * NH);
      if (n < 0) continue;
      ir[q] = a.invr[n]; mx[q] = a.mx[n]; my[q] = a.my[n]; im[q] = a.cinvM[n]; imb[q] = a.iMb[n];
      bb[q] = a.bb[n];
    }
    for (int n = threadIdx.x; n < NN; n += blockDim.x) s_m0[n] = B.w[n % NP] * B.w[n / NP] * I.jx * I.jy;
    if (threadIdx.x < 2 * NP) {
      const int d = threadIdx.x / NP, k = threadIdx.x % NP;
      const double wf = B.w[k] * (d == 0 ? I.jy : I.jx), aJ = alpha * (d == 0 ? invJx : invJy);
      s_p[d][k] = alpha * (double)(NP * NP) * (d == 0 ? I.idx : I.idy) * wf;
      s_s[d][0][k] = aJ * B.D[0][0] * wf;
      s_s[d][1][k] = -aJ * B.D[L][L] * wf;
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int m = threadIdx.x + q * 2 * NH;
      if (node(m) < 0) continue;
      const int el = m / NN, nd = m % NN;
      s_ir[el][nd] = ir[q];
      s_ux[el][nd] = mx[q] * ir[q]; s_uy[el][nd] = my[q] * ir[q];
      s_Mb[el][nd] = mbar(imb[q], im[q]);
    }
  }
  __syncthreads();
  // ---- lines: derivatives, diag(A)'s stiffness and faces
  const int dir = threadIdx.x >= NH;  // 0: rows and x faces, 1: columns and y faces
  const ElemView w = elem_view<NP>(tl, I, dir, threadIdx.x - dir * NH);
  const int e = w.e, t = w.t;
  const int st = dir == 0 ? 1 : NP, at = dir == 0 ? t * NP : t;  // node k of the line: at + k st
  const FixScale c = fix_scale(dir == 0 ? invJx : invJy);
  if (w.valid) {
    struct Partner { double ir, Mb; };
    auto partner = [&](int s) {
      Partner P;
      int it;
      const int d = s == 0 ? -1 : 1, pn = at + (s == 0 ? L : 0) * st;
      const long long pb = neighbour<NP>(tl, I, w.ex, w.ey, dir == 0 ? d : 0, dir == 0 ? 0 : d, &it);
      if (it >= 0) { P.ir = s_ir[it][pn]; P.Mb = s_Mb[it][pn]; }
      else { P.ir = a.invr[pb + pn]; P.Mb = mbar(a.iMb[pb + pn], a.cinvM[pb + pn]); }
      return P;
    };
    const int sf = dir == 0 ? first_side(w.ext, TX) : first_side(w.eyt, TY);
    const Partner pA = partner(sf), pB = partner(1 - sf);
    double v[NP], out[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) v[k] = s_ux[e][at + k * st];
    line_rows<NP>(B, c, v, out);
#pragma unroll
    for (int k = 0; k < NP; ++k) { s_dx[dir][e][at + k * st] = __double_as_longlong(out[k]); v[k] = s_uy[e][at + k * st]; }
    line_rows<NP>(B, c, v, out);
#pragma unroll
    for (int k = 0; k < NP; ++k) { s_dy[dir][e][at + k * st] = __double_as_longlong(out[k]); v[k] = s_Mb[e][at + k * st]; }
    const Partner p0 = sf == 0 ? pA : pB, pL = sf == 0 ? pB : pA;
    double acc[NP];
    acc[0] = v[0] * s_s[dir][0][t];
    if (gt_nonneg(s_ir[e][at], p0.ir)) acc[0] = fma(v[0] + p0.Mb, s_p[dir][t], acc[0]);
    acc[L] = v[L] * s_s[dir][1][t];
    if (!gt_nonneg(pL.ir, s_ir[e][at + L * st])) acc[L] = fma(v[L] + pL.Mb, s_p[dir][t], acc[L]);
    // stiffness self-coupling of diag(A): d/d(1/rho_i) = c sum_k W2[i][k] Mb_k
    const FixScale cd = fix_scale(alpha * B.w[t] * (dir == 0 ? I.jy * invJx : I.jx * invJy));
    line_op<NP, false, false, true>(B.fW2, B.W2, &cd, v, acc, [](int k) { return k == 0 || k == L; }, out);
#pragma unroll
    for (int k = 0; k < NP; ++k) s_ib[dir][e][at + k * st] = out[k];
  }
  __syncthreads();
  // ---- pointwise, in place: adjoints of the derivatives
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const int m = threadIdx.x + q * 2 * NH;
    if (node(m) < 0) continue;
    const int el = m / NN, nd = m % NN;
    const double uxx = __longlong_as_double(s_dx[0][el][nd]), uyx = __longlong_as_double(s_dy[0][el][nd]);
    const double uxy = __longlong_as_double(s_dx[1][el][nd]), uyy = __longlong_as_double(s_dy[1][el][nd]);
    const double s = uxx + uyy;
    const double Qb2 = bb[q] * (2.0 * alpha * s_m0[nd]);
    s_dx[0][el][nd] = __double_as_longlong(Qb2 * (s + uxx));
    s_dy[0][el][nd] = __double_as_longlong(Qb2 * uxy);
    s_dx[1][el][nd] = __double_as_longlong(Qb2 * uyx);
    s_dy[1][el][nd] = __double_as_longlong(Qb2 * (s + uyy));
  }
  __syncthreads();
  // ---- lines, in place: transposes
  if (w.valid) {
    double v[NP];
    FixSums<NP> r;
#pragma unroll
    for (int k = 0; k < NP; ++k) v[k] = __longlong_as_double(s_dx[dir][e][at + k * st]);
    row_scaled<NP, true>(B, c, v, r);
#pragma unroll
    for (int k = 0; k < NP; ++k) { s_dx[dir][e][at + k * st] = r.G[k]; v[k] = __longlong_as_double(s_dy[dir][e][at + k * st]); }
    s_ex[dir][e][t] = r.e;
    row_scaled<NP, true>(B, c, v, r);
#pragma unroll
    for (int k = 0; k < NP; ++k) s_dy[dir][e][at + k * st] = r.G[k];
    s_ey[dir][e][t] = r.e;
  }
  // ---- pointwise: transposes of both directions, conversion to d/d rho and d/d alpha
  double b[NQ], cm[NQ], cM[NQ], Zm[NQ], Zs[NQ], Q[NQ][3], an[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const long long n = node(threadIdx.x + q * 2 * NH);
    if (n < 0) continue;
    b[q] = a.b[n]; cm[q] = a.cm[n]; cM[q] = a.cM[n]; Zm[q] = a.Zm[n]; Zs[q] = a.Zs[n]; an[q] = a.anode[n];
#pragma unroll
    for (int v = 0; v < 3; ++v) Q[q][v] = a.Qs[v][n];
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const int m = threadIdx.x + q * 2 * NH;
    const long long n = node(m);
    if (n < 0) continue;
    const int el = m / NN, nd = m % NN, i = nd % NP, j = nd / NP;
    const double uxb = node_total<60>(s_dx[0][el][nd], s_ex[0][el][j], s_dx[1][el][nd], s_ex[1][el][i], 0.0, 1);
    const double uyb = node_total<60>(s_dy[0][el][nd], s_ey[0][el][j], s_dy[1][el][nd], s_ey[1][el][i], 0.0, 1);
    const double ir = s_ir[el][nd], Mb = s_Mb[el][nd];
    const double ib = fma(Mb, s_m0[nd], s_ib[0][el][nd] + s_ib[1][el][nd]);
    const double zms = fma(cm[q], Zm[q], Zs[q]);  // Zm + Zs, with Zm's mass coefficient
    const double r = fma(uxb, s_ux[el][nd], fma(uyb, s_uy[el][nd], fma(ib, ir, zms)));
    a.Qs[0][n] = fma(uxb, ir, Q[q][0]);
    a.Qs[1][n] = fma(uyb, ir, Q[q][1]);
    a.Qs[2][n] = fma(-ir, r, Q[q][2]);
    // d/dalpha: Zs/alpha + Mb (M - mass)/alpha + bb b/alpha
    a.anode[n] = fma(fma(Mb, cM[q] - cm[q], fma(bb[q], b[q], Zs[q])), I.ialpha, an[q]);
  }
}

}  // namespace igrgpu
