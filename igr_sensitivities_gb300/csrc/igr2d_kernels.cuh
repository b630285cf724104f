// 2D IGR-Euler forward kernels (sm_103a, FP64 CUDA cores).
//
// Thread mapping: a CTA owns a TX x TY tile of elements of one instance. The
// line work (1D contractions with the LGL differentiation matrix and the faces
// across the line's ends) takes one thread per element *line*; in most kernels
// rows and columns run side by side, one half of 2 NH threads each, between
// pointwise passes over all threads (coalesced, loads before stores). The
// remaining ones (tangent right-hand side, adjoint PDE) run a row phase and then
// a column phase on NT threads.
//
// GB300 issues about 1.2 TFLOP/s of FP64 against 6.6 TB/s of HBM (about
// 5.6 B per FP64 flop), so these kernels are bound by FP64 issue and trade
// memory and integer instructions for FP64 ones: the line contractions are
// integer sums (igr_fix.cuh), per-stage operator coefficients are computed
// once and re-read by every solver iteration, reciprocals of mesh constants
// come precomputed from the host, the SIP face terms are folded into the
// stiffness transpose, and out-of-tile (halo) work is packed into one warp
// per direction (see elem_view) so that it is paid once per tile, converged.
#pragma once
#include "igr_device.cuh"

namespace igrgpu {

template <int NP>
struct Tiling2D {
  static constexpr int TX = NP <= 4 ? 4 : 2;  // element tile (keeps static smem < 48 KB)
  static constexpr int TY = 4;
  static constexpr int TE = TX * TY;       // elements per tile
  static constexpr int NN = NP * NP;       // nodes per element
  // Stride of an element in shared memory. A phase reads 8-byte nodes down its lines: with the 16 nodes of a P3
  // element packed, a warp's 8 elements hit the same banks (8 wavefronts for 2); 18 spreads them over all banks and
  // keeps the rows 16-byte aligned (128-bit accesses, also without conflicts). 5 does it for P1; 9 and 25 are odd.
  static constexpr int SN = NP == 4 ? 18 : (NP == 2 ? 5 : NN);
  static constexpr int NT = TE * NP;       // threads per CTA (one per line)
  static constexpr int NH = (NT + 31) / 32 * 32;  // threads of each half where rows and columns run side by side
  static constexpr int L = NP - 1;
};

// A thread's element and line in one phase.
struct ElemView {
  int e, t, ext, eyt, ex, ey;
  bool valid;
  long long base;  // first node of the element
};

// Thread -> (element of the tile, line) for phase 0 (xi-phase, x faces) or
// phase 1 (eta-phase, y faces). For P3 (64 threads = 2 warps of 8 elements x
// 4 lines) warp 0 takes the 8 elements on the two tile edges normal to the
// phase's faces and warp 1 the 8 interior ones, so the out-of-tile partner
// work of a phase runs in one warp, with every lane on the same path.
template <int NP>
__device__ __forceinline__ ElemView elem_view(const Tile2D& tl, const Inst2D& I, int phase, int tid) {
  constexpr int TX = Tiling2D<NP>::TX, TY = Tiling2D<NP>::TY;
  ElemView v;
  if (NP == 4 && TX == 4 && TY == 4) {
    const int w = tid >> 5, k = (tid >> 2) & 7;
    v.t = tid & 3;
    const int across = (w == 0) ? ((k & 4) ? 3 : 0) : ((k & 4) ? 2 : 1);
    const int along = k & 3;
    v.ext = phase == 0 ? across : along;
    v.eyt = phase == 0 ? along : across;
  } else {
    const int e = tid / NP;
    v.t = tid % NP;
    v.ext = e % TX;
    v.eyt = e / TX;
  }
  v.e = v.ext + TX * v.eyt;
  v.ex = tl.ex0 + v.ext;
  v.ey = tl.ey0 + v.eyt;
  v.valid = tid < Tiling2D<NP>::NT && v.ex < I.nex && v.ey < I.ney;
  v.base = I.off + (long long)NP * NP * ((long long)v.ex + (long long)I.nex * v.ey);
  return v;
}

template <int NP>
__device__ __forceinline__ ElemView elem_view(const Tile2D& tl, const Inst2D& I, int phase) {
  return elem_view<NP>(tl, I, phase, threadIdx.x);
}

// Neighbour element (dx, dy in {-1,0,1}) with periodic wrap; returns its base
// node and its index inside the tile (or -1 when it is not in this tile).
template <int NP>
__device__ __forceinline__ long long neighbour(const Tile2D& tl, const Inst2D& I, int ex, int ey, int ddx, int ddy,
                                               int* in_tile) {
  constexpr int TX = Tiling2D<NP>::TX, TY = Tiling2D<NP>::TY;
  int nx = ex + ddx, ny = ey + ddy;
  nx = nx < 0 ? I.nex - 1 : (nx >= I.nex ? 0 : nx);
  ny = ny < 0 ? I.ney - 1 : (ny >= I.ney ? 0 : ny);
  const int lx = nx - tl.ex0, ly = ny - tl.ey0;
  *in_tile = (lx >= 0 && lx < TX && ly >= 0 && ly < TY) ? (lx + TX * ly) : -1;
  return I.off + (long long)NP * NP * ((long long)nx + (long long)I.nex * ny);
}

// The diagonal of the LGL differentiation matrix vanishes at interior nodes
// (exactly 0.0 in double for P3 as built by basis.jl:38-49; |D_ii| < 1e-15 for
// P4), so those products are skipped. Callers unroll the loops, making i and k
// compile-time constants and the skip free of branches.
__device__ __forceinline__ constexpr bool d_zero(int np, int i, int k) { return i == k && i > 0 && i < np - 1; }

// sum_k D[i][k] v[k] (reference derivative of a line at node i)
template <int NP>
__device__ __forceinline__ double dot_row(const BasisDev& B, int i, const double* v) {
  double s = 0.0;
  bool first = true;
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    if (d_zero(NP, i, k)) continue;
    s = first ? B.D[i][k] * v[k] : fma(B.D[i][k], v[k], s);
    first = false;
  }
  return s;
}

// Derivative at the first (last == false) or last end node of a line, with
// the row chosen at run time by register selects (no divergence, no local
// memory): the form the halo loads need.
template <int NP>
__device__ __forceinline__ double dot_end(const BasisDev& B, bool last, const double* v) {
  double s = (last ? B.D[NP - 1][0] : B.D[0][0]) * v[0];
#pragma unroll
  for (int k = 1; k < NP; ++k) s = fma(last ? B.D[NP - 1][k] : B.D[0][k], v[k], s);
  return s;
}

// acc + sum_i D[i][k] v[i] (transpose contraction, node k)
template <int NP>
__device__ __forceinline__ double dot_col(const BasisDev& B, int k, const double* v, double acc) {
#pragma unroll
  for (int i = 0; i < NP; ++i) {
    if (d_zero(NP, i, k)) continue;
    acc = fma(B.D[i][k], v[i], acc);
  }
  return acc;
}

// Which face of a phase to process first: the out-of-tile one for edge
// elements, so the halo loads of warp 0 run converged.
__device__ __forceinline__ int first_side(int pos_across, int extent) { return pos_across == extent - 1 ? 1 : 0; }

// ---------------------------------------------------------------------------
// Stage setup: IGR source b (elliptic.jl:159-197), diag(A) (elliptic.jl:205-264)
// and the per-node operator coefficients reused by every solver iteration:
//   cm  = w_i w_j Jx Jy / rho                     (mass)
//   ckx = alpha w_i w_j (Jy/Jx) / rho             (x stiffness)
//   cky = alpha w_i w_j (Jx/Jy) / rho             (y stiffness)
//   cpx = alpha (w_j Jy) eta max(1/rho_L,1/rho_R)/dx   at x-face nodes (penalty)
//   cpy = alpha (w_i Jx) eta max(1/rho_L,1/rho_R)/dy   at y-face nodes
//   cinvM = 1 / diag(A)
// ---------------------------------------------------------------------------
struct SetupArgs2D {
  const Tile2D* tiles; const Inst2D* inst; BasisDev B;
  const double *mx, *my, *invr;
  double *b;  // IGR source (null: not formed; mx, my are then not read)
  double *cm, *ckx, *cky, *cinvM, *cpx, *cpy;
  double *cM;  // diag(A) itself (optional; the reverse needs it for d/d alpha)
  int always;  // compute the coefficients even when alpha <= 0 (operator application on its own)
};

// What bounds it: FP64 issue, at a third of the FP64 instructions of its FP64-contraction form: the velocity derivatives
// and both diagonal contractions (with their scales and the face terms) are integer line operations, and the face
// constants are tabulated once per CTA. Rows and columns run side by side like the operator's, between two pointwise
// passes. 8 x 128^2 P3: 259 us with FP64 contractions, 113 us with integer ones, 103 us in halves, 110 us with IEEE 1/x again
// (restarts to the bit) and sums without a mean error. 64^2: 16.5, 13.9, 12.4.
template <int NP>
__global__ void __launch_bounds__(2 * Tiling2D<NP>::NH) k2_setup(SetupArgs2D a) {
  using TL = Tiling2D<NP>;
  constexpr int TE = TL::TE, NN = TL::NN, SN = TL::SN, L = TL::L, TX = TL::TX, TY = TL::TY, NH = TL::NH;
  constexpr int NQ = (TE * NN + 2 * NH - 1) / (2 * NH);  // nodes per thread
  __shared__ __align__(16) double s_ir[TE][SN], s_ux[TE][SN], s_uy[TE][SN];
  // per direction: derivatives of the velocities (columns: twice that of u_x), the line's share of diag(A), face penalties
  __shared__ __align__(16) double s_dx[2][TE][SN], s_dy[2][TE][SN], s_m[2][TE][SN];
  __shared__ double s_f[2][TE][NP][2];
  // per node: w_i w_j Jx Jy, alpha w_i w_j Jy/Jx, alpha w_i w_j Jx/Jy, alpha times the first  [node j*NP+i]
  __shared__ double s_c[4][NN];
  // per face node of a side: alpha eta w J / d (penalty) and the self terms' -+alpha D_ee w J / J' (x: left, right; y: bottom, top)
  __shared__ double s_p[2][NP], s_s[2][2][NP];
  const Tile2D tl = a.tiles[blockIdx.x];
  const Inst2D I = a.inst[tl.inst];
  chained_start();
  const BasisDev& B = a.B;
  const double invJx = I.ijx, invJy = I.ijy;
  if (I.alpha <= 0.0 && !a.always) return;  // no elliptic solve for this instance (forward.jl:24-28)
  // the thread's nodes: node(m) or -1; m = el NN + nd
  auto node = [&](int m) -> long long {
    const int el = m / NN, nd = m % NN, ex = tl.ex0 + el % TX, ey = tl.ey0 + el / TX;
    return m < TE * NN && ex < I.nex && ey < I.ney ? I.off + (long long)NN * (ex + (long long)I.nex * ey) + nd : -1;
  };
  // ---- pointwise: velocities and 1/rho
  {
    double ir[NQ], ux[NQ], uy[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const long long n = node(threadIdx.x + q * 2 * NH);
      if (n < 0) continue;
      ir[q] = a.invr[n];
      if (a.b) { ux[q] = a.mx[n]; uy[q] = a.my[n]; }
    }
    for (int n = threadIdx.x; n < NN; n += blockDim.x) {
      const int i = n % NP, j = n / NP;
      const double ww = B.w[i] * B.w[j];
      s_c[0][n] = ww * I.jx * I.jy;
      s_c[1][n] = I.alpha * ww * I.jy * invJx;
      s_c[2][n] = I.alpha * ww * I.jx * invJy;
      s_c[3][n] = s_c[0][n] * I.alpha;
    }
    if (threadIdx.x < 2 * NP) {
      const int d = threadIdx.x / NP, k = threadIdx.x % NP;
      const double wf = B.w[k] * (d == 0 ? I.jy : I.jx), aJ = I.alpha * (d == 0 ? invJx : invJy);
      s_p[d][k] = I.alpha * (double)(NP * NP) * (d == 0 ? I.idx : I.idy) * wf;
      s_s[d][0][k] = aJ * B.D[0][0] * wf;
      s_s[d][1][k] = -aJ * B.D[L][L] * wf;
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int m = threadIdx.x + q * 2 * NH;
      if (node(m) < 0) continue;
      const int el = m / NN, nd = m % NN;
      s_ir[el][nd] = ir[q];
      if (a.b) { s_ux[el][nd] = ux[q] * ir[q]; s_uy[el][nd] = uy[q] * ir[q]; }
    }
  }
  __syncthreads();
  // ---- lines: derivatives, stiffness diagonal with the face terms
  const int dir = threadIdx.x >= NH;  // 0: rows and x faces, 1: columns and y faces
  const ElemView w = elem_view<NP>(tl, I, dir, threadIdx.x - dir * NH);
  if (w.valid) {
    const int e = w.e, t = w.t;
    const int st = dir == 0 ? 1 : NP, at = dir == 0 ? t * NP : t;  // node k of the line: at + k st
    auto partner = [&](int s) {  // 1/rho across the line's face s
      int it;
      const int d = s == 0 ? -1 : 1, pn = at + (s == 0 ? L : 0) * st;
      const long long pb = neighbour<NP>(tl, I, w.ex, w.ey, dir == 0 ? d : 0, dir == 0 ? 0 : d, &it);
      return it >= 0 ? s_ir[it][pn] : a.invr[pb + pn];
    };
    const int sf = dir == 0 ? first_side(w.ext, TX) : first_side(w.eyt, TY);
    const double pA = partner(sf), pB = partner(1 - sf);
    double v[NP], out[NP];
    if (a.b) {
      const FixScale c1 = fix_scale(dir == 0 ? invJx : invJy);
#pragma unroll
      for (int k = 0; k < NP; ++k) v[k] = s_ux[e][at + k * st];
      line_rows<NP>(B, fix_scale(dir == 0 ? invJx : 2.0 * invJy), v, out);
#pragma unroll
      for (int k = 0; k < NP; ++k) { s_dx[dir][e][at + k * st] = out[k]; v[k] = s_uy[e][at + k * st]; }
      line_rows<NP>(B, c1, v, out);
#pragma unroll
      for (int k = 0; k < NP; ++k) s_dy[dir][e][at + k * st] = out[k];
    }
    double acc[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) v[k] = s_ir[e][at + k * st];
    // right side of the face at node 0, left side of the one at node L
    const double f0 = s_p[dir][t] * max_nonneg(sf == 0 ? pA : pB, v[0]), fL = s_p[dir][t] * max_nonneg(v[L], sf == 0 ? pB : pA);
    s_f[dir][e][t][0] = f0; s_f[dir][e][t][1] = fL;
    acc[0] = fma(s_s[dir][0][t], v[0], f0);
    acc[L] = fma(s_s[dir][1][t], v[L], fL);
    const FixScale cd = fix_scale(I.alpha * B.w[t] * (dir == 0 ? I.jy * invJx : I.jx * invJy));
    line_op<NP, true, false, true>(B.fW2, B.W2, &cd, v, acc, [](int k) { return k == 0 || k == L; }, out);
#pragma unroll
    for (int k = 0; k < NP; ++k) s_m[dir][e][at + k * st] = out[k];
  }
  __syncthreads();
  // ---- pointwise: source, diagonal, coefficients
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const int m = threadIdx.x + q * 2 * NH;
    const long long n = node(m);
    if (n < 0) continue;
    const int el = m / NN, nd = m % NN, i = nd % NP, j = nd / NP;
    if (a.b) {
      const double uxx = s_dx[0][el][nd], uyx = s_dy[0][el][nd], uxy2 = s_dx[1][el][nd], uyy = s_dy[1][el][nd];
      const double s = uxx + uyy;
      double R = fma(s, s, uxx * uxx);
      R = fma(uxy2, uyx, R);
      R = fma(uyy, uyy, R);
      a.b[n] = s_c[3][nd] * R;
    }
    const double ir = s_ir[el][nd], mass = s_c[0][nd] * ir;
    const double M = mass + (s_m[0][el][nd] + s_m[1][el][nd]);
    a.cm[n] = mass;
    a.ckx[n] = s_c[1][nd] * ir;
    a.cky[n] = s_c[2][nd] * ir;
    a.cpx[n] = i == 0 || i == L ? s_f[0][el][j][i == L] : 0.0;
    a.cpy[n] = j == 0 || j == L ? s_f[1][el][i][j == L] : 0.0;
    a.cinvM[n] = 1.0 / M;
    if (a.cM) a.cM[n] = M;
  }
}

// ---------------------------------------------------------------------------
// SIP operator application y = A x (elliptic.jl:30-145) with a solver
// epilogue. The face terms of a face-node pair (L, R) are
//   F = hw*(kx_L d_L + kx_R d_R) + p (x_L - x_R),  hw = -1/(2 w_0)
//   y_L += F, y_R -= F                    (consistency + penalty)
//   sx_L += hw kx_L jump, sx_R += hw kx_R jump   (symmetry term, folded into
//                                                  the stiffness transpose)
// where d is the reference derivative of x at the face node on each side.
// Each side computes F itself (owner computes), so no atomics are needed.
// ---------------------------------------------------------------------------
enum { EPI_CHEB = 0, EPI_JACOBI = 1, EPI_RESID = 2, EPI_PCG0 = 3, EPI_PCG = 4 };

struct ApplyArgs2D {
  const Tile2D* tiles; const Inst2D* inst; BasisDev B;
  const double* x;                       // x_k (read with halo)
  const double *cm, *ckx, *cky, *cpx, *cpy, *b, *cinvM;
  const double* d_in;                    // Chebyshev d_k (null on the first iteration)
  double *d_out, *x_out;                 // d_{k+1}, x_{k+1}
  double *tape_x, *tape_r;               // optional tape of x_k and r_k = b - A x_k
  double *y_out;                         // EPI_RESID: raw y = A x
  double ca, cc, omega;                  // d_{k+1} = ca d_k + cc M^-1 r_k ; Jacobi omega
  // Jacobi-preconditioned CG (pcg_fixed!, elliptic.jl:329-347):
  //  EPI_PCG0: x = x_0; r_0 = b - A x_0 -> r_out, p_0 = M^-1 r_0 -> p_out, partial of r_0 . p_0
  //  EPI_PCG : x = p_k; with pcg_p set, p_k = M^-1 r_k + beta p_{k-1} is formed on load from
  //            (pcg_r, pcg_p), beta = pcg_beta[inst] = rz_k / (rz_{k-1} + 1e-30), and stored to p_out;
  //            A p_k -> ap_out, partial of p_k . A p_k
  // The inner-product partial of each tile goes to partials[tile]; the instance's last block adds
  // them (isum: rz_0 for EPI_PCG0; pAp_k and alpha_k for EPI_PCG).
  const double *pcg_r, *pcg_p, *pcg_beta;
  double *p_out, *r_out, *ap_out;
  double* partials;
  InstSum isum;
};

// Partner data across one face: its value and its flux k (D x) at the face node.
struct Partner1 { double x, t; };

// Shared memory of one tile's operator application: x, the sums of the rows and
// of the columns (fixed point, with each line's exponent) and the end-node
// fluxes of every line.
template <int NP>
struct ApplySmem {
  alignas(16) double x[Tiling2D<NP>::TE][Tiling2D<NP>::SN];
  alignas(16) long long y[2][Tiling2D<NP>::TE][Tiling2D<NP>::SN];
  int e[2][Tiling2D<NP>::TE][NP];
  double t[2][Tiling2D<NP>::TE][NP][2];
};

// y = A x on tile tl (of instance I) with the EPI epilogue, by the CTA's
// 2 NH threads (all of which call it; it synchronises the CTA). Returns this
// thread's PCG inner-product partial (EPI_PCG0 / EPI_PCG; 0 otherwise).
// k2_apply runs it on tile blockIdx.x; the persistent PCG kernel on the CTA's tile.
// Rows and columns run side by side, one half of the CTA each: the two directions are independent up to their sums, so a
// line's chain of loads, integer sums and FP64 faces is all that a warp runs before the CTA meets, and the epilogue is
// pointwise over all threads with coalesced accesses. PCG's direction update p_k = M^-1 r_k + beta p_{k-1} is pointwise
// too and is formed once per node, in front of the lines.
// What bounds it: the integer ALU (65% busy), FP64 issue (61%) and L2 latency, with 32 warps per SM. 8 x 128^2 P3,
// Chebyshev: 127 us with FP64 contractions; 79 us with integer ones and one thread per pair of lines (18 warps); 69 us in
// halves; 65 us with the pointwise loads ahead of its stores; 68 us with sums without a mean error. 64^2: 12.3, 11.3, 10.2, 9.9.
template <int NP, int EPI>
__device__ __forceinline__ double apply_tile(const ApplyArgs2D& a, const Tile2D tl, const Inst2D& I, ApplySmem<NP>& sm) {
  using TL = Tiling2D<NP>;
  constexpr int TE = TL::TE, NN = TL::NN, L = TL::L, TX = TL::TX, TY = TL::TY, NH = TL::NH;
  constexpr int NQ = (TE * NN + 2 * NH - 1) / (2 * NH);  // nodes per thread
  constexpr bool PCG = EPI == EPI_PCG0 || EPI == EPI_PCG;
  // b - cm x enters the last sum and the rest with a minus sign where the epilogue wants the residual
  constexpr bool RES = EPI == EPI_CHEB || EPI == EPI_JACOBI || EPI == EPI_PCG0;
  const BasisDev& B = a.B;
  const double hw = B.hw;
  const bool form_p = EPI == EPI_PCG && a.pcg_p != nullptr;
  const double beta = form_p ? a.pcg_beta[tl.inst] : 0.0;
  auto ldx = [&](long long n) -> double {
    if (form_p) return fma(beta, a.pcg_p[n], a.pcg_r[n] * a.cinvM[n]);
    return a.x[n];
  };
  // the thread's nodes: node(q) or -1; m = el NN + nd
  auto node = [&](int m) -> long long {
    const int el = m / NN, nd = m % NN, ex = tl.ex0 + el % TX, ey = tl.ey0 + el / TX;
    return m < TE * NN && ex < I.nex && ey < I.ney ? I.off + (long long)NN * (ex + (long long)I.nex * ey) + nd : -1;
  };
  const int dir = threadIdx.x >= NH;  // 0: rows and x faces, 1: columns and y faces
  const ElemView w = elem_view<NP>(tl, I, dir, threadIdx.x - dir * NH);
  const int e = w.e, t = w.t;
  const int st = dir == 0 ? 1 : NP, at = dir == 0 ? t * NP : t;  // node k of the line: at + k st
  const double* ck = dir == 0 ? a.ckx : a.cky;
  if (PCG) {
    double x[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const long long n = node(threadIdx.x + q * 2 * NH);
      if (n >= 0) x[q] = ldx(n);
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int m = threadIdx.x + q * 2 * NH;
      const long long n = node(m);
      if (n < 0) continue;
      sm.x[m / NN][m % NN] = x[q];
      if (form_p) a.p_out[n] = x[q];
      if (a.tape_x) a.tape_x[n] = x[q];
    }
    __syncthreads();
  }
  double x0 = 0.0, xL = 0.0, k0 = 0.0, kL = 0.0;
  FixFlux<NP> f;
  if (w.valid) {
    double x[NP], k[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      x[i] = PCG ? sm.x[e][at + i * st] : a.x[w.base + at + i * st];
      k[i] = ck[w.base + at + i * st];
    }
    if (!PCG && dir == 0) {
#pragma unroll
      for (int i = 0; i < NP; ++i) sm.x[e][at + i] = x[i];
    }
    flux_line<NP>(B, x, k, f);
    sm.t[dir][e][t][0] = f.t0; sm.t[dir][e][t][1] = f.tL;
    x0 = x[0]; xL = x[L]; k0 = k[0]; kL = k[L];
  }
  __syncthreads();
  if (w.valid) {
    const double* cp = dir == 0 ? a.cpx : a.cpy;
    auto fetch = [&](int s) {
      Partner1 P;
      int it;
      const int d = s == 0 ? -1 : 1;
      const long long pb = neighbour<NP>(tl, I, w.ex, w.ey, dir == 0 ? d : 0, dir == 0 ? 0 : d, &it);
      const int pn = at + (s == 0 ? L : 0) * st;  // partner face node
      if (it >= 0) {
        P.x = sm.x[it][pn];
        P.t = sm.t[dir][it][t][1 - s];
      } else {
        double p[NP];
#pragma unroll
        for (int k = 0; k < NP; ++k) p[k] = ldx(pb + at + k * st);
        P.x = s == 0 ? p[L] : p[0];
        P.t = flux_end<NP>(B, s == 0, p, ck[pb + pn]);
      }
      return P;
    };
    const int sf = dir == 0 ? first_side(w.ext, TX) : first_side(w.eyt, TY);
    const Partner1 pA = fetch(sf), pB = fetch(1 - sf);
    const Partner1 pl = sf == 0 ? pA : pB, pr = sf == 0 ? pB : pA;
    // left face: own node 0 is the R side; right face: own node L is the L side
    const double jl = pl.x - x0, jr = xL - pr.x;
    const double Fl = fma(cp[w.base + at], jl, hw * (pl.t + f.t0));
    const double Fr = fma(cp[w.base + at + L * st], jr, hw * (f.tL + pr.t));
    FixSums<NP> sums;
    row_sums<NP>(B, f, hw * k0 * jl, hw * kL * jr, -Fl, Fr, sums);
#pragma unroll
    for (int k = 0; k < NP; ++k) sm.y[dir][e][at + k * st] = sums.G[k];
    sm.e[dir][e][t] = sums.e;
  }
  // ---- pointwise: mass term, sums, epilogue. Everything is loaded before anything is stored (the compiler has to assume
  // that a store changes what a later load reads), and before the barrier.
  double cm[NQ], b[NQ], im[NQ], din[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const long long n = node(threadIdx.x + q * 2 * NH);
    if (n < 0) continue;
    cm[q] = a.cm[n];
    if (RES) {
      b[q] = a.b[n];
      im[q] = a.cinvM[n];
      din[q] = EPI == EPI_CHEB && a.d_in ? a.d_in[n] : 0.0;
    }
  }
  __syncthreads();
  double part = 0.0;  // PCG inner-product partial of this thread
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const int m = threadIdx.x + q * 2 * NH;
    const long long n = node(m);
    if (n < 0) continue;
    const int el = m / NN, nd = m % NN;
    const double x = sm.x[el][nd];
    const double acc = RES ? fma(-cm[q], x, b[q]) : cm[q] * x;
    const double y = node_total<59>(sm.y[0][el][nd], sm.e[0][el][nd / NP], sm.y[1][el][nd], sm.e[1][el][nd % NP], acc,
                                    RES ? -1 : 1);  // A x, or b - A x (RES)
    if (EPI == EPI_RESID) a.y_out[n] = y;
    if (EPI == EPI_PCG) {
      a.ap_out[n] = y;
      part = fma(x, y, part);
    }
    if (EPI == EPI_PCG0) {
      const double z0 = y * im[q];
      a.r_out[n] = y;
      a.p_out[n] = z0;
      part = fma(y, z0, part);
    }
    if (EPI == EPI_CHEB || EPI == EPI_JACOBI) {
      if (a.tape_x) a.tape_x[n] = x;
      if (a.tape_r) a.tape_r[n] = y;
    }
    if (EPI == EPI_CHEB) {
      const double z = y * im[q];
      const double d = a.d_in ? fma(a.ca, din[q], a.cc * z) : a.cc * z;
      a.d_out[n] = d;
      a.x_out[n] = x + d;
    }
    if (EPI == EPI_JACOBI) a.x_out[n] = fma(a.omega * y, im[q], x);  // x + omega (b - A x) / M   (elliptic.jl:358)
  }
  return part;
}

template <int NP, int EPI>
__global__ void __launch_bounds__(2 * Tiling2D<NP>::NH) k2_apply(ApplyArgs2D a) {
  constexpr bool PCG = EPI == EPI_PCG0 || EPI == EPI_PCG;
  constexpr int P2 = pow2_at_least(2 * Tiling2D<NP>::NH);
  __shared__ ApplySmem<NP> sm;
  __shared__ double s_red[PCG ? P2 : 1];
  const Tile2D tl = a.tiles[blockIdx.x];
  const Inst2D I = a.inst[tl.inst];
  chained_start();
  const double part = apply_tile<NP, EPI>(a, tl, I, sm);
  if (PCG) {
    const double tot = block_sum<P2>(part, s_red);
    inst_sum_last_block(a.isum, tl.inst, I.ntiles, tot, a.partials, blockIdx.x, I.tile0, I.ntiles);
  }
}

// ---------------------------------------------------------------------------
// Hyperbolic DG RHS (hyperbolic.jl:27-119) fused with the SSP-RK3 stage
// combination (forward.jl:53-68):  q_out = c0*q^n + c1*q_s + c2*dt*k(q_s, Sigma).
// Also writes 1/rho of q_out for the next stage's setup, optionally the LLF
// wave speeds at face nodes (the reverse reads them instead of recomputing
// square roots), and flags non-finite values or rho <= 0 in the status word.
// ---------------------------------------------------------------------------
struct HypArgs2D {
  const Tile2D* tiles; const Inst2D* inst; BasisDev B;
  const double *q[4], *invr, *S;   // stage input
  const double *qn[4];             // step-start state (stages 2 and 3)
  double c0, c1, c2;
  double *qo[4], *invro;           // stage output (may alias qn: pointwise)
  double *k_out[4];                // optional: raw RHS k (compute_hyperbolic_rhs!)
  double *ws_x, *ws_y;             // optional: |u_n| + c at x-face / y-face nodes
  int* status;
};

// Pointwise physics at one node (euler.jl:145-214): both directional fluxes
// with P_bar = P + Sigma from one evaluation of the pressure.
struct NodePhys {
  double ux, uy, P, pb;
  double fx[4], fy[4];
};
__device__ __forceinline__ NodePhys node_phys(double g, double mx, double my, double E, double S, double ir) {
  NodePhys p;
  p.ux = mx * ir; p.uy = my * ir;
  const double m2r = fma(mx, mx, my * my) * ir;
  p.P = (g - 1.0) * fma(-0.5, m2r, E);
  p.pb = p.P + S;
  const double epb = E + p.pb;
  p.fx[0] = fma(mx, p.ux, p.pb); p.fx[1] = my * p.ux; p.fx[2] = mx; p.fx[3] = epb * p.ux;
  p.fy[0] = p.fx[1]; p.fy[1] = fma(my, p.uy, p.pb); p.fy[2] = my; p.fy[3] = epb * p.uy;
  return p;
}
// |u_n| + c, c = sqrt(gamma P / rho)
__device__ __forceinline__ double wavespeed(double g, double un, double P, double ir) {
  return fabs(un) + sqrt(g * P * ir);
}

// x[v] of an array in registers
__device__ __forceinline__ double pick4(const double* x, int v) {
  const double lo = (v & 1) ? x[1] : x[0], hi = (v & 1) ? x[3] : x[2];
  return (v & 2) ? hi : lo;
}

// The LLF flux of one face less the own side's flux, doubled: f_partner - f_own + lambda (q_L - q_R)
// (euler.jl:222-236), the form the DG lifting takes it in. dq = q_partner - q_own; lam has the sign that
// makes lam dq = lambda (q_L - q_R).
__device__ __forceinline__ double llf_jump(double fp, double fo, double lam, double dq) { return fma(lam, dq, fp - fo); }

// Flux data of one node: the transported quantities q, the flux components that are not one of them (fx_2 and fy_2 are
// q_0 and q_1, fy_0 = fx_1), and what the y wave speed needs.
struct FluxNode { double q[4], fx0, f1, fx3, fy1, fy3, aux; };

template <int NP, bool AUX>
struct StageSmem {
  double q[4][Tiling2D<NP>::TE][Tiling2D<NP>::NN];
  double f[5][Tiling2D<NP>::TE][Tiling2D<NP>::NN];            // fx_0, fx_1 = fy_0, fx_3, fy_1, fy_3
  double aux[AUX ? Tiling2D<NP>::TE : 1][Tiling2D<NP>::NN];
  long long k[2][4][Tiling2D<NP>::TE][Tiling2D<NP>::NN];      // row and column parts of c2 dt k (fixed point)
  int ke[2][4][Tiling2D<NP>::TE][NP];                         // their exponents
  double w[2][Tiling2D<NP>::TE][NP][2];                       // wave speeds at the line ends
};

// DG volume and LLF face terms of one tile with the SSP-RK3 combination q_out = c0 q^n + c1 q_s + c2 dt k (raw: k itself)
// for the physics PH (the Euler fluxes or their tangent):
//   at(n)                 the node's FluxNode
//   speed(dir, n, q, aux, own)  wave speed at a face node, q the quantity that is the mass flux; own: of this tile
//   qn(v, n), put(v, n, value)
// Node work is spread over all 2 NH threads of the CTA; line work runs with rows and columns side by side, one half each.
// What bounds it: FP64 issue. Volume terms, their scaling, the row and column parts and the stage combination's sum are
// integer work (igr_fix.cuh); the stage coefficient is folded into the scale of the derivatives and face terms, so that
// q_out = c0 q^n + c1 q_s + [c2 dt k] is one rounded sum and k itself is never formed. Euler, 8 x 128^2 P3: 427 us with
// FP64 contractions, 248 us with integer ones (252 with the state weights in FP64) and 1/x and square roots of FP32 seeds, 274 us
// with the IEEE ones again and sums without a mean error (FP64 pipe 72% busy); 64^2: 24.9, 22.4 with one thread per pair
// of lines, 18.6 in halves, 18.7 now.
template <int NP, bool AUX, class PH>
__device__ __forceinline__ void dg_stage(const PH& ph, const BasisDev& B, const Tile2D tl, const Inst2D& I, double c0, double c1,
                                         double c2, bool raw, StageSmem<NP, AUX>& sm) {
  using TL = Tiling2D<NP>;
  constexpr int TE = TL::TE, NN = TL::NN, L = TL::L, TX = TL::TX, TY = TL::TY, NH = TL::NH;
  constexpr int NQ = (TE * NN + 2 * NH - 1) / (2 * NH);  // nodes per thread
  const int dir = threadIdx.x >= NH;  // 0: rows and x faces, 1: columns and y faces
  const ElemView w = elem_view<NP>(tl, I, dir, threadIdx.x - dir * NH);
  const int e = w.e, t = w.t;
  const int st = dir == 0 ? 1 : NP, at = dir == 0 ? t * NP : t;  // node k of the line: at + k st
  const double c2dt = raw ? 1.0 : c2 * I.dt;
  const double sl = -c2dt * (dir == 0 ? I.ijx : I.ijy);

  // ---- nodes: fluxes
  long long node[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const int m = threadIdx.x + q * 2 * NH;
    const int el = m / NN, nd = m % NN, ex = tl.ex0 + el % TX, ey = tl.ey0 + el / TX;
    const bool live = m < TE * NN && ex < I.nex && ey < I.ney;
    const long long n = I.off + (long long)NN * (ex + (long long)I.nex * ey) + nd;
    node[q] = live ? n : -1;
    if (!live) continue;
    const FluxNode f = ph.at(n);
#pragma unroll
    for (int v = 0; v < 4; ++v) sm.q[v][el][nd] = f.q[v];
    sm.f[0][el][nd] = f.fx0; sm.f[1][el][nd] = f.f1; sm.f[2][el][nd] = f.fx3;
    sm.f[3][el][nd] = f.fy1; sm.f[4][el][nd] = f.fy3;
    if (AUX) sm.aux[AUX ? el : 0][nd] = f.aux;
  }
  __syncthreads();
  // The line's flux of component v: the mass flux is the quantity q[dir] itself.
  auto flux = [&](int v, int el, int nd) {
    if (v == 2) return sm.q[dir][el][nd];
    return sm.f[dir == 0 ? v - (v >> 1) : (v == 0 ? 1 : (v == 1 ? 3 : 4))][el][nd];
  };
  // ---- lines: wave speeds at the ends, volume term. The field loops stay rolled: their bodies are a few hundred integer
  // instructions, and four copies of them cost more in instruction fetch than they save.
  if (w.valid) {
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int nd = at + (s == 0 ? 0 : L) * st;
      sm.w[dir][e][t][s] = ph.speed(dir, w.base + nd, sm.q[dir][e][nd], AUX ? sm.aux[AUX ? e : 0][nd] : 0.0, true);
    }
    const FixScale c = fix_scale(sl);
#pragma unroll 1
    for (int v = 0; v < 4; ++v) {
      double f[NP];
#pragma unroll
      for (int k = 0; k < NP; ++k) f[k] = flux(v, e, at + k * st);
      FixSums<NP> r;
      row_scaled<NP, false>(B, c, f, r, raw);
#pragma unroll
      for (int k = 0; k < NP; ++k) sm.k[dir][v][e][at + k * st] = r.G[k];
      sm.ke[dir][v][e][t] = r.e;
    }
  }
  __syncthreads();
  // ---- lines: faces, owner computes its side
  if (w.valid) {
    double pq[2][4], pf[2][3], lam[2];  // the partners' quantities, fluxes (0, 1, 3) and the signed lambda
    const int sf = dir == 0 ? first_side(w.ext, TX) : first_side(w.eyt, TY);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int s = h == 0 ? sf : 1 - sf, d = s == 0 ? -1 : 1;
      int it;
      const long long pb = neighbour<NP>(tl, I, w.ex, w.ey, dir == 0 ? d : 0, dir == 0 ? 0 : d, &it);
      const int nd = at + (s == 0 ? L : 0) * st;
      double q[4], f[3], ws;
      if (it >= 0) {
#pragma unroll
        for (int v = 0; v < 4; ++v) q[v] = sm.q[v][it][nd];
        f[0] = flux(0, it, nd); f[1] = flux(1, it, nd); f[2] = flux(3, it, nd);
        ws = sm.w[dir][it][t][1 - s];
      } else {
        const FluxNode p = ph.at(pb + nd);
#pragma unroll
        for (int v = 0; v < 4; ++v) q[v] = p.q[v];
        f[0] = dir == 0 ? p.fx0 : p.f1; f[1] = dir == 0 ? p.f1 : p.fy1; f[2] = dir == 0 ? p.fx3 : p.fy3;
        ws = ph.speed(dir, pb + nd, p.q[dir], p.aux, false);
      }
      const double own = sm.w[dir][e][t][s];
      const double mag = max_nonneg(s == 0 ? own : ws, s == 0 ? ws : own);
#pragma unroll
      for (int r = 0; r < 2; ++r) {  // register arrays by the run-time side
        if (r != s) continue;
        lam[r] = r == 0 ? mag : -mag;
#pragma unroll
        for (int v = 0; v < 4; ++v) pq[r][v] = q[v];
#pragma unroll
        for (int v = 0; v < 3; ++v) pf[r][v] = f[v];
      }
    }
    double add[2][4];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int nd = at + (s == 0 ? 0 : L) * st;
      const double cf = s == 0 ? -0.5 * B.iw0 * sl : 0.5 * B.iwL * sl;
      double dq[4];
#pragma unroll
      for (int v = 0; v < 4; ++v) dq[v] = pq[s][v] - sm.q[v][e][nd];
      add[s][0] = cf * llf_jump(pf[s][0], flux(0, e, nd), lam[s], dq[0]);
      add[s][1] = cf * llf_jump(pf[s][1], flux(1, e, nd), lam[s], dq[1]);
      add[s][2] = cf * fma(lam[s], dq[2], dir == 0 ? dq[0] : dq[1]);  // the mass flux is q[dir]
      add[s][3] = cf * llf_jump(pf[s][2], flux(3, e, nd), lam[s], dq[3]);
    }
#pragma unroll 1
    for (int v = 0; v < 4; ++v) {
      FixSums<NP> r;
#pragma unroll
      for (int k = 0; k < NP; ++k) r.G[k] = sm.k[dir][v][e][at + k * st];
      r.e = sm.ke[dir][v][e][t];
      row_add_ends<NP>(r, pick4(add[0], v), pick4(add[1], v));
#pragma unroll
      for (int k = 0; k < NP; ++k) sm.k[dir][v][e][at + k * st] = r.G[k];
      sm.ke[dir][v][e][t] = r.e;
    }
  }
  // ---- nodes: RK combination; q^n is loaded before the barrier and before anything is stored
  const bool with_qn = !raw && __double_as_longlong(c0) != 0;
  const FixScale w0 = fix_scale(c0), w1 = fix_scale(c1);
  double qn[NQ][4];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    if (node[q] < 0) continue;
#pragma unroll
    for (int v = 0; v < 4; ++v) qn[q][v] = with_qn ? ph.qn(v, node[q]) : 0.0;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const long long n = node[q];
    if (n < 0) continue;
    const int m = threadIdx.x + q * 2 * NH;
    const int el = m / NN, nd = m % NN, j = nd / NP, i = nd % NP;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const double qs = sm.q[v][el][nd];
      const long long r = sm.k[0][v][el][nd], c = sm.k[1][v][el][nd];
      const int er = sm.ke[0][v][el][j], ec = sm.ke[1][v][el][i];
      ph.put(v, n, with_qn ? node_blend(r, er, c, ec, qs, w1, qn[q][v], w0)
                           : node_total<60>(r, er, c, ec, raw ? 0.0 : qs, 1));  // without q^n: c1 = 1
    }
  }
}

// The Euler fluxes (hyperbolic.jl) with the wave speeds computed here.
struct EulerStage {
  const HypArgs2D& a;
  double g;
  __device__ __forceinline__ FluxNode at(long long n) const {
    FluxNode f;
#pragma unroll
    for (int v = 0; v < 4; ++v) f.q[v] = a.q[v][n];
    const NodePhys p = node_phys(g, f.q[0], f.q[1], f.q[3], a.S[n], a.invr[n]);
    f.fx0 = p.fx[0]; f.f1 = p.fx[1]; f.fx3 = p.fx[3]; f.fy1 = p.fy[1]; f.fy3 = p.fy[3];
    f.aux = p.P;
    return f;
  }
  __device__ __forceinline__ double speed(int dir, long long n, double m, double P, bool own) const {
    const double ir = a.invr[n];
    const double ws = wavespeed(g, m * ir, P, ir);
    double* out = dir == 0 ? a.ws_x : a.ws_y;
    if (own && out) out[n] = ws;
    return ws;
  }
  __device__ __forceinline__ double qn(int v, long long n) const { return a.qn[v][n]; }
  __device__ __forceinline__ void put(int v, long long n, double x) const {
    if (a.k_out[v]) a.k_out[v][n] = x;
    if (a.qo[v]) a.qo[v][n] = x;
    if (v == 2 && a.invro) a.invro[n] = 1.0 / x;
    if (a.status && (v == 2 ? not_positive_finite(x) : nonfinite_bits(x))) flag_nonfinite(a.status);
  }
};

template <int NP>
__global__ void __launch_bounds__(2 * Tiling2D<NP>::NH) k2_hyp_rk(HypArgs2D a) {
  __shared__ StageSmem<NP, true> sm;
  const Tile2D tl = a.tiles[blockIdx.x];
  const Inst2D I = a.inst[tl.inst];
  chained_start();
  dg_stage<NP, true>(EulerStage{a, I.gamma}, a.B, tl, I, a.c0, a.c1, a.c2, a.k_out[0] != nullptr, sm);
}

}  // namespace igrgpu
