// dg_adjoint.cuh -- tangent-linear and adjoint kernels of the shallow-water
// RK-DG right-hand side (no reference counterpart: DGCUDA has no
// derivatives).
//
// L(u, b) = (1/J) [ V(u, b) + S(u) ] with, per element and mode i,
//   V_i = sum_q GR_qi Gr_q + GS_qi Gs_q  + sum_q B_qi w_q J src_q
//   S_i = -/+ sum_j (len/2) w_j F*(U_L(j), U_R(j); n) E_i(j)     (left / right)
// Gr = fx ys - fy xs, Gs = fy xr - fx yr, src = (0, -g h b_x, -g h b_y).
// Both derivative codes use the same hand-derived 3x3 Jacobians, applied to
// vectors without forming them (sw_jac_mul, sw_jac_tmul):
//   A(U; n) = d(F(U).n)/dU, the physical normal flux of shallow water;
//   Rusanov F* = 1/2 (F(U_L).n + F(U_R).n + lam (U_L - U_R)),
//   lam = max(lam_L, lam_R), lam_X = |q_X / h_X| + sqrt(g h_X), q = m.n:
//     dF*/dU_L = 1/2 (A_L + lam I + (U_L - U_R) dlam/dU_L)
//     dF*/dU_R = 1/2 (A_R - lam I + (U_L - U_R) dlam/dU_R)
//   with the branch of the max (and the sign of q) taken from the state.
// Tangent-linear: dL = (dL/du) du + (dL/db) db (matrix-vector with A);
// adjoint: (dL/du)^T Lbar and (dL/db)^T Lbar (with A^T).  The dot-product
// test <Lbar, dL> = <ubar, du> + <bbar, db> holds to rounding.
#pragma once
#include "dg_fixed.cuh"

namespace dg {

// A(U; n) = d(F(U).n)/dU for shallow water, U = (h, hu, hv), applied to a
// vector without forming the matrix.  With u = hu/h, v = hv/h, qh = (hu,hv).n/h
// and gh = g h the rows are
//   [0, nx, ny],  [gh nx - u qh, u nx + qh, u ny],  [gh ny - v qh, v nx, v ny + qh].
// y = A x
__device__ __forceinline__ void sw_jac_mul(double u, double v, double qh, double gh, double nx,
                                           double ny, const double *x, double *y) {
  const double xn = fma(nx, x[1], ny * x[2]);
  const double t = fma(-qh, x[0], xn);
  const double g0 = gh * x[0];
  y[0] = xn;
  y[1] = fma(u, t, fma(qh, x[1], g0 * nx));
  y[2] = fma(v, t, fma(qh, x[2], g0 * ny));
}
// z = A^T f
__device__ __forceinline__ void sw_jac_tmul(double u, double v, double qh, double gh, double nx,
                                            double ny, const double *f, double *z) {
  const double wf = fma(u, f[1], v * f[2]);
  const double fn = fma(nx, f[1], ny * f[2]);
  const double fw = f[0] + wf;
  z[0] = fma(-qh, wf, gh * fn);
  z[1] = fma(nx, fw, qh * f[1]);
  z[2] = fma(ny, fw, qh * f[2]);
}

// one trace of a side: the pieces of A(U; n), c = sqrt(g h) and
// lam = |qh| + c
struct SwTrace {
  double ih, u, v, qh, gh, c, lam;
};
__device__ __forceinline__ SwTrace sw_trace(double g, const double *U, double nx, double ny) {
  SwTrace w;
  w.ih = rcp_fx(U[0]);
  w.u = U[1] * w.ih;
  w.v = U[2] * w.ih;
  w.qh = fma(U[1], nx, U[2] * ny) * w.ih;
  w.gh = g * U[0];
  w.c = sqrt_fx(w.gh);
  w.lam = fabs(w.qh) + w.c;
  return w;
}
// d lam / dU = (-sg qh / h + c / (2 h), sg nx / h, sg ny / h), sg = sign(qh)
// (d sqrt(g h)/dh = g / (2 c) = c / (2 h))
__device__ __forceinline__ void sw_dlam(const SwTrace &w, double nx, double ny, double dl[3]) {
  const double sih = w.qh >= 0.0 ? w.ih : -w.ih;
  dl[0] = fma(-w.qh, sih, 0.5 * w.c * w.ih);
  dl[1] = sih * nx;
  dl[2] = sih * ny;
}

// d(ghost)/d(U_L) of a boundary code (reflect mirrors the momentum,
// transmissive copies, inflow / outflow ghosts do not depend on U_L)
__device__ __forceinline__ void sw_ghost_jac(int code, double nx, double ny, double M[3][3]) {
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 3; b++) M[a][b] = 0.0;
  if (code == -4) {
    M[0][0] = M[1][1] = M[2][2] = 1.0;
  } else if (code == -1) {
    M[0][0] = 1.0;
    M[1][1] = 1.0 - 2 * nx * nx;
    M[1][2] = -2 * nx * ny;
    M[2][1] = -2 * ny * nx;
    M[2][2] = 1.0 - 2 * ny * ny;
  }
}

// ---------------------------------------------------------------------------
// linear traces of a field (no admissibility check): Tv[e][f][j][n]
template <int P>
__global__ void __launch_bounds__(kBlock) k_lin_trace(const __grid_constant__ Tab<P> tab,
                                                      const double *__restrict__ u,
                                                      const double *__restrict__ scale,
                                                      double sc, double *__restrict__ Tv, int K,
                                                      int Kp) {
  constexpr int N = 3, NP = Tab<P>::NP, N1 = Tab<P>::N1;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= K) return;
  const double f0 = scale ? sc * scale[e] : sc;
  double *Te = Tv + (size_t)e * (3 * N1 * N);
#pragma unroll
  for (int n = 0; n < N; n++) {
    double c[NP];
#pragma unroll
    for (int i = 0; i < NP; i++) c[i] = f0 * u[(size_t)(n * NP + i) * Kp + e];
#pragma unroll
    for (int f = 0; f < 3; f++)
#pragma unroll
      for (int j = 0; j < N1; j++) {
        double a = c[0] * tab.E[f][j][0];
#pragma unroll
        for (int i = 1; i < NP; i++) a = fma(c[i], tab.E[f][j][i], a);
        Te[(f * N1 + j) * N + n] = a;
      }
  }
}

// ---------------------------------------------------------------------------
// TL face: dF*(j) = (dF*/dU_L dU_L + dF*/dU_R dU_R) len/2 w_j into dFh.
// ADJ face: Fbar(j) = len/2 w_j (-Tbar_L(j) + Tbar_R(p-j)) from the
// adjoint traces, then Ubar_L = A_L^T Fbar -> UbL[s][j], Ubar_R = A_R^T
// Fbar -> UbR[s][j] (for a boundary side Ubar_R goes back to U_L).
template <int P, bool ADJ>
__global__ void __launch_bounds__(kBlock)
    k_sw_face_lin(const __grid_constant__ Tab<P> tab, const __grid_constant__ EqP q,
                  const double *__restrict__ T, const double *__restrict__ Tv,
                  const int4 *__restrict__ side, const double *__restrict__ sgeo,
                  double *__restrict__ out0, double *__restrict__ out1, int S) {
  constexpr int N = 3, N1 = P + 1;
  // a thread per edge point, as k_face
  const int i = blockIdx.x * blockDim.x + threadIdx.x, s = i / N1, j = i % N1;
  if (s >= S) return;
  const int4 sd = side[s];
  const double nx = sgeo[s], ny = sgeo[S + s], hl = sgeo[2 * (size_t)S + s];
  const double *TL = T + ((size_t)sd.x * 3 + sd.z) * (N1 * N);
  const double *VL = Tv + ((size_t)sd.x * 3 + sd.z) * (N1 * N);
  const bool inner = sd.y >= 0;
  const double *TR = inner ? T + ((size_t)sd.y * 3 + sd.w) * (N1 * N) : nullptr;
  const double *VR = inner ? Tv + ((size_t)sd.y * 3 + sd.w) * (N1 * N) : nullptr;
  {
    double UL[N], UR[N], M[3][3];
#pragma unroll
    for (int n = 0; n < N; n++) UL[n] = TL[j * N + n];
    if (inner) {
#pragma unroll
      for (int n = 0; n < N; n++) UR[n] = TR[(N1 - 1 - j) * N + n];
    } else {
      ghost_state<ShallowWater>(q, sd.y, UL, UR, 0.0, 0.0, 0.0, nx, ny);
      sw_ghost_jac(sd.y, nx, ny, M);
    }
    // Rusanov: dF*/dU_L = 1/2 (A_L + lam I + d dlam_L^T), dF*/dU_R = 1/2 (A_R
    // - lam I + d dlam_R^T), d = U_L - U_R, the dlam term on the side of the
    // max only; the 1/2 goes into the edge scale
    const SwTrace wL = sw_trace(q.g, UL, nx, ny), wR = sw_trace(q.g, UR, nx, ny);
    const bool left = wL.lam >= wR.lam;
    const double lam = left ? wL.lam : wR.lam;
    double dl[3];
    sw_dlam(left ? wL : wR, nx, ny, dl);
    const double sc = 0.5 * hl * tab.w1[j];
    if (!ADJ) {
      double dUL[N], dUR[N], aL[N], aR[N];
#pragma unroll
      for (int n = 0; n < N; n++) dUL[n] = VL[j * N + n];
      if (inner) {
#pragma unroll
        for (int n = 0; n < N; n++) dUR[n] = VR[(N1 - 1 - j) * N + n];
      } else {
#pragma unroll
        for (int a = 0; a < N; a++)
          dUR[a] = fma(M[a][0], dUL[0], fma(M[a][1], dUL[1], M[a][2] * dUL[2]));
      }
      sw_jac_mul(wL.u, wL.v, wL.qh, wL.gh, nx, ny, dUL, aL);
      sw_jac_mul(wR.u, wR.v, wR.qh, wR.gh, nx, ny, dUR, aR);
      const double *dX = left ? dUL : dUR;
      const double dlam = fma(dl[0], dX[0], fma(dl[1], dX[1], dl[2] * dX[2]));
#pragma unroll
      for (int a = 0; a < N; a++) {
        const double v = fma(UL[a] - UR[a], dlam, fma(lam, dUL[a] - dUR[a], aL[a] + aR[a]));
        out0[(size_t)s * (N1 * N) + j * N + a] = v * sc;
      }
    } else {
      double Fb[N];
#pragma unroll
      for (int n = 0; n < N; n++) {
        const double r = inner ? VR[(N1 - 1 - j) * N + n] : 0.0;
        Fb[n] = sc * (r - VL[j * N + n]);
      }
      double bL[N], bR[N];
      sw_jac_tmul(wL.u, wL.v, wL.qh, wL.gh, nx, ny, Fb, bL);
      sw_jac_tmul(wR.u, wR.v, wR.qh, wR.gh, nx, ny, Fb, bR);
      const double dF = fma(UL[0] - UR[0], Fb[0], fma(UL[1] - UR[1], Fb[1], (UL[2] - UR[2]) * Fb[2]));
#pragma unroll
      for (int b = 0; b < N; b++) {
        bL[b] = fma(lam, Fb[b], bL[b]);
        bR[b] = fma(-lam, Fb[b], bR[b]);
        if (left) bL[b] = fma(dl[b], dF, bL[b]);
        else bR[b] = fma(dl[b], dF, bR[b]);
      }
      if (!inner) {  // U_R = ghost(U_L): its adjoint returns to U_L
#pragma unroll
        for (int b = 0; b < N; b++)
          bL[b] = fma(M[0][b], bR[0], fma(M[1][b], bR[1], fma(M[2][b], bR[2], bL[b])));
      }
#pragma unroll
      for (int n = 0; n < N; n++) {
        out0[(size_t)s * (N1 * N) + j * N + n] = bL[n];
        out1[(size_t)s * (N1 * N) + j * N + n] = inner ? bR[n] : 0.0;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// TL element: dout = ca du^n + cb du_s + cc dt (1/J) [dV + dS], dS gathered
// from dFh like the forward surface term.
template <int P>
__global__ void __launch_bounds__(kBlock)
    k_sw_element_tl(const __grid_constant__ Tab<P> tab, const __grid_constant__ EqP q,
                     const double *__restrict__ us, const double *__restrict__ bz_all,
                     const double *__restrict__ vin, const double *__restrict__ dbz_all,
                     const double *__restrict__ vn, double *__restrict__ vout,
                     const double *__restrict__ F0, const int *__restrict__ esd,
                     const double *__restrict__ geo, double ca, double cb, double ccdt, int K,
                     int Kp) {
  constexpr int N = 3, NP = Tab<P>::NP, NQ = Tab<P>::NQ, N1 = Tab<P>::N1;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= K) return;
  double c[N][NP], v[N][NP], acc[N][NP], bz[NP], dbz[NP];
#pragma unroll
  for (int n = 0; n < N; n++)
#pragma unroll
    for (int i = 0; i < NP; i++) {
      c[n][i] = us[(size_t)(n * NP + i) * Kp + e];
      v[n][i] = vin[(size_t)(n * NP + i) * Kp + e];
      acc[n][i] = 0.0;
    }
#pragma unroll
  for (int i = 0; i < NP; i++) {
    bz[i] = bz_all ? bz_all[(size_t)i * Kp + e] : 0.0;
    dbz[i] = dbz_all ? dbz_all[(size_t)i * Kp + e] : 0.0;
  }
  const double xr = geo[e], yr = geo[(size_t)Kp + e], xs = geo[2 * (size_t)Kp + e],
               ys = geo[3 * (size_t)Kp + e], iJ = geo[4 * (size_t)Kp + e];
  const double g = q.g;
#pragma unroll
  for (int k = 0; k < NQ; k++) {
    double U[N];
#pragma unroll
    for (int n = 0; n < N; n++) {
      double a = c[n][0] * tab.B[k][0];
#pragma unroll
      for (int i = 1; i < NP; i++) a = fma(c[n][i], tab.B[k][i], a);
      U[n] = a;
    }
    // A_x = A(U; (1, 0)) and A_y = A(U; (0, 1)): qh is u resp. v
    const double ih = rcp(U[0]);
    const double uu = U[1] * ih, vv = U[2] * ih, gh = g * U[0];
    double br = 0.0, bs = 0.0;
#pragma unroll
    for (int i = 1; i < NP; i++) {
      br = fma(bz[i], tab.GR[k][i], br);
      bs = fma(bz[i], tab.GS[k][i], bs);
    }
    const double bx = fma(ys, br, -yr * bs), by = fma(xr, bs, -xs * br);
    double dU[N];
#pragma unroll
    for (int n = 0; n < N; n++) {
      double a = v[n][0] * tab.B[k][0];
#pragma unroll
      for (int i = 1; i < NP; i++) a = fma(v[n][i], tab.B[k][i], a);
      dU[n] = a;
    }
    double dfx[N], dfy[N];
    sw_jac_mul(uu, vv, uu, gh, 1.0, 0.0, dU, dfx);
    sw_jac_mul(uu, vv, vv, gh, 0.0, 1.0, dU, dfy);
#pragma unroll
    for (int n = 0; n < N; n++) {
      const double gr = fma(dfx[n], ys, -dfy[n] * xs), gs = fma(dfy[n], xr, -dfx[n] * yr);
#pragma unroll
      for (int i = 1; i < NP; i++)
        acc[n][i] = fma(tab.GR[k][i], gr, fma(tab.GS[k][i], gs, acc[n][i]));
    }
    if (bz_all || dbz_all) {
      double dbr = 0.0, dbs = 0.0;
#pragma unroll
      for (int i = 1; i < NP; i++) {
        dbr = fma(dbz[i], tab.GR[k][i], dbr);
        dbs = fma(dbz[i], tab.GS[k][i], dbs);
      }
      const double dbx = fma(ys, dbr, -yr * dbs), dby = fma(xr, dbs, -xs * dbr);
      const double sx = -g * fma(dU[0], bx, U[0] * dbx), sy = -g * fma(dU[0], by, U[0] * dby);
#pragma unroll
      for (int i = 0; i < NP; i++) {
        acc[1][i] = fma(sx, tab.B[k][i], acc[1][i]);
        acc[2][i] = fma(sy, tab.B[k][i], acc[2][i]);
      }
    }
  }
  // surface
#pragma unroll
  for (int f = 0; f < 3; f++) {
    const int sd = esd[(size_t)f * Kp + e];
    const bool right = sd & 1;
    const size_t so = (size_t)(sd >> 1) * (N1 * N);
#pragma unroll
    for (int j = 0; j < N1; j++) {
      const int jj = right ? (N1 - 1 - j) : j;
#pragma unroll
      for (int n = 0; n < N; n++) {
        const double fv = (right ? 1.0 : -1.0) * F0[so + jj * N + n];
#pragma unroll
        for (int i = 0; i < NP; i++) acc[n][i] = fma(fv, tab.E[f][j][i], acc[n][i]);
      }
    }
  }
  const double s = ccdt * iJ;
#pragma unroll
  for (int n = 0; n < N; n++)
#pragma unroll
    for (int i = 0; i < NP; i++) {
      const size_t o = (size_t)(n * NP + i) * Kp + e;
      double r = fma(s, acc[n][i], cb * v[n][i]);
      if (ca != 0.0) r = fma(ca, vn[o], r);
      vout[o] = r;
    }
}

// ---------------------------------------------------------------------------
// The adjoint element stage with its contractions in fixed point (dg_fixed.cuh:
// one warp per variable, one lane per element).  With v = ccdt (1/J) obar,
//   ubar = cb obar + (dV/du)^T v + (surface, gathered from UbL / UbR)
//          [+ a0 x0 + a1 x1]
// and bbar += (dV/db)^T v.  The contractions: U(q) = B us, the projections of
// v on the gradients and (momenta) on the basis at the area points, and back
// from the points' adjoints and the side terms to the modes.  With Tv, the
// traces of tc (1/J) ubar, the next stage's k_lin_trace, follow.
// Before, p = 2, 45k triangles, us a stage: FP64 element 129, k_lin_trace 24,
// combination 6 (face 59, forward traces 9); a gradient over 10 steps 9.42 ->
// 5.77 ms.
struct AdjArgs {
  const double *us, *obar, *x0, *x1;  // x0, x1 null: no extra terms
  double *ubar, *bbar, *Tv;           // Tv null: no traces
  const double *F0, *F1, *bslope, *geo;
  const int *esd;
  double cb, ccdt, a0, a1, tc;
  int K, Kp;
};

template <int P>
__global__ void __launch_bounds__(96, P <= 2 ? 8 : 5)
    k_adj_element_fx(const __grid_constant__ fx::FxTab<P> tab, const __grid_constant__ EqP q,
                     const __grid_constant__ AdjArgs a) {
  using namespace fx;
  constexpr int N = 3, NP = Tab<P>::NP, NQ = Tab<P>::NQ, N1 = P + 1, NF = 3 * N1;
  // rows of kPitch doubles: block b of N NQ rows, variable n at point k in row
  // (b NQ + k) N + n: b = 0 U, then its adjoint; 1, 2 the projections on the
  // gradients; the momenta's on the basis, then the slopes' adjoints, in
  // rows 3 NQ N + 2 k + (n - 1)
  __shared__ double st[(3 * NQ * N + 2 * NQ) * kPitch];
  __shared__ int mxs[(N + 1) * N * kTile];
  const int lane = threadIdx.x & 31, n = threadIdx.x >> 5, e0 = blockIdx.x * kTile;
  const int e = e0 + lane, ec = e < a.K ? e : a.K - 1;
  const bool live = e < a.K;
  const size_t Kp = a.Kp;
  const double *geo = a.geo;
  const double iJ = geo[4 * Kp + ec];
  auto at = [&](int b, int k, int v) -> double & { return st[((b * NQ + k) * N + v) * kPitch + lane]; };
  auto src = [&](int k, int v) -> double & { return st[(3 * NQ * N + 2 * k + (v - 1)) * kPitch + lane]; };
  {  // U(q)
    double c[NP];
    int mx = 0;
#pragma unroll
    for (int i = 0; i < NP; i++) {
      c[i] = a.us[(size_t)(n * NP + i) * Kp + ec];
      mx = max(mx, abs_hi(c[i]));
    }
    const Row row = make_row(mx);
    int h[NP], l[NP];
#pragma unroll
    for (int i = 0; i < NP; i++) to_limbs(c[i], row, h[i], l[i]);
    const int base = base_exp(row, tab.eB);
#pragma unroll
    for (int k = 0; k < NQ; k++) {
      Sum s;
      zero(s);
#pragma unroll
      for (int i = 0; i < NP; i++) mac(s, h[i], l[i], tab.B[k][i]);
      at(0, k, n) = finish(s, base);
    }
    if (row.odd()) fix(&at(0, 0, n), N * kPitch, NQ, row);
  }
  {  // v's projections
    const double f = a.ccdt * iJ;
    double c[NP];
    int mx = 0;
#pragma unroll
    for (int i = 0; i < NP; i++) {
      c[i] = f * a.obar[(size_t)(n * NP + i) * Kp + ec];
      mx = max(mx, abs_hi(c[i]));
    }
    const Row row = make_row(mx);
    int h[NP], l[NP];
#pragma unroll
    for (int i = 0; i < NP; i++) to_limbs(c[i], row, h[i], l[i]);
    const int base = base_exp(row, tab.eP), baseB = base_exp(row, tab.eB);
#pragma unroll
    for (int k = 0; k < NQ; k++) {
#pragma unroll
      for (int b = 0; b < 2; b++) {
        Sum s;
        zero(s);
#pragma unroll
        for (int i = 1; i < NP; i++) mac(s, h[i], l[i], tab.G[k][b][i]);
        at(1 + b, k, n) = finish(s, base);
      }
      if (n > 0) {
        Sum s;
        zero(s);
#pragma unroll
        for (int i = 0; i < NP; i++) mac(s, h[i], l[i], tab.B[k][i]);
        src(k, n) = finish(s, baseB);
      }
    }
    if (row.odd()) {
      fix(&at(1, 0, n), N * kPitch, 2 * NQ, row);
      if (n > 0) fix(&src(0, n), 2 * kPitch, NQ, row);
    }
  }
  // the side terms, read after the points
  const double *Fp[3];
  bool right[3];
#pragma unroll
  for (int f = 0; f < 3; f++) {
    const int sd = a.esd[(size_t)f * Kp + ec];
    right[f] = sd & 1;
    Fp[f] = (right[f] ? a.F1 : a.F0) + (size_t)(sd >> 1) * (N1 * N) + n;
    asm volatile("prefetch.global.L1 [%0];" ::"l"(Fp[f]));
  }
  __syncthreads();
  {  // the points' adjoints; the warps share the points out
    const double xr = geo[ec], yr = geo[Kp + ec], xs = geo[2 * Kp + ec], ys = geo[3 * Kp + ec];
    int mx[N + 1] = {0, 0, 0, 0};
#pragma unroll 1
    for (int k = n; k < NQ; k += N) {
      const double U0 = at(0, k, 0), ih = rcp(U0);
      const double uu = at(0, k, 1) * ih, vv = at(0, k, 2) * ih, gh = q.g * U0;
      double fxb[N], fyb[N], zx[N], zy[N];
#pragma unroll
      for (int v = 0; v < N; v++) {
        const double Gr = at(1, k, v), Gs = at(2, k, v);
        fxb[v] = fma(ys, Gr, -yr * Gs);
        fyb[v] = fma(xr, Gs, -xs * Gr);
      }
      sw_jac_tmul(uu, vv, uu, gh, 1.0, 0.0, fxb, zx);
      sw_jac_tmul(uu, vv, vv, gh, 0.0, 1.0, fyb, zy);
      double Ub[N];
#pragma unroll
      for (int v = 0; v < N; v++) Ub[v] = zx[v] + zy[v];
      if (a.bbar) {
        const double bx = a.bslope ? a.bslope[(size_t)k * Kp + ec] : 0.0;
        const double by = a.bslope ? a.bslope[(size_t)(NQ + k) * Kp + ec] : 0.0;
        const double Sx = src(k, 1), Sy = src(k, 2);
        Ub[0] = fma(-q.g, fma(bx, Sx, by * Sy), Ub[0]);
        const double hb = -q.g * U0;
        const double bxb = hb * Sx, byb = hb * Sy;  // adjoints of bx, by
        const double brb = fma(ys, bxb, -xs * byb), bsb = fma(xr, byb, -yr * bxb);
        src(k, 1) = brb;
        src(k, 2) = bsb;
        mx[N] = max(mx[N], max(abs_hi(brb), abs_hi(bsb)));
      }
#pragma unroll
      for (int v = 0; v < N; v++) {
        at(0, k, v) = Ub[v];
        mx[v] = max(mx[v], abs_hi(Ub[v]));
      }
    }
#pragma unroll
    for (int v = 0; v <= N; v++) mxs[(v * N + n) * kTile + lane] = mx[v];
  }
  __syncthreads();
  if (n == 0 && a.bbar) {  // the bed's adjoint: the variable without projections on the basis
    int mx = 0;
#pragma unroll
    for (int w = 0; w < N; w++) mx = max(mx, mxs[(N * N + w) * kTile + lane]);
    const Row row = make_row(mx);
    Sum s[NP];
#pragma unroll
    for (int i = 1; i < NP; i++) zero(s[i]);
#pragma unroll
    for (int k = 0; k < NQ; k++)
#pragma unroll
      for (int b = 0; b < 2; b++) {
        int h, l;
        to_limbs(src(k, 1 + b), row, h, l);
#pragma unroll
        for (int i = 1; i < NP; i++) mac(s[i], h, l, tab.G[k][b][i]);
      }
    const int base = base_exp(row, tab.eP);
    double r[NP];
    r[0] = 0.0;
#pragma unroll
    for (int i = 1; i < NP; i++) r[i] = finish(s[i], base);
    if (row.odd()) {  // through the slopes' rows, which are free now
#pragma unroll
      for (int i = 1; i < NP; i++) st[(3 * NQ * N + i) * kPitch + lane] = r[i];
      fix(&st[(3 * NQ * N + 1) * kPitch + lane], kPitch, NP - 1, row);
#pragma unroll
      for (int i = 1; i < NP; i++) r[i] = st[(3 * NQ * N + i) * kPitch + lane];
    }
    if (live)
#pragma unroll
      for (int i = 1; i < NP; i++) a.bbar[(size_t)i * Kp + e] += r[i];
  }
  double c[NP];
  {
    double F[NF];
#pragma unroll
    for (int f = 0; f < 3; f++)
#pragma unroll
      for (int j = 0; j < N1; j++) F[f * N1 + j] = Fp[f][(right[f] ? N1 - 1 - j : j) * N];
    int mx = 0;
#pragma unroll
    for (int w = 0; w < N; w++) mx = max(mx, mxs[(n * N + w) * kTile + lane]);
#pragma unroll
    for (int k = 0; k < NF; k++) mx = max(mx, abs_hi(F[k]));
    const Row row = make_row(mx);
    Sum s[NP];
#pragma unroll
    for (int i = 0; i < NP; i++) zero(s[i]);
#pragma unroll
    for (int k = 0; k < NF; k++) {
      int h, l;
      to_limbs(F[k], row, h, l);
#pragma unroll
      for (int i = 0; i < NP; i++) mac(s[i], h, l, tab.S[k][i]);
    }
#pragma unroll
    for (int k = 0; k < NQ; k++) {
      int h, l;
      to_limbs(at(0, k, n), row, h, l);
#pragma unroll
      for (int i = 0; i < NP; i++) mac(s[i], h, l, tab.Q[k][i]);
    }
    const int base = base_exp(row, tab.eP);
#pragma unroll
    for (int i = 0; i < NP; i++) c[i] = finish(s[i], base);
    if (row.odd()) {  // through the thread's own projection rows, which are free now
#pragma unroll
      for (int i = 0; i < NP; i++) at(1, i, n) = c[i];
      fix(&at(1, 0, n), N * kPitch, NP, row);
#pragma unroll
      for (int i = 0; i < NP; i++) c[i] = at(1, i, n);
    }
#pragma unroll
    for (int i = 0; i < NP; i++) {
      const size_t o = (size_t)(n * NP + i) * Kp + ec;
      double v = fma(a.cb, a.obar[o], c[i]);
      if (a.x0) v += fma(a.a0, a.x0[o], a.a1 * a.x1[o]);
      c[i] = v;
    }
    if (live)
#pragma unroll
      for (int i = 0; i < NP; i++) a.ubar[(size_t)(n * NP + i) * Kp + e] = c[i];
  }
  if (!a.Tv) return;
  {  // traces of tc (1/J) ubar
    const double f = a.tc * iJ;
    int mx = 0;
#pragma unroll
    for (int i = 0; i < NP; i++) {
      c[i] *= f;
      mx = max(mx, abs_hi(c[i]));
    }
    const Row row = make_row(mx);
    int h[NP], l[NP];
#pragma unroll
    for (int i = 0; i < NP; i++) to_limbs(c[i], row, h[i], l[i]);
    const int base = base_exp(row, tab.eE);
#pragma unroll
    for (int k = 0; k < NF; k++) {
      Sum s;
      zero(s);
#pragma unroll
      for (int i = 0; i < NP; i++) mac(s, h[i], l[i], tab.E[k][i]);
      st[(k * N + n) * kPitch + lane] = finish(s, base);
    }
    if (row.odd()) fix(&st[n * kPitch + lane], N * kPitch, NF, row);
    __syncthreads();
    constexpr int C = NF * N;
#pragma unroll 2
    for (int el = n; el < kTile; el += N) {
      if (e0 + el >= a.K) break;
      double *Te = a.Tv + (size_t)(e0 + el) * C;
#pragma unroll
      for (int r = 0; r < C; r += 32)
        if (r + lane < C) Te[r + lane] = st[(r + lane) * kPitch + el];
    }
  }
}

}  // namespace dg
