// dg_fixed.cuh -- the element stage with its basis contractions in fixed
// point on the integer multiply-add pipe (p = 1..4, all equations).
//
// What bounds the stage: GB300 runs 2 FP64 FMAs per SM and cycle (measured
// 1.97), and the contractions with the constant basis tables -- values at the
// area points, the projection of the volume and side fluxes, the next stage's
// edge traces -- are four fifths of the stage's FP64 work.  It runs 32 integer
// multiply-adds 32 x 32 + 64 -> 64 bits (mad.wide.s32: 4 issue cycles of a
// sub-partition's heavy FMA pipe), beside the FP64 pipe, so three of them per
// product are still five times the FP64 rate:
//
//  * a row of inputs (one element and variable) shares the exponent of its
//    largest entry; each entry becomes a 57-bit integer X (four bits more
//    than a double's significand, so entries down to 1/16 of the largest are
//    exact) in two limbs X = h 2^28 + l, l in [-2^27, 2^27];
//  * the tables are rounded on the host to T = th 2^28 + tl, tl in [-2^27, 2^27),
//    one exponent per table: |T| < 2^56, the projection's, which are the larger
//    ones, |T| <= 2^58 with the |T| of a sum below 2^61 together (dg_fixed.cu);
//  * three multiply-adds per product into two 64-bit sums: H += h th, M += h
//    tl + l th.  At most 63 products meet in one sum (p = 4 with a bed: 3 x 16
//    area and 15 edge points), so |H| <= 2^62 and |M| < 2^63.  The product
//    l tl is left out: below 2^54 against 2^113 (2^115) of full scale;
//  * H + (M >> 28) is the dot product in units of 2^56 of the products' own; it
//    is normalised and rounded to a double with integer instructions.
//  RMS errors against rational arithmetic for modes that decay from a mean of 1 to
//  2, p = 1 to 4 (FP64 FMAs): area values 1.0, 1.2, 1.2, 1.3e-16 (1.7, 2.7, 3.2, 3.5e-16),
//  traces 1.1, 1.3, 1.2, 1.6e-16 (1.9, 2.4, 3.3, 3.8e-16), the projection of their
//  advection 0.2, 0.3, 0.5, 0.7e-16 (3.6, 4.3, 6.4, 8.4e-16).  Whole runs against
//  113-bit arithmetic (10 steps, all equations and schemes): no farther than with
//  FP64 contractions at p = 1, where the state's own rounding is all, and down to a
//  fifth of its distance for Euler at p = 4.
//
// Layout: a block is 32 elements (one per lane) and one warp per variable, so
// a row's exponent, limbs and sums stay in one thread, every state row is
// read and written as whole 256-byte lines, and a table entry is the same for
// all threads (a constant-bank operand of the multiply-add that uses it, with
// the loops unrolled: indexed constant loads cost 15 % at p = 3).  What needs
// all variables of a point crosses the warps through shared memory: area
// values -> fluxes (the warps share the points out) -> projection, and the
// new traces, which leave for T as contiguous rows.
//
// Measured, Euler with the limiter, ms per launch (before: the contractions
// as f16 digit slices on the tensor cores, 34 MMAs per 7 x 7 digit product on
// 16 x 8 x 16 blocks of which half is padding): p = 3, 2.1M triangles 5.41 ->
// 2.80.  The other equations (before: FP64 FMAs), microseconds at 131k triangles
// (p = 4: 80k; advection 131k), p = 1 to 4: shallow water with a bed 92 -> 39,
// 268 -> 82, 676 -> 182, 891 -> 225; Maxwell 71 -> 33, 205 -> 62, 527 -> 135, 710
// -> 164; advection with a velocity field 35 -> 23, 86 -> 37, 206 -> 71, 371 ->
// 114.  At p = 3 (ncu, 524k) the FP64 pipe -- fluxes, RK combination, limiter --
// is 57 % busy, the heavy FMA pipe 66 % and the integer ALU 38 %.
#pragma once
#include "dg_kernels.cuh"
namespace dg {
namespace fx {

constexpr int kTile = 32;                // elements of a block
constexpr int kPitch = kTile + 1;        // shared row pitch: rows and columns both conflict-free

// tables of order P in limbs, and what the FP64 parts need of Tab<P>
template <int P>
struct FxTab {
  static constexpr int NP = Tab<P>::NP, NQ = Tab<P>::NQ, N1 = Tab<P>::N1, NF = 3 * N1;
  Limb B[NQ][NP];                        // eval: phi_i at area point q
  Limb G[NQ][2][NP];                     // projection: w dphi_i/dr, w dphi_i/ds
  Limb S[NF][NP];                        // projection: phi_i at edge points
  Limb Q[NQ][NP];                        // projection of a bed source: phi_i at area points
  Limb E[NF][NP];                        // traces: phi_i at edge points
  int eB, eP, eE;                        // biased exponents of eval, projection, traces
  int c0;                                // phi_0 has one value at all area points (on the edges it has)
  double r[NQ], s[NQ], B0[NQ];           // area points, phi_0 there
  double phi0;                           // phi_0 (area point 0)
};

// ---- shared memory of a block ----------------------------------------------
// rows of kPitch doubles: g of variable n at point q in row q N + n, h in row
// (NQ + q) N + n; the area value of (n, q) waits in its g row; with a bed the
// sources of variables 1, 2 in rows 2 NQ N + 2 q + (n - 1); the new traces of
// (n, edge point i) in row i N + n, rows of the same thread's own g and h
template <class Eq, int P>
struct Shape {
  static constexpr int N = Eq::N, NP = Tab<P>::NP, NQ = Tab<P>::NQ, N1 = Tab<P>::N1, NF = 3 * N1;
  static_assert(NF <= 2 * NQ, "the traces of a variable fit its g and h rows");
  static constexpr int kRows = 2 * NQ * N + (Eq::kBathymetry ? 2 * NQ : 0);
  static constexpr int kThreads = 32 * N;
};

// a / b < c / d, where the cross products do not tell
static __device__ __noinline__ bool smaller_quotient(double a, double b, double c, double d) {
  return a / b < c / d;
}

// the trace of an element that has its mean alone, as the contraction rounds it
static __device__ __noinline__ double mean_trace(double c0, Limb E0, int eE) {
  const Row row = make_row(abs_hi(c0));
  int h, l;
  to_limbs(c0, row, h, l);
  Sum s;
  zero(s);
  mac(s, h, l, E0);
  double v = finish(s, base_exp(row, eE));
  if (row.odd()) fix(&v, 1, 1, row);
  return v;
}

// barrier of the block's N warps
template <int N>
__device__ __forceinline__ void block_sync() {
  if constexpr (N == 1) __syncwarp();
  else __syncthreads();
}
template <int N>
__device__ __forceinline__ bool block_or(bool b) {
  if constexpr (N == 1) return __any_sync(0xffffffffu, b);
  else return __syncthreads_or(b);
}

// ---------------------------------------------------------------------------
// From the new coefficients c of the thread's variable (element e, live or a
// clamped copy) to the traces in T: the trace contraction, the limiter (LIM:
// limit_tr_body's rules with the means from mean[n * mstride + .]), the
// positivity rule (check) and the store (STORE; without it the limiter
// alone).  `out` holds c already; what the limiter or the rule changes is
// written to it.  All threads of the block.
template <class Eq, int P, bool LIM, bool STORE = true>
__device__ __forceinline__ void traces_out(const FxTab<P> &tab, const EqP &q,
                                           const double (&c)[Tab<P>::NP], double *out,
                                           double *T, const int *__restrict__ nbr,
                                           const double *mean, size_t mstride, bool check, int K,
                                           int Kp, int e0, int lane, int n, double *st, int *flag) {
  using S = Shape<Eq, P>;
  constexpr int N = S::N, NP = S::NP, NF = S::NF;
  const int e = e0 + lane;
  const bool live = e < K;
  double *outn = out + (size_t)(n * NP) * Kp + e;
  int nb[3] = {0, 0, 0};
  double cn[3] = {0, 0, 0};
  if constexpr (LIM) {  // the neighbours' means, read ahead of the traces
    const int ec = live ? e : K - 1;
#pragma unroll
    for (int f = 0; f < 3; f++) nb[f] = nbr[(size_t)f * Kp + ec];
#pragma unroll
    for (int f = 0; f < 3; f++) cn[f] = mean[(size_t)n * mstride + nb[f]];
  }
  {
    int mx = 0;
#pragma unroll
    for (int i = 0; i < NP; i++) mx = max(mx, abs_hi(c[i]));
    const Row row = make_row(mx);
    int xh[NP], xl[NP];
#pragma unroll
    for (int i = 0; i < NP; i++) to_limbs(c[i], row, xh[i], xl[i]);
    long long kmax = (long long)0x8000000000000000ull, kmin = 0x7FFFFFFFFFFFFFFFll;
    const int base = base_exp(row, tab.eE);
    const bool odd = row.odd();
    Sum s0;  // the constant mode's part, the same at every point
    zero(s0);
    mac(s0, xh[0], xl[0], tab.E[0][0]);
#pragma unroll
    for (int k = 0; k < NF; k++) {
      Sum s = s0;
#pragma unroll
      for (int i = 1; i < NP; i++) mac(s, xh[i], xl[i], tab.E[k][i]);
      const double v = finish(s, base);
      if constexpr (STORE) st[(k * N + n) * kPitch + lane] = v;
      if constexpr (LIM) {
        const long long kk = order_key(v);
        kmax = max(kmax, kk);
        kmin = min(kmin, kk);
      }
    }
    if (row.odd()) {
      if constexpr (!STORE) {  // scaling by a power of two keeps the order
        double v[2] = {from_order_key(kmax), from_order_key(kmin)};
        fix(v, 1, 2, row);
        kmax = order_key(v[0]);
        kmin = order_key(v[1]);
      } else {
        fix(&st[n * kPitch + lane], N * kPitch, NF, row);
      }
      if constexpr (LIM && STORE) {
        kmax = (long long)0x8000000000000000ull;
        kmin = 0x7FFFFFFFFFFFFFFFll;
#pragma unroll 1
        for (int k = 0; k < NF; k++) {
          const long long kk = order_key(st[(k * N + n) * kPitch + lane]);
          kmax = max(kmax, kk);
          kmin = min(kmin, kk);
        }
      }
      if (LIM && row.m == 0x7FF) {
        // as FP64 traces have it: a NaN limits nothing and stays, infinities beside
        // a finite mean are overshoots like any other
        bool inf = live;
#pragma unroll 1
        for (int i = 0; i < NP && live; i++) {
          const double v = outn[(size_t)i * Kp];
          inf &= i == 0 ? abs_hi(v) < 0x7FF00000 : v == v;
        }
        const double top = __hiloint2double(inf ? 0x7FF00000 : (int)0xFFF00000, 0);
        kmax = order_key(top);
        kmin = order_key(-top);
      }
    }
    if constexpr (LIM) {
      // products reused as addends are rounded explicitly, as in limit_tr_body
      const double Uc = __dmul_rn(c[0], tab.phi0);
      double Umin, Umax;
      mean_bounds(c[0], cn[0], cn[1], cn[2], tab.phi0, Umin, Umax);
      // lo, hi >= +0, so a positive up or dn exceeds them exactly when its
      // bits, as integers, do (negative ones and -0 are below every +0)
      const double up = from_order_key(kmax) - Uc, dn = Uc - from_order_key(kmin);
      const double lo = Uc - Umin, hi = Umax - Uc;
      const long long lob = __double_as_longlong(lo), hib = __double_as_longlong(hi);
      const bool above = __double_as_longlong(up) > lob, below = __double_as_longlong(dn) > hib;
      if (above || below) {
        // alpha = min(lo / up, hi / dn) over the bounds passed, as IEEE division
        // rounds it: the smaller quotient by cross products, then one division
        bool low = above;
        if (above && below) {
          const double pl = lo * dn, ph = hi * up;
          const long long d = __double_as_longlong(pl) - __double_as_longlong(ph);
          low = d < 0;
          // within a few units of rounding of each other, or the larger one zero,
          // denormal or infinite: they do not tell
          if (((unsigned long long)(d + 8) <= 16ull ||
               (unsigned)max(__double2hiint(pl), __double2hiint(ph)) - 0x00100000u >= 0x7FE00000u) &&
              (lob | hib) != 0)
            low = smaller_quotient(lo, up, hi, dn);
        }
        // (a collapsed bound, +0 on its bits, without dividing)
        const double num = low ? lo : hi;
        const double al = __double_as_longlong(num) == 0 ? 0.0 : num / (low ? up : dn);
        const double c1 = c[1] * al, c2 = c[2] * al;
        if (live) {
          outn[(size_t)Kp] = c1;
          outn[2 * (size_t)Kp] = c2;
#pragma unroll
          for (int i = 3; i < NP; i++) outn[(size_t)i * Kp] = 0.0;
        }
        if constexpr (!STORE) return;
        // the limited traces, as trace_tile forms them from the limited modes
        const Row lrow = make_row(max(abs_hi(c[0]), max(abs_hi(c1), abs_hi(c2))));
        int h0, l0, h1, l1, h2, l2;
        to_limbs(c[0], lrow, h0, l0);
        to_limbs(c1, lrow, h1, l1);
        to_limbs(c2, lrow, h2, l2);
        Sum s0;
        zero(s0);
        mac(s0, h0, l0, tab.E[0][0]);
        const int lbase = base_exp(lrow, tab.eE);
#pragma unroll 3
        for (int k = 0; k < NF; k++) {
          Sum s = s0;
          mac(s, h1, l1, tab.E[k][1]);
          mac(s, h2, l2, tab.E[k][2]);
          st[(k * N + n) * kPitch + lane] = finish(s, lbase);
        }
        if (lrow.odd()) fix(&st[n * kPitch + lane], N * kPitch, NF, lrow);
      }
    }
  }
  if constexpr (!STORE) return;
  block_sync<N>();
  // ---- positivity of the traces: the warps share the points out ----
  if (check) {
    bool bad = false;
#pragma unroll 1
    for (int k = n; k < NF; k += N) {
      double u[N];
#pragma unroll
      for (int v = 0; v < N; v++) u[v] = st[(k * N + v) * kPitch + lane];
      bad |= !Eq::physical(q, u);
    }
    if (block_or<N>(bad)) {
      if (bad) flag[lane] = 1;
      block_sync<N>();
      if (flag[lane]) {  // flatten: higher modes to zero, traces to the mean
        const double a0 = mean_trace(c[0], tab.E[0][0], tab.eE);
#pragma unroll 1
        for (int k = 0; k < NF; k++) st[(k * N + n) * kPitch + lane] = a0;
        if (live)
#pragma unroll
          for (int i = 1; i < NP; i++) outn[(size_t)i * Kp] = 0.0;
      }
      block_sync<N>();
    }
  }
  pdl_end();
  // ---- T: each warp stores whole elements, NF N contiguous doubles ----
  constexpr int C = NF * N;
#pragma unroll 2
  for (int el = n; el < kTile; el += N) {
    if (e0 + el >= K) break;
    double *Te = T + (size_t)(e0 + el) * C;
#pragma unroll
    for (int r = 0; r < C; r += 32)
      if (r + lane < C) Te[r + lane] = st[(r + lane) * kPitch + el];
  }
}

// side fluxes of one variable at the element's edge points, -F on a left face,
// +F (mirrored points) on a right face, the sign as a bit flip
template <int N, int N1>
__device__ __forceinline__ void load_F(const double *const (&Fp)[3], const bool (&right)[3],
                                       double (&F)[3 * N1]) {
#pragma unroll
  for (int f = 0; f < 3; f++) {
    const long long sg = right[f] ? 0ll : (long long)0x8000000000000000ull;
#pragma unroll
    for (int j = 0; j < N1; j++)
      F[f * N1 + j] = __longlong_as_double(
          sg ^ __double_as_longlong(Fp[f][(right[f] ? N1 - 1 - j : j) * N]));
  }
}

// ---------------------------------------------------------------------------
// The element stage (element_body's inputs, outputs and rules) of the tile of
// 32 elements from e0.  MODE 0: no traces; 1: the traces of the output into
// T, with the positivity rule where a.check is set; 2: the same with the
// limiter (mode 0 of the output is the stored mean a.M); 3: as 1, and the sum of
// RK4's increments beside the output, a.acc = a.acc0 + a.ck dt L(us) (a.acc0 null:
// zero).  MODE 0 with a.acc0, RK4's last stage: out = un + (a.acc0 + cc dt L(us)),
// one rounding of the state for the four increments.
template <class Eq, int P, int MODE>
__device__ __forceinline__ void element_tile(const FxTab<P> &tab, const EqP &q, const ElemArgs &a,
                                             int e0, double *st, int *mxs, int *flag) {
  using S = Shape<Eq, P>;
  constexpr int N = S::N, NP = S::NP, NQ = S::NQ, N1 = S::N1, NF = S::NF;
  const int lane = threadIdx.x & 31, n = N == 1 ? 0 : (int)(threadIdx.x >> 5);
  const int K = a.K;
  const size_t Kp = a.Kp;
  const int e = e0 + lane, ec = e < K ? e : K - 1;
  const bool live = e < K;
  const double *usn = a.us + (size_t)(n * NP) * Kp + ec;
  if (n == 0) flag[lane] = flag[32 + lane] = 0;

  // ---- area values of the thread's variable ----
  {
    double c[NP];
#pragma unroll
    for (int i = 0; i < NP; i++) c[i] = usn[(size_t)i * Kp];
    int mx = 0;
#pragma unroll
    for (int i = 0; i < NP; i++) mx = max(mx, abs_hi(c[i]));
    const Row row = make_row(mx);
    int xh[NP], xl[NP];
#pragma unroll
    for (int i = 0; i < NP; i++) to_limbs(c[i], row, xh[i], xl[i]);
    const int base = base_exp(row, tab.eB);
    Sum s0;  // the constant mode's part, the same at every point
    zero(s0);
    mac(s0, xh[0], xl[0], tab.B[0][0]);
    const bool c0 = tab.c0;
#pragma unroll
    for (int k = 0; k < NQ; k++) {
      Sum s = s0;
      if (!c0) {
        zero(s);
        mac(s, xh[0], xl[0], tab.B[k][0]);
      }
#pragma unroll
      for (int i = 1; i < NP; i++) mac(s, xh[i], xl[i], tab.B[k][i]);
      st[(k * N + n) * kPitch + lane] = finish(s, base);
    }
    if (row.odd()) fix(&st[n * kPitch + lane], N * kPitch, NQ, row);
  }
  // where the side fluxes of the thread's variable lie; read after the fluxes
  const double *Fp[3];
  bool right[3];
#pragma unroll
  for (int f = 0; f < 3; f++) {
    const int sd = a.esd[(size_t)f * Kp + ec];
    right[f] = sd & 1;
    Fp[f] = a.Fh + (size_t)(sd >> 1) * (N1 * N) + n;
  }
#pragma unroll
  for (int f = 0; f < 3; f++) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(Fp[f]));
    if (N1 * N > 16) asm volatile("prefetch.global.L1 [%0];" ::"l"(Fp[f] + (N1 - 1) * N));
  }
  block_sync<N>();

  // ---- fluxes folded with the metric; the warps share the points out ----
  const double *geo = a.geo;
  const bool has_b = Eq::kBathymetry && a.bslope;
  bool badv = false;
  {
    const double xr = geo[ec], yr = geo[Kp + ec], xs = geo[2 * Kp + ec], ys = geo[3 * Kp + ec];
    double x1 = 0.0, y1 = 0.0;
    if constexpr (Eq::kField) {
      if (q.field) {
        x1 = a.vtx[ec];
        y1 = a.vtx[Kp + ec];
      }
    }
    int mx[N];
    auto point = [&](int k, const double (&u)[N]) {
      double g[N], h[N];
      if constexpr (Eq::kField) {
        double vx = q.ax, vy = q.ay, fx[N], fy[N];
        if (q.field)
          Eq::velocity(q, fma(xr, tab.r[k], fma(xs, tab.s[k], x1)),
                       fma(yr, tab.r[k], fma(ys, tab.s[k], y1)), vx, vy);
        Eq::flux_at(vx, vy, u, fx, fy);
#pragma unroll
        for (int v = 0; v < N; v++) {
          g[v] = fma(fx[v], ys, -fy[v] * xs);
          h[v] = fma(fy[v], xr, -fx[v] * yr);
        }
      } else {
        folded_flux<Eq>(q, u, xr, yr, xs, ys, g, h);
      }
#pragma unroll
      for (int v = 0; v < N; v++) {
        st[(k * N + v) * kPitch + lane] = g[v];
        st[((NQ + k) * N + v) * kPitch + lane] = h[v];
        mx[v] = max(mx[v], max(abs_hi(g[v]), abs_hi(h[v])));
      }
      if constexpr (Eq::kBathymetry) {
        if (has_b) {  // (0, -g h b_x, -g h b_y) w J: bslope holds w J grad b / w-free factors
          const double gh = -q.g * u[0];
#pragma unroll
          for (int v = 1; v < 3; v++) {
            const double sv = gh * a.bslope[(size_t)((v - 1) * NQ + k) * Kp + ec];
            st[(2 * NQ * N + 2 * k + (v - 1)) * kPitch + lane] = sv;
            mx[v] = max(mx[v], abs_hi(sv));
          }
        }
      }
    };
    bool bad = false;
#pragma unroll
    for (int v = 0; v < N; v++) mx[v] = 0;
#pragma unroll 1
    for (int k = n; k < NQ; k += N) {
      double u[N];
#pragma unroll
      for (int v = 0; v < N; v++) u[v] = st[(k * N + v) * kPitch + lane];
      bad |= !Eq::physical(q, u);
      point(k, u);
    }
#pragma unroll
    for (int v = 0; v < N; v++) mxs[(v * N + n) * kTile + lane] = mx[v];
    if (block_or<N>(bad)) {
      // a non-physical area value: the element's mean replaces it everywhere
      if (bad) flag[32 + lane] = 1;
      block_sync<N>();
      badv = flag[32 + lane] != 0;
      if (badv) {
#pragma unroll
        for (int v = 0; v < N; v++) mx[v] = 0;
#pragma unroll 1
        for (int k = n; k < NQ; k += N) {
          double u[N];
#pragma unroll
          for (int v = 0; v < N; v++) u[v] = a.us[(size_t)(v * NP) * Kp + ec] * tab.B0[k];
          point(k, u);
        }
#pragma unroll
        for (int v = 0; v < N; v++) mxs[(v * N + n) * kTile + lane] = mx[v];
      }
      block_sync<N>();
    }
  }

  // ---- projection of the volume and side fluxes, RK combination ----
  double c[NP];
  {
    double F[NF];
    load_F<N, N1>(Fp, right, F);
    int mx = 0;
#pragma unroll
    for (int w = 0; w < N; w++) mx = max(mx, mxs[(n * N + w) * kTile + lane]);
#pragma unroll
    for (int k = 0; k < NF; k++) mx = max(mx, abs_hi(F[k]));
    const Row row = make_row(mx);
    constexpr int i0 = MODE == 2 ? 1 : 0;  // the limiter's stage takes its mean from a.M
    // the projection over the area points rolled where its code is longest
    // (p = 4: advection 134 -> 112 us, the others within 1 %; shallow water p = 3
    // with its third K block 189 -> 181 us), else unrolled (Maxwell p = 3 144 ->
    // 139, Euler p = 3 2.84 -> 2.79 ms)
    constexpr int kUG = P == 4 || (P == 3 && Eq::kBathymetry) ? 1 : NQ;
    Sum s[NP];
#pragma unroll
    for (int i = 0; i < NP; i++) zero(s[i]);
#pragma unroll
    for (int k = 0; k < NF; k++) {
      int h, l;
      to_limbs(F[k], row, h, l);
#pragma unroll
      for (int i = i0; i < NP; i++) mac(s[i], h, l, tab.S[k][i]);
    }
#pragma unroll kUG
    for (int k = 0; k < NQ; k++) {
      int h, l;
      to_limbs(st[(k * N + n) * kPitch + lane], row, h, l);
#pragma unroll
      for (int i = 1; i < NP; i++) mac(s[i], h, l, tab.G[k][0][i]);  // grad phi_0 = 0
      to_limbs(st[((NQ + k) * N + n) * kPitch + lane], row, h, l);
#pragma unroll
      for (int i = 1; i < NP; i++) mac(s[i], h, l, tab.G[k][1][i]);
      if constexpr (Eq::kBathymetry) {
        if (has_b && n > 0) {
          to_limbs(st[(2 * NQ * N + 2 * k + (n - 1)) * kPitch + lane], row, h, l);
#pragma unroll
          for (int i = 0; i < NP; i++) mac(s[i], h, l, tab.Q[k][i]);
        }
      }
    }
    const int base = base_exp(row, tab.eP);
#pragma unroll
    for (int i = i0; i < NP; i++) c[i] = finish(s[i], base);
    if (row.odd()) {  // through the thread's own g rows, which are free now
#pragma unroll
      for (int i = i0; i < NP; i++) st[(i * N + n) * kPitch + lane] = c[i];
      fix(&st[n * kPitch + lane], N * kPitch, NP, row);
#pragma unroll
      for (int i = i0; i < NP; i++) c[i] = st[(i * N + n) * kPitch + lane];
    }
    const double sc = a.cc * *a.dtp * geo[4 * Kp + ec];
    if constexpr (MODE == 3) {
      const double sk = a.ck * *a.dtp * geo[4 * Kp + ec];
      const double *in = a.acc0 + (size_t)(n * NP) * Kp + ec;
      double r[NP];
#pragma unroll
      for (int i = 0; i < NP; i++) r[i] = a.acc0 ? fma(sk, c[i], in[(size_t)i * Kp]) : sk * c[i];
      if (live)
#pragma unroll
        for (int i = 0; i < NP; i++) a.acc[(size_t)(n * NP + i) * Kp + e] = r[i];
    }
    const double *unn = a.un + (size_t)(n * NP) * Kp + ec;
    double *outn = a.out + (size_t)(n * NP) * Kp + ec;
#pragma unroll
    for (int i = 0; i < NP; i++) {
      double v;
      if (MODE == 2 && i == 0) {
        v = a.M[(size_t)n * Kp + ec];
      } else if (MODE == 0 && a.acc0) {
        v = unn[(size_t)i * Kp] + fma(sc, c[i], a.acc0[(size_t)(n * NP + i) * Kp + ec]);
      } else {
        const double cin = (badv && i > 0) ? 0.0 : usn[(size_t)i * Kp];
        v = fma(sc, c[i], a.unit_cb ? cin : a.cb * cin);
        if (a.has_un) v = fma(a.ca, unn[(size_t)i * Kp], v);
      }
      c[i] = v;
    }
    if (live) {
#pragma unroll
      for (int i = 0; i < NP; i++) outn[(size_t)i * Kp] = c[i];
      if (badv && a.us != a.out) {
        double *w = a.us + (size_t)(n * NP) * Kp + e;
#pragma unroll
        for (int i = 1; i < NP; i++) w[(size_t)i * Kp] = 0.0;
      }
    }
  }
  if constexpr (MODE > 0)
    traces_out<Eq, P, MODE == 2>(tab, q, c, a.out, a.T, a.nbr, a.M, Kp, MODE == 2 || a.check, K,
                                 a.Kp, e0, lane, n, st, flag);
}

// Blocks per SM, which set the registers: warps in different phases fill both
// pipes, until spills cost more.  Measured (Euler p = 3, 2.1M triangles, ms at
// 4 to 8 blocks): 3.59, 2.93, 2.79, 2.74, 2.78; Euler p = 4 (5 to 8): 1.24,
// 1.21, 1.27, 1.39; shallow water p = 2, 131k (us at 5 to 12): 93 88 86 86 81 82
// 80; Maxwell p = 3 (5 to 12): 156 150 138 139 135 135 139; advection p = 3, 131k and
// 35k (20, 22, 24, 28): 77 71 73 70 and 31.8 31.2 31.6 32.8.
template <class Eq, int P>
constexpr int min_blocks() {
  if (Eq::N == 4) return P <= 2 ? 8 : P == 3 ? 7 : 6;
  if (Eq::N == 3) return P <= 2 ? 12 : P == 4 ? 7 : Eq::kBathymetry ? 8 : 9;
  return P == 1 ? 16 : P == 4 ? 20 : P == 3 ? 22 : 24;
}

template <class Eq, int P, int MODE>
__global__ void __launch_bounds__(Shape<Eq, P>::kThreads, min_blocks<Eq, P>())
    k_element_fx(const __grid_constant__ FxTab<P> tab, const __grid_constant__ EqP q,
                 const __grid_constant__ ElemArgs a) {
  using S = Shape<Eq, P>;
  __shared__ double st[S::kRows * kPitch];
  __shared__ int mxs[S::N * S::N * kTile];
  __shared__ int flag[2 * kTile];
  pdl_begin();
  element_tile<Eq, P, MODE>(tab, q, a, blockIdx.x * kTile, st, mxs, flag);
}

// Edge traces of a state (trace_body's rules), with the same contraction as
// the stage: bit for bit the traces k_element_fx writes for the same
// coefficients.  LIM: the state is limited first, with its own means as the
// neighbours' bounds (the limiter and the positivity rule change no mean, so
// the elements need no order); STORE = false: limited only (k_limit), no
// traces.  Limiting and tracing in one pass at the start of a run: Euler p =
// 3, 2.1M triangles, k_limit + k_trace_fx 2.89 + 0.44 ms -> 0.66.
template <class Eq, int P, bool LIM, bool STORE>
__device__ __forceinline__ void trace_tile(const FxTab<P> &tab, const EqP &q, double *u,
                                           double *T, const int *__restrict__ nbr,
                                           int K, int Kp, int e0, double *st, int *flag) {
  constexpr int N = Eq::N, NP = Tab<P>::NP;
  const int lane = threadIdx.x & 31, n = N == 1 ? 0 : (int)(threadIdx.x >> 5);
  const int ec = min(e0 + lane, K - 1);
  if (STORE && n == 0) flag[lane] = 0;
  double c[NP];
#pragma unroll
  for (int i = 0; i < NP; i++) c[i] = u[(size_t)(n * NP + i) * Kp + ec];
  traces_out<Eq, P, LIM, STORE>(tab, q, c, u, T, nbr, u, (size_t)NP * Kp, true, K, Kp, e0, lane,
                                n, st, flag);
}

template <class Eq, int P, bool LIM, bool STORE>
__global__ void __launch_bounds__(Shape<Eq, P>::kThreads)
    k_trace_fx(const __grid_constant__ FxTab<P> tab, const __grid_constant__ EqP q, double *u,
               double *T, const int *__restrict__ nbr, int K, int Kp) {
  using S = Shape<Eq, P>;
  __shared__ double st[STORE ? S::NF * S::N * kPitch : 1];
  __shared__ int flag[kTile];
  pdl_begin();
  trace_tile<Eq, P, LIM, STORE>(tab, q, u, T, nbr, K, Kp, blockIdx.x * kTile, st, flag);
}

// ---- batched ensembles: the blocks [b_lo, b_lo + gridDim.x / sub) of the
// problems of one order, each block of the map `sub` tiles of 32 elements ----
__device__ __forceinline__ int batch_tile(const int *__restrict__ blk2prob,
                                          const int *__restrict__ blk0, int b_lo, int sub,
                                          int &pi) {
  const int b = b_lo + (int)blockIdx.x / sub;
  pi = blk2prob[b];
  return ((b - blk0[pi]) * sub + (int)blockIdx.x % sub) * kTile;
}

template <class Eq, int P>
__global__ void __launch_bounds__(Shape<Eq, P>::kThreads, min_blocks<Eq, P>())
    k_element_batch_fx(const __grid_constant__ FxTab<P> tab, const BatchProb *__restrict__ probs,
                       const int *__restrict__ blk2prob, const int *__restrict__ blk0, int b_lo,
                       int sub, int stage, int check) {
  using S = Shape<Eq, P>;
  __shared__ double st[S::kRows * kPitch];
  __shared__ int mxs[S::N * S::N * kTile];
  __shared__ int flag[2 * kTile];
  int pi;
  const int e0 = batch_tile(blk2prob, blk0, b_lo, sub, pi);
  const BatchProb &pr = probs[pi];
  if (e0 >= pr.K) return;
  const ElemArgs a = batch_elem_args(pr, stage, check);
  element_tile<Eq, P, 1>(tab, pr.q, a, e0, st, mxs, flag);
}

// the traces of the states U, and with LIM the limiter of a stage's output first
template <class Eq, int P, bool LIM>
__global__ void __launch_bounds__(Shape<Eq, P>::kThreads)
    k_trace_batch_fx(const __grid_constant__ FxTab<P> tab, const BatchProb *__restrict__ probs,
                     const int *__restrict__ blk2prob, const int *__restrict__ blk0, int b_lo,
                     int sub, int stage) {
  using S = Shape<Eq, P>;
  __shared__ double st[S::NF * S::N * kPitch];
  __shared__ int flag[kTile];
  int pi;
  const int e0 = batch_tile(blk2prob, blk0, b_lo, sub, pi);
  const BatchProb &pr = probs[pi];
  if (e0 >= pr.K) return;
  trace_tile<Eq, P, LIM, true>(tab, pr.q, LIM && stage < 2 ? pr.W : pr.U, pr.T, pr.nbr, pr.K,
                               pr.Kp, e0, st, flag);
}

}  // namespace fx
}  // namespace dg
