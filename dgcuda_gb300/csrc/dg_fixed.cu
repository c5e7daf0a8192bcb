// dg_fixed.cu -- host side of the fixed-point contractions: the limb tables
// of the element stage's basis tables.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "dg_fixed.cuh"
#include "dg_internal.h"

namespace dg {
namespace fx {
namespace {

int host_bexp(double x) {
  unsigned long long b;
  std::memcpy(&b, &x, 8);
  return (int)((b >> 52) & 0x7FF);
}

// t in units of 2^(M - 1078): a signed integer, |T| <= 2^58, as h 2^28 + l with l
// in [-2^27, 2^27)
Limb limb(double t, int M) {
  const long long T = std::llrint(std::ldexp(t, 1078 - M));
  Limb r;
  r.h = (int)((T + (1ll << (kLow - 1))) >> kLow);
  r.l = (int)(T - ((long long)r.h << kLow));
  return r;
}

// The unit of the projection's tables, 2^(M - 1078): the smallest with every |T|
// <= 2^58 and the |T| that meet in one sum adding up to 2^61 at most, so that sums of
// at most 63 products with inputs below 2^57 stay in 64 bits.  For the library's
// tables two bits below the largest entry's exponent, the unit of the other
// tables: the product that the sums leave out, l tl, is what their error was made
// of (the header of dg_fixed.cuh has the figures).
struct Unit {
  double top = 0, sum = 0;  // the largest |t|, the largest sum of |t|
  template <class... D>
  void add(D... t) {
    ((top = std::max(top, std::fabs(t)), part += std::fabs(t)), ...);
  }
  void end() {
    sum = std::max(sum, part);
    part = 0;
  }
  int exponent() const {
    int k = 0;
    if (sum > 0) std::frexp(sum, &k);  // sum <= 2^k
    return std::max(1, std::max(host_bexp(top) - 2, k + 1017));
  }

 private:
  double part = 0;
};

template <int P>
void build(const Tab<P> &t, FxTab<P> *o) {
  constexpr int NP = Tab<P>::NP, NQ = Tab<P>::NQ, N1 = Tab<P>::N1, NF = 3 * N1;
  int mB = 1, mE = 1;
  for (int q = 0; q < NQ; q++)
    for (int i = 0; i < NP; i++) mB = std::max(mB, host_bexp(t.B[q][i]));
  for (int k = 0; k < NF; k++)
    for (int i = 0; i < NP; i++) mE = std::max(mE, host_bexp(t.E[k / N1][k % N1][i]));
  Unit u;
  for (int i = 0; i < NP; i++, u.end()) {  // to the modes: edge points, slopes, a bed
    for (int k = 0; k < NF; k++) u.add(t.E[k / N1][k % N1][i]);
    for (int q = 0; q < NQ; q++) u.add(t.GR[q][i], t.GS[q][i], t.B[q][i]);
  }
  for (int q = 0; q < NQ; q++) {  // the adjoint's projections on the slopes
    for (int i = 0; i < NP; i++) u.add(t.GR[q][i]);
    u.end();
    for (int i = 0; i < NP; i++) u.add(t.GS[q][i]);
    u.end();
  }
  o->eB = mB;
  o->eP = u.exponent();
  o->eE = mE;
  o->c0 = 1;
  for (int q = 1; q < NQ; q++)
    if (t.B[q][0] != t.B[0][0]) o->c0 = 0;
  for (int q = 0; q < NQ; q++) {
    for (int i = 0; i < NP; i++) {
      o->B[q][i] = limb(t.B[q][i], o->eB);
      o->G[q][0][i] = limb(t.GR[q][i], o->eP);
      o->G[q][1][i] = limb(t.GS[q][i], o->eP);
      o->Q[q][i] = limb(t.B[q][i], o->eP);
    }
    o->r[q] = t.r[q];
    o->s[q] = t.s[q];
    o->B0[q] = t.B[q][0];
  }
  for (int k = 0; k < NF; k++) {
    const double *E = t.E[k / N1][k % N1];
    for (int i = 0; i < NP; i++) {
      o->S[k][i] = limb(E[i], o->eP);
      o->E[k][i] = limb(E[i], o->eE);
    }
  }
  o->phi0 = t.B[0][0];
}

}  // namespace
}  // namespace fx

size_t fx_tab_bytes(int p) {
  switch (p) {
    case 1: return sizeof(fx::FxTab<1>);
    case 2: return sizeof(fx::FxTab<2>);
    case 3: return sizeof(fx::FxTab<3>);
    case 4: return sizeof(fx::FxTab<4>);
  }
  return 0;
}

void build_fx_tab(int p, const void *tabimg, void *out) {
  switch (p) {
    case 1: fx::build(*static_cast<const Tab<1> *>(tabimg), static_cast<fx::FxTab<1> *>(out)); break;
    case 2: fx::build(*static_cast<const Tab<2> *>(tabimg), static_cast<fx::FxTab<2> *>(out)); break;
    case 3: fx::build(*static_cast<const Tab<3> *>(tabimg), static_cast<fx::FxTab<3> *>(out)); break;
    case 4: fx::build(*static_cast<const Tab<4> *>(tabimg), static_cast<fx::FxTab<4> *>(out)); break;
  }
}

}  // namespace dg

// the limb tables of order p (1..4) built from the library's basis tables, as
// fx::FxTab<p> holds them
extern "C" dg_status dg_fx_table_image(int p, void *out, size_t bytes) {
  if (p < 1 || p > 4 || !out) return dg::fail(DG_BAD_ARG, "order must be 1..4");
  if (bytes < dg::fx_tab_bytes(p)) return dg::fail(DG_BAD_ARG, "buffer too small");
  std::vector<char> tab(dg::tab_bytes(p));
  dg::build_tab(p, DG_TABLES[p], tab.data());
  dg::build_fx_tab(p, tab.data(), out);
  return DG_OK;
}
