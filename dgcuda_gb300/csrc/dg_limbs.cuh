// dg_limbs.cuh -- doubles as 57-bit fixed point in two limbs, X = h 2^28 + l,
// and sums of their products in integer multiply-adds: the arithmetic of the
// fixed-point element stage (dg_fixed.cuh, which says why) and of the face
// kernels' momentum sums.
#pragma once
#include <cuda_runtime.h>

#ifdef __CUDACC__
namespace dg {
namespace fx {

constexpr int kLow = 28;                 // bits of the low limb

struct Limb {
  int h, l;
};

// ---- rows -----------------------------------------------------------------
// a row whose largest entry has biased exponent m.  A row of zeros (or
// denormals only) takes an exponent that shifts every entry out: all its
// limbs and sums are zero.  Other rows outside [100, 1900], where a result
// could leave the normal range, and rows with an infinity or a NaN are
// odd(): finish() forms their sums as if m were 1023 and fix() scales them, to NaN
// in the latter.  Below 2^-967 a zero or a denormal counts as 2^-1023: an error
// under the smallest normal number, which lifting such rows first would take away
// at 2 to 9 % of the element stage's time
struct Row {
  int m;
  __device__ __forceinline__ bool odd() const { return (unsigned)(m - 100) > 1800u; }
};
__device__ __forceinline__ Row make_row(int maxhi) {
  Row r;
  r.m = maxhi >> 20;
  if (r.m == 0) r.m = 1023;
  return r;
}
__device__ __forceinline__ int abs_hi(double x) { return __double2hiint(x) & 0x7FFFFFFF; }

// x on row r: the two limbs of a 57-bit integer, the low one balanced, l in [-2^27,
// 2^27].  Truncation and a low limb of x's sign would both have a mean, which
// repeats from stage to stage: with 56 bits and l in [0, 2^28) the error of a run
// of 20 steps was 2.4 times FP64's at p = 4 (advection, contractions alone), with these
// 0.84 times, p = 1 to 3 0.58, 0.52, 0.52
__device__ __forceinline__ void to_limbs(double x, const Row &r, int &h, int &l) {
  const int hi = __double2hiint(x);
  const unsigned lo = (unsigned)__double2loint(x);
  const int e = (hi >> 20) & 0x7FF;
  const unsigned mh = ((unsigned)hi & 0xFFFFFu) | 0x100000u;
  unsigned long long X = (((unsigned long long)mh << 32) | lo) << 4;
  X >>= min(r.m - e, 63);
  const int sg = (hi >> 31) | 1;
  h = (int)((X + (1u << (kLow - 1))) >> kLow) * sg;
  l = ((int)((unsigned)X << (32 - kLow)) >> (32 - kLow)) * sg;
}

struct Sum {
  long long H, M;
};
__device__ __forceinline__ void zero(Sum &s) {
  s.H = 0;
  s.M = 1ll << (kLow - 1);  // the rounding of M >> 28
}
__device__ __forceinline__ void mac(Sum &s, int h, int l, const Limb &t) {
  s.H += (long long)h * t.h;
  s.M += (long long)h * t.l;
  s.M += (long long)l * t.h;
}

// the results of an odd row, `count` doubles `step` apart, formed with exponent
// 1023 in place of the row's
static __device__ __noinline__ void fix(double *v, int step, int count, Row r) {
  for (int k = 0; k < count; k++, v += step)
    *v = r.m == 0x7FF ? __longlong_as_double(0x7FF8000000000000ll) : ldexp(*v, r.m - 1023);
}

// the exponent finish() attaches for results of row r and a table of biased
// exponent M
__device__ __forceinline__ int base_exp(Row r, int M) {
  return (r.odd() ? 1023 : r.m) + M - 1016;
}
// the sum as a double, S 2^(base - 1085) with S = H + (M >> 28): magnitude
// (of a negative S as |S| - 1: half an ulp of a result of full scale over 8),
// normalised so that 63 bits are used, rounded to 53 (half away from zero),
// exponent and sign attached
__device__ __forceinline__ double finish(const Sum &s, int base) {
  const long long S = s.H + (s.M >> kLow);
  const int sg = (int)(S >> 63);
  const unsigned ah = (unsigned)((int)(S >> 32) ^ sg), al = (unsigned)((int)S ^ sg);
  const bool small = ah == 0;  // below 2^32: normalise a 2^31 instead
  const unsigned top = small ? al >> 1 : ah, low = small ? al << 31 : al;
  int b;  // index of the leading bit of top < 2^31, -1 for top = 0
  asm("bfind.u32 %0, %1;" : "=r"(b) : "r"(top));
  const unsigned nh = __funnelshift_l(low, top, 30 - b), nl = low << ((30 - b) & 31);
  const unsigned long long f = ((((unsigned long long)nh << 32) | nl) + 0x200ull) >> 10;
  unsigned hi = (unsigned)(f >> 32) + ((unsigned)((small ? base - 62 : base - 31) + b) << 20);
  if ((ah | al) == 0) hi = 0;  // f is 0 then
  return __hiloint2double((int)(hi | ((unsigned)sg & 0x80000000u)), (int)(unsigned)f);
}

// ---- sums of two products of variables (face kernels) -----------------------
// a double on a row of its own, so that it keeps all its bits beside a much
// larger one: x = (h 2^28 + l) 2^(m - 1078), t the upper half of l.  m: 1023 for a
// zero, 0 for a denormal, which in_range() then leaves to FP64
struct Num {
  int m, h, l, t;
};
__device__ __forceinline__ Num make_num(double x) {
  const int hi = __double2hiint(x);
  const unsigned lo = (unsigned)__double2loint(x);
  const unsigned mh = ((unsigned)hi & 0xFFFFFu) | 0x100000u;
  const int sg = (hi >> 31) | 1;
  Num n;
  n.m = (hi >> 20) & 0x7FF;
  n.h = (int)((mh << 7) | (lo >> 25)) * sg;
  n.l = (int)((lo << 3) & ((1u << kLow) - 1)) * sg;
  if (n.m == 0) {
    n.h = n.l = 0;
    if (((hi & 0x7FFFFFFF) | (int)lo) == 0) n.m = 1023;
  }
  n.t = n.l >> (kLow / 2);
  return n;
}
// whether the products of numbers with exponents in [lo, hi] stay in the normal
// range, and the sums of two of them (an infinity or a NaN has 2047)
__device__ __forceinline__ bool in_range(int lo, int hi) { return lo >= 620 && hi < 1400; }
// x y in units of 2^(x.m + y.m - 2156 + 51), below 2^61
__device__ __forceinline__ long long prod(const Num &x, const Num &y) {
  long long M = 1ll << 22;
  M += (long long)x.h * y.l;
  M += (long long)x.l * y.h;
  M += (long long)x.t * y.t;  // l l' >> 28
  return ((long long)x.h * y.h << 5) + (M >> (kLow - 5));
}
__device__ __forceinline__ long long square(const Num &x) {
  long long M = 1ll << 22;
  M += (long long)x.h * (2 * x.l);
  M += (long long)x.t * x.t;
  return ((long long)x.h * x.h << 5) + (M >> (kLow - 5));
}
// the sum of the products p and q, whose numbers' exponents add up to ep and eq,
// times 2^k: the smaller scale is shifted to the larger one (a zero product,
// whose exponents may be stand-ins, takes the other's)
__device__ __forceinline__ double sum2(long long p, int ep, long long q, int eq, int k = 0) {
  if (p == 0) ep = eq;
  if (q == 0) eq = ep;
  const int d = ep - eq;
  Sum s;
  s.H = d >= 0 ? p + (q >> min(d, 63)) : q + (p >> min(-d, 63));
  s.M = 0;
  return finish(s, max(ep, eq) - 1020 + k);
}
// xa ya + xb yb
__device__ __forceinline__ double dot(const Num &xa, const Num &ya, const Num &xb, const Num &yb) {
  return sum2(prod(xa, ya), xa.m + ya.m, prod(xb, yb), xb.m + yb.m);
}
// -(a^2 + b^2) / 2
__device__ __forceinline__ double neg_half_square(const Num &a, const Num &b) {
  const double v = sum2(square(a), 2 * a.m, square(b), 2 * b.m, -1);
  return __hiloint2double(__double2hiint(v) ^ (int)0x80000000, __double2loint(v));
}

}  // namespace fx
}  // namespace dg
#endif
