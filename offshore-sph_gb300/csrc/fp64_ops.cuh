// fp64_ops.cuh -- reciprocal, square root and exponential in few FP64
// operations, for the kernels that the FP64 pipe bounds.
#pragma once

#include "sph_internal.cuh"

namespace sph {

// ---------------------------------------------------------------------------
// FP64 building blocks
// ---------------------------------------------------------------------------
// hardware estimates of 1/x and 1/sqrt(x) (normal x): the result's upper word
__device__ __forceinline__ double rcp_est(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
__device__ __forceinline__ double rsqrt_est(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
// 1/x: y (1 + e + e^2), e = 1 - x y; the estimate's error cubed is far below
// an ulp
__device__ __forceinline__ double rcp64(double x) {
  const double y = rcp_est(x);
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
// r = sqrt(x) and ir = 1/sqrt(x): y (1 + e/2 + 3/8 e^2), e = 1 - x y^2
__device__ __forceinline__ void sqrt_rsqrt64(double x, double &r, double &ir) {
  const double y = rsqrt_est(x);
  const double t = x * y;
  const double e = fma(-t, y, 1.0);
  const double c = fma(0.375, e, 0.5) * e;
  r = fma(t, c, t);
  ir = fma(y, c, y);
}

// a <= b for non-negative doubles (false when either is NaN and a is not
// below b's pattern), without an FP64 instruction
__device__ __forceinline__ bool le_bits(double a, double b) {
  return (unsigned long long)__double_as_longlong(a) <= (unsigned long long)__double_as_longlong(b);
}

// exp(-z) for 0 <= z < 16: table lookup and a short polynomial (P. T. P. Tang,
// Table-driven implementation of the exponential function in IEEE
// floating-point arithmetic, ACM TOMS 15, 1989), with 2048 entries so that a
// cubic suffices: z = (n ln 2) / 2048 + s, |s| <= 1.7e-4,
// exp(-z) = 2^(-n / 2048) (1 - s + s^2 / 2 - s^3 / 6) to 4e-17.  The index
// comes from FP32, so the FP64 pipe sees 6 operations.
constexpr int kExpN = 2048;
struct ExpTable {
  double v[kExpN];
};
struct DD {
  double hi, lo;
};
constexpr DD dd_two_prod(double a, double b) {  // Dekker's product
  const double p = a * b;
  const double c1 = 134217729.0 * a, c2 = 134217729.0 * b;
  const double ah = c1 - (c1 - a), bh = c2 - (c2 - b);
  const double al = a - ah, bl = b - bh;
  return {p, ((ah * bh - p) + ah * bl + al * bh) + al * bl};
}
constexpr DD dd_mul(DD a, DD b) {
  const DD p = dd_two_prod(a.hi, b.hi);
  const double l = p.lo + (a.hi * b.lo + a.lo * b.hi);
  const double s = p.hi + l;
  return {s, l - (s - p.hi)};
}
// ln 2 in three parts: the first with its last 20 bits zero, so that n times
// it is exact for n < 2^16
constexpr double kLn2Hi = 0x1.62e42fefp-1, kLn2Lo = 0x1.473de6af278edp-34;
constexpr ExpTable make_exp_table() {
  // c = 2^(-1/2048) = exp(-ln 2 / 2048) as a double-double Taylor sum
  const DD x = {-0x1.62e42fefa39efp-1 / kExpN, -0x1.abc9e3b39803fp-56 / kExpN};
  DD term = {1.0, 0.0}, c = {1.0, 0.0};
  for (int k = 1; k <= 8; k++) {
    term = dd_mul(term, x);
    const DD inv = {1.0 / k, 0.0};
    // term / k with one correction of the quotient
    const DD q0 = dd_mul(term, inv);
    const DD back = dd_mul(q0, DD{(double)k, 0.0});
    const double fix = ((term.hi - back.hi) + (term.lo - back.lo)) / k;
    const double qh = q0.hi + (q0.lo + fix);
    term = DD{qh, (q0.lo + fix) - (qh - q0.hi)};
    const double s = c.hi + term.hi;
    const double err = (c.hi - s) + term.hi;
    const double lo = err + (c.lo + term.lo);
    const double s2 = s + lo;
    c = DD{s2, lo - (s2 - s)};
  }
  ExpTable t = {};
  DD v = {1.0, 0.0};
  for (int i = 0; i < kExpN; i++) {
    t.v[i] = v.hi;
    v = dd_mul(v, c);
  }
  return t;
}
__device__ constexpr ExpTable g_exp_table = make_exp_table();

__device__ __forceinline__ double exp_neg(double z) {
  const float nf = fmaf(d2f_trunc(z), (float)(kExpN / 0.693147180559945309417), 12582912.0f);
  const int n = (int)(__float_as_uint(nf) - 0x4B400000u);
  const double nd = f2d(nf - 12582912.0f);
  double s = fma(nd, -kLn2Hi / kExpN, z);
  s = fma(nd, -kLn2Lo / kExpN, s);
  const double p = fma(s, -1.0 / 6.0, 0.5);
  const double t = fma(s * s, p, -s);
  const double T = __ldg(&g_exp_table.v[n & (kExpN - 1)]);
  const double b = __hiloint2double(__double2hiint(T) - ((n >> 11) << 20), __double2loint(T));
  return fma(b, t, b);
}

}  // namespace sph
