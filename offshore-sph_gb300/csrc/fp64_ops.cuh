// fp64_ops.cuh -- reciprocal, square root and exponential in few FP64
// operations, and the launch constants of the FP64 pair kernels, for the
// kernels that the FP64 pipe bounds.
#pragma once

#include "sph_internal.cuh"

namespace sph {

// ---------------------------------------------------------------------------
// FP64 building blocks
// ---------------------------------------------------------------------------
// One FP64 instruction costs the SM as much issue time as 64 integer or FP32
// ones, so reciprocal and square root run on the integer pipe: a 24-bit FP32
// estimate and one Newton-type step of third order on 64-bit fixed-point
// mantissas,
//   1/x:        y (1 + e + e^2),          e = 1 - x y
//   1/sqrt(x):  y (1 + e/2 + 3/8 e^2),    e = 1 - x y^2
// (the binomial series of (1 - e)^-1 and (1 - e)^-1/2), rounded once to 53
// bits.  The error before that rounding is below 2^-60, so the results are
// within 0.51 ulp.  About 35 and 57 instructions instead of 3 and 6 FP64 ones
// (Halley steps on the hardware's 2^-20 estimates).
static __device__ __noinline__ double rcp64_slow(double x) { return 1.0 / x; }

__device__ __forceinline__ float rcp_est_f(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rsqrt_est_f(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// an estimate y0 in about [0.5, 1] as a fraction of 2^32 (24 bits of it)
__device__ __forceinline__ unsigned int est_q32(float y0) {
  y0 = fminf(fmaxf(y0, 0.5f), 0.99999994f);
  return (__float_as_uint(y0) << 8) | 0x80000000u;
}
// y0 (1 + c) in units of 2^-63 from y0 in units of 2^-32 and c in units of
// 2^-CB, |c| < 2^-20
template <int CB>
__device__ __forceinline__ unsigned long long refine_q63(unsigned int y0, long long c) {
  const unsigned int ys = y0 >> 1;  // y0 in units of 2^-31
  const unsigned long long lo = (unsigned long long)ys * (unsigned int)c;
  const long long s = (long long)(int)ys * (int)(c >> 32) + (long long)(lo >> 32);  // units of 2^(1 - CB)
  return ((unsigned long long)y0 << 31) + (unsigned long long)(s << (64 - CB));
}
// the double with 53-bit integer significand (m rounded to bit `drop`) whose
// leading bit has the biased exponent e
template <int DROP>
__device__ __forceinline__ double pack64(unsigned long long m, int e, unsigned int sign = 0u) {
  const unsigned long long r = (m + (1ull << (DROP - 1))) >> DROP;  // may carry into the exponent
  const unsigned int hi = (unsigned int)(r >> 32) + ((unsigned int)(e - 1) << 20);
  return __hiloint2double((int)(hi | sign), (int)(unsigned int)r);
}

// the product of two 64-bit fractions, within 3 units
__device__ __forceinline__ unsigned long long mul_hi(unsigned long long a, unsigned long long b) {
  const unsigned int a1 = (unsigned int)(a >> 32), a0 = (unsigned int)a;
  const unsigned int b1 = (unsigned int)(b >> 32), b0 = (unsigned int)b;
  return (unsigned long long)a1 * b1 + (((unsigned long long)a1 * b0) >> 32) + (((unsigned long long)a0 * b1) >> 32);
}
// 1 / v for v in [1, 2) in units of 2^-63, in units of 2^-63
__device__ __forceinline__ unsigned long long rcp_q63(unsigned int vh, unsigned int vl) {
  const unsigned int y0 = est_q32(rcp_est_f(__uint_as_float(0x3f800000u | ((vh >> 8) & 0x7fffffu))));
  const unsigned long long p = (unsigned long long)vh * y0 + (((unsigned long long)vl * y0) >> 32);
  const long long e1 = (long long)(0x8000000000000000ull - p);  // 1 - x y, units of 2^-63
  const int eh = (int)(e1 >> 21);
  const long long c = e1 + (long long)(((unsigned long long)((long long)eh * eh)) >> 21);
  return refine_q63<63>(y0, c);
}

__device__ __forceinline__ double rcp64(double x) {
  const unsigned int hi = (unsigned int)__double2hiint(x), lo = (unsigned int)__double2loint(x);
  const unsigned int e = (hi >> 20) & 0x7ffu;
  if (e - 2u > 2042u) return rcp64_slow(x);  // zero, denormal, infinite, NaN, or a denormal result
  const unsigned int mh = (hi & 0xfffffu) | 0x100000u;
  return pack64<10>(rcp_q63(__funnelshift_l(lo, mh, 11), lo << 11), 2045 - (int)e, hi & 0x80000000u);
}

// 1/x in two parts y + yl, 1/x^2 and 1/x^4 for x > 0, each rounded once
static __device__ __noinline__ void rcp_powers_slow(double x, double &y, double &yl, double &y2, double &y4) {
  y = 1.0 / x;
  yl = fma(-y, x, 1.0) * y;
  y2 = y * y;
  y4 = y2 * y2;
}
__device__ __forceinline__ void rcp_powers(double x, double &y, double &yl, double &y2, double &y4) {
  const unsigned int hi = (unsigned int)__double2hiint(x), lo = (unsigned int)__double2loint(x);
  const int e = (int)(hi >> 20) - 1023;
  if ((unsigned int)(e + 250) > 500u) {  // a power out of range, or x not positive
    rcp_powers_slow(x, y, yl, y2, y4);
    return;
  }
  const unsigned int mh = (hi & 0xfffffu) | 0x100000u;
  const unsigned long long a = rcp_q63(__funnelshift_l(lo, mh, 11), lo << 11);  // (2^62, 2^63]
  y = pack64<10>(a, 1022 - e);
  // what that rounded off, -512 to 511 units of 2^(-63 - e): as a float, and its
  // exponent moved (0 becomes about 2^-190 of y)
  const unsigned int f = __float_as_uint((float)(((int)(unsigned int)a << 22) >> 22));
  yl = __hiloint2double((int)((f & 0x80000000u) | (((f & 0x7fffffffu) >> 3) + ((unsigned int)(833 - e) << 20))), 0);
  const unsigned long long b = mul_hi(a, a);  // units of 2^-62
  const int n = __clzll((long long)b);        // 1 to 3
  y2 = pack64<10>(b << (n - 1), 1024 - n - 2 * e);
  const unsigned long long d = mul_hi(b << n, b << n);  // units of 2^(-60 - 2 n), [2^62, 2^64)
  const int m = (int)(d >> 63);
  y4 = pack64<10>(d >> m, 1025 + m - 2 * n - 4 * e);
}

// A positive number v 4^k, v in [1, 4) in units of 2^-62.
struct Quad64 {
  unsigned int vh, vl;
  int k;
};
__device__ __forceinline__ Quad64 quad64(double x) {  // x > 0 normal
  const unsigned int hi = (unsigned int)__double2hiint(x), lo = (unsigned int)__double2loint(x);
  const int ue = (int)(hi >> 20) - 1023;
  const unsigned int odd = (unsigned int)ue & 1u;
  const unsigned int mh = (hi & 0xfffffu) | 0x100000u;
  return {__funnelshift_l(lo, mh, 10u + odd), lo << (10u + odd), ue >> 1};
}

// y = 1 / sqrt(v 4^-k), in [0.5, 1], in units of 2^-63
__device__ __forceinline__ unsigned long long rsqrt_q63(const Quad64 &v) {
  const unsigned int vh = v.vh, vl = v.vl;
  // v in FP32, truncated: its leading bit is bit 31 or 30 of vh
  const unsigned int odd = vh >> 31;
  const float vf = __uint_as_float(((126u + odd) << 23) + (vh >> (7u + odd)));
  const unsigned int y0 = est_q32(rsqrt_est_f(vf));
  const unsigned long long t = (unsigned long long)y0 * y0;  // y^2, units of 2^-64
  const unsigned long long p = mul_hi(((unsigned long long)vh << 32) | vl, t);
  const long long e1 = (long long)(0x4000000000000000ull - p);  // 1 - x y^2, units of 2^-62
  const int eh = (int)(e1 >> 20);
  const unsigned int e2 = (unsigned int)(((unsigned long long)((long long)eh * eh)) >> 22);  // e^2, units of 2^-62
  const long long c = (e1 >> 1) + (long long)((3u * e2) >> 3);
  return refine_q63<62>(y0, c);
}
// sqrt(v 4^-k) in units of 2^-61 from it
__device__ __forceinline__ unsigned long long sqrt_q61(const Quad64 &v, unsigned long long y) {
  return mul_hi(((unsigned long long)v.vh << 32) | v.vl, y);
}
// r = sqrt(v) and ir = 1 / sqrt(v)
__device__ __forceinline__ void sqrt_rsqrt64(const Quad64 &v, double &r, double &ir) {
  const unsigned long long y = rsqrt_q63(v);
  ir = pack64<10>(y, 1022 - v.k);
  r = pack64<9>(sqrt_q61(v, y), 1023 + v.k);
}

// A positive constant m 2^(e - 62), m in [2^62, 2^63).
struct Fix64 {
  unsigned long long m;
  int e;
};
inline Fix64 fix64(double x, double lo = 0.0) {  // x + lo, lo below x's last bit
  int e = 0;
  const double f = frexp(x, &e);  // [0.5, 1)
  return {(unsigned long long)ldexp(f, 63) + (unsigned long long)(long long)ldexp(lo, 63 - e), e - 1};
}
// (a + al) / (b + bl) to 63 bits: the quotient and its remainder's
inline Fix64 fix64_quot(double a, double al, double b, double bl) {
  const double q = a / b;
  return fix64(q, (fma(-q, b, a) + (al - q * bl)) / b);
}

// exp(-z) for 0 <= z < 11: table lookup and a short polynomial (P. T. P. Tang,
// Table-driven implementation of the exponential function in IEEE
// floating-point arithmetic, ACM TOMS 15, 1989), in 64-bit fixed point: z / ln 2
// = n / 2048 + t, |t| <= 1/4096, x = |t| ln 2,
// exp(-z) = 2^(-n / 2048) (1 -+ (x + x^3 / 6) + x^2 / 2 + x^4 / 24), the sum's
// error below 2^-57.
constexpr int kExpN = 2048;
struct ExpTable {
  unsigned long long v[kExpN];  // 2^(-i / 2048) in units of 2^-62
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
    t.v[i] = (unsigned long long)(v.hi * 0x1p62) + (unsigned long long)(long long)(v.lo * 0x1p62);
    v = dd_mul(v, c);
  }
  return t;
}
__device__ constexpr ExpTable g_exp_table = make_exp_table();

// exp(-v c / log2(e)), i.e. 2^(-v c), for v c < 16: a squared distance and
// log2(e) / h^2
__device__ __forceinline__ double exp2_neg(const Quad64 &v, const Fix64 &c) {
  const unsigned long long p = mul_hi(((unsigned long long)v.vh << 32) | v.vl, c.m << 1);  // units of 2^-61
  const unsigned long long u = p >> min(max(3 - 2 * v.k - c.e, 0), 63);                    // v c, units of 2^-58
  const unsigned int n = (unsigned int)((u + (1ull << 46)) >> 47);
  const long long t = (long long)(u - ((unsigned long long)n << 47));  // units of 2^-58
  const unsigned long long T = __ldg(&g_exp_table.v[n & (kExpN - 1)]);
  // x = |t| ln 2 in units of 2^-75
  const unsigned long long x = mul_hi((unsigned long long)(t < 0 ? -t : t) << 17, 0xb17217f7d1cf79acull);
  const unsigned int xh = (unsigned int)(x >> 31);  // units of 2^-44
  const unsigned long long x2 = (unsigned long long)xh * xh;  // units of 2^-88
  const unsigned int x2h = (unsigned int)(x2 >> 32);          // units of 2^-56
  const unsigned int x3 = __umulhi(__umulhi(x2h, xh), 0x2aaaaaabu);   // x^3 / 6, units of 2^-68
  const unsigned int x4 = __umulhi(__umulhi(x2h, x2h), 0x0aaaaaabu);  // x^4 / 24, units of 2^-80
  const unsigned long long even = (x2 >> 14) + (x4 >> 5), odd = x + ((unsigned long long)x3 << 7);
  // t >= 0: 1 - (odd - even); t < 0: 1 + (odd + even)
  const unsigned long long m = mul_hi(T, t < 0 ? odd + even : odd - even) >> 11;
  const unsigned long long e = t < 0 ? T + m : T - m;  // just around [2^61, 2^62]
  const int low = __clz((int)(e >> 32)) - 1;             // 0 to 2
  return pack64<10>(e << low, 1023 - low - (int)(n >> 11));
}
// exp(-z), 0 <= z < 11
__device__ __forceinline__ double exp_neg(double z) {
  constexpr Fix64 log2e = {0x5c551d94ae0bf85eull, 0};
  return exp2_neg(quad64(z), log2e);
}

// 1 / ((v + c) r), v a pair's squared distance, c > 0, r > 0: sum and product
// on the integers as well, one rounding in all
static __device__ __noinline__ double rcp_sum_slow(double d2, double c, double r) { return 1.0 / ((d2 + c) * r); }
__device__ __forceinline__ double rcp_sum_prod(const Quad64 &v, const Fix64 &c, double r, double d2, double cd) {
  const unsigned int rh = (unsigned int)__double2hiint(r), rl = (unsigned int)__double2loint(r);
  const int er = (int)(rh >> 20);  // sign included: a negative r is out of range
  if ((unsigned int)(er - 2) > 2042u) return rcp_sum_slow(d2, cd, r);
  const int e = max(2 * v.k + 2, c.e + 1);
  const unsigned long long vm = ((unsigned long long)v.vh << 32) | v.vl;
  const unsigned long long s = (vm >> min(e - 2 * v.k, 63)) + (c.m >> min(e - c.e, 63));  // units of 2^(e - 62)
  const int n = __clz((int)(s >> 32));  // 1 to 3
  const unsigned long long rm = ((unsigned long long)(((rh & 0xfffffu) << 11) | 0x80000000u | (rl >> 21)) << 32) | (rl << 11);
  unsigned long long p = mul_hi(s << n, rm);  // [2^62, 2^64)
  const int lead = (int)(p >> 63);
  p <<= 1 - lead;
  // (v + c) r = (p / 2^63) 2^(e + 1 - n + er - 1023 + lead)
  return pack64<10>(rcp_q63((unsigned int)(p >> 32), (unsigned int)p), 2044 - (e - n + er + lead));
}

// u^2 / 2^64, within 2 units
__device__ __forceinline__ unsigned long long square_hi(unsigned long long u) {
  const unsigned int u1 = (unsigned int)(u >> 32), u0 = (unsigned int)u;
  return (unsigned long long)u1 * u1 + (((unsigned long long)u1 * u0) >> 31);
}

// q = r / h from the pair's squared distance, y = 1 / sqrt(v) and ih = 1 / h, in
// units of 2^-61; q < 2 + 2^-40
__device__ __forceinline__ unsigned long long q_q61(const Quad64 &v, unsigned long long y, const Fix64 &ih) {
  // r = s 2^k, s in [1, 2) in units of 2^-61; q = (s ih.m) 2^(k + ih.e), the product in [1, 4)
  return mul_hi(sqrt_q61(v, y) << 2, ih.m << 1) >> min(max(1 - v.k - ih.e, 0), 63);
}

// 1 - q / 2 for the Wendland kernel, 0 from q = 2 on: an exact difference of
// integers, rounded once
__device__ __forceinline__ double wendland_in(const Quad64 &v, const Fix64 &ih) {
  const unsigned long long q = q_q61(v, rsqrt_q63(v), ih);  // units of 2^-62 for q / 2
  if (q >= 1ull << 62) return 0.0;
  const unsigned long long t = (1ull << 62) - q;
  const int n = __clzll((long long)t);
  return pack64<10>(t << (n - 1), 1024 - n);
}

// g(q) of the cubic spline's gradient factor -(al / h^2) g, q = r / h:
// 3 - 2.25 q for q <= 1, 0.75 (2 - q)^2 / q up to 2, from the pair's squared
// distance and ih = 1 / h, h; q < 2 + 2^-40.  Fixed point.  2 - q is an exact
// difference of integers and is normalised before it is squared, so that g has
// the relative accuracy of 2 - q up to the support's edge (multiplied out, as
// 3 / q + 0.75 q - 3, it cancels there: 2e-8 off at q = 1.9999).
__device__ __forceinline__ double cubic_g(const Quad64 &v, const Fix64 &ih, const Fix64 &h) {
  const unsigned long long y = rsqrt_q63(v);
  const unsigned long long q = q_q61(v, y, ih);
  constexpr unsigned long long one = 1ull << 61;
  unsigned long long g;  // the result is g 2^(e - 1086)
  int e;
  if (q <= one) {
    g = 3 * one - 2 * q - (q >> 2);
    e = 1086 - 61;
  } else {
    if (q >= 2 * one) return 0.0;
    // 1 / q = y h 2^-k in units of 2^-61: y in [0.5, 1], h.m / 2^62 in [1, 2)
    const unsigned long long iq = mul_hi(y, h.m << 1) >> min(max(1 - (h.e - v.k), 0), 63);
    const unsigned long long t = 2 * one - q;
    const int n = __clzll((long long)t);                             // t = (t << n) 2^(-61 - n)
    const unsigned long long p = mul_hi(square_hi(t << n), iq << 2);  // t^2 / q in units of 2^(-57 - 2 n)
    g = p - (p >> 2);
    e = 1086 - 57 - 2 * n;
  }
  const int n = __clzll((long long)g);
  return pack64<10>(g << (n - 1), e - n);
}

// ---------------------------------------------------------------------------
// Positions as 64-bit integers, for pair differences on the integer pipe: a
// position in units of 2^-s modulo 2^64, with s such that the interaction
// radius is below 2^62 units (fix_shift), so that the difference of two
// candidates' integers is that of their positions, exactly.  The lowest bit is not
// the position's: it marks a coordinate with bits below 2^(1 - s) (one closer to
// zero than R / 256, unless it ends in zeros), whose pairs take FP64 differences.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int fix_shift(double R) {
  return 61 - ((int)(((unsigned int)__double2hiint(R) >> 20) & 0x7ffu) - 1023);
}
__device__ __forceinline__ long long to_fix(double x, int s) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  const int e = (int)((u >> 52) & 0x7ffu);
  unsigned long long m = (u & 0xfffffffffffffull) | (e ? 0x10000000000000ull : 0ull), cut = 0ull;
  const int sh = e - 1075 + s;
  if (sh > 0) {
    m = sh < 64 ? m << sh : 0ull;
  } else {
    const unsigned long long low = sh > -63 ? (2ull << -sh) - 1ull : ~0ull;
    cut = (m & low) ? 1ull : 0ull;
    m = sh > -64 ? (m & ~low) >> -sh : 0ull;
  }
  return (long long)(((u >> 63) ? 0ull - m : m) | cut);
}
__device__ __forceinline__ bool fix_cut(longlong2 a) { return ((a.x | a.y) & 1ll) != 0ll; }

// A pair's geometry: the differences, the squared distance (each rounded once)
// and the latter's significand for sqrt_rsqrt64.
struct PairGeom {
  double dx, dy, d2;
  Quad64 v;
};
// |d| < 2^63 units of 2^-s as a double
__device__ __forceinline__ double fix_diff(unsigned long long a, int s, bool neg) {
  if (a == 0ull) return 0.0;
  const int n = __clzll((long long)a);
  return pack64<10>(a << (n - 1), 1086 - n - s, neg ? 0x80000000u : 0u);
}
__device__ __forceinline__ PairGeom pair_geom(longlong2 a, longlong2 b, int s) {
  PairGeom p;
  const long long ix = (long long)((unsigned long long)a.x - (unsigned long long)b.x);
  const long long iy = (long long)((unsigned long long)a.y - (unsigned long long)b.y);
  const unsigned long long ux = ix < 0 ? -(unsigned long long)ix : (unsigned long long)ix;
  const unsigned long long uy = iy < 0 ? -(unsigned long long)iy : (unsigned long long)iy;
  p.dx = fix_diff(ux, s, ix < 0);
  p.dy = fix_diff(uy, s, iy < 0);
  // both shifted so that the larger's leading bit is bit 62
  const int sh = __clzll((long long)(ux | uy | 1ull)) - 1;
  const unsigned long long d = square_hi(ux << sh) + square_hi(uy << sh);  // [2^60, 2^63)
  const bool big = (d >> 62) != 0ull;
  const unsigned long long v = big ? d : d << 2;
  p.v = {(unsigned int)(v >> 32), (unsigned int)v, (big ? 63 : 62) - sh - s};
  const unsigned int odd = (unsigned int)(v >> 63);
  p.d2 = (ux | uy) == 0ull ? 0.0 : pack64<10>(v >> odd, 1023 + 2 * p.v.k + (int)odd);
  return p;
}
// the same by FP64 operations
__device__ __forceinline__ PairGeom pair_geom_fp64(double dx, double dy) {
  PairGeom p;
  p.dx = dx;
  p.dy = dy;
  p.d2 = fma(dx, dx, dy * dy);
  p.v = quad64(p.d2);
  return p;
}
// out of line: for a coordinate whose integer is not all of it (to_fix), and
// where the padding of the FP32 test could let differences past the integers'
// range through (a domain of some millions of radii)
static __device__ __noinline__ PairGeom pair_geom_wide(double dx, double dy) { return pair_geom_fp64(dx, dy); }

// a <= b for non-negative doubles (false when either is NaN and a is not
// below b's pattern), without an FP64 instruction
__device__ __forceinline__ bool le_bits(double a, double b) {
  return (unsigned long long)__double_as_longlong(a) <= (unsigned long long)__double_as_longlong(b);
}

// ---------------------------------------------------------------------------
// Launch constants of the FP64 pair kernels
// ---------------------------------------------------------------------------
struct Pair64 {
  int xsph, sumdens;
  // uniform fluid h (UH)
  double h, ih, lim;           // h, 1/h, (support h)^2
  double lim_lo, lim_hi;       // Gaussian: below / above, q <= 3 is decided
  double h2;                   // cubic: d2 <= h^2 is the inner piece.  Gaussian: d2 <= h2 has no gradient
  double o_t, o_r, o_rl;       // cubic, outer piece: (o_t / r) (2 + o_r r)^2, o_r = -1 / h in two parts
  double i_r, i_0;             // inner piece: i_r r + i_0.  Wendland: (i_r r + i_0) in^5, in = 1 + o_r r, o_r = -1 / (2 h)
  double g_d;                  // Gaussian: -2 / h^2, the gradient factor's derivative over r
  double scale;                // of the gradient factor that is summed (cubic -al / h^2, Gaussian and Wendland i_0)
  Fix64 hf, ihf, hb2f;         // h, 1/h, hb2
  Fix64 l2e;                   // log2(e) / h^2
  double al;                   // normalisation of W
  double hb2, pic;             // viscosity: pic dot / ((d2 + hb2) (rho_i + rho_j))
  double r02;                  // r0^2
  int lj_free;                 // r0 < 1.5 h: the Lennard-Jones pairs all have q <= 3
};

// the Lennard-Jones length: r <= r0 has no pair for a negative or NaN r0
inline double lj_reach(const sph_wcsph_t &wc) { return wc.r0 > 0.0 ? wc.r0 : 0.0; }

inline Pair64 pair64_consts(const sph_config_t &cfg, const sph_wcsph_t &wc) {
  Pair64 c;
  c.xsph = wc.use_xsph != 0;
  c.sumdens = wc.use_summation_density != 0;
  const double h = cfg.h_fixed > 0.0 ? cfg.h_fixed : 1.0;
  const double ih = 1.0 / h, hh = h * h;
  c.h = h;
  c.ih = ih;
  c.h2 = hh;
  c.o_t = c.i_r = c.i_0 = 0.0;
  c.o_r = -ih;
  c.o_rl = -fma(-ih, h, 1.0) / h;
  c.g_d = -2.0 / hh;
  if (cfg.kernel == SPH_KERNEL_CUBIC) {
    // al / (h r) times -0.75 (2 - q)^2 and -3 q (1 - 0.75 q) (CubicSpline.py:40-70)
    c.al = kCubicFac / hh;
    c.lim = 4.0 * h * h;
    c.o_t = -0.75 * c.al / h;
    c.i_0 = -3.0 * c.al / hh;
    c.i_r = 2.25 * c.al / (hh * h);
  } else if (cfg.kernel == SPH_KERNEL_WENDLAND) {
    // al / (h r) (1 - q/2)^5 (-14/3) q (1 + 2.5 q) (Wendland.py:36-64)
    c.al = kWendFac / hh;
    c.lim = 4.0 * h * h;
    c.o_r *= 0.5;
    c.o_rl *= 0.5;
    c.i_0 = (-14.0 / 3.0) * c.al / hh;
    c.i_r = (-35.0 / 3.0) * c.al / (hh * h);
  } else {
    // -2 al / h^2 exp(-q^2) (Gaussian.py:37-59)
    c.al = kInvPi / hh;
    c.lim = 9.0 * h * h;
    c.i_0 = -2.0 * c.al / hh;
    c.h2 = 1e-24 / hh;  // r h <= 1e-12: no gradient
  }
  c.lim_lo = c.lim * (1.0 - 1e-9);
  c.lim_hi = c.lim * (1.0 + 1e-9);
  c.hb2 = 0.01 * hh;
  c.hf = fix64(h);
  c.ihf = fix64_quot(1.0, 0.0, h, 0.0);
  c.hb2f = fix64(c.hb2);
  c.l2e = fix64_quot(0x1.71547652b82fep+0, 0x1.777d0ffda0d24p-56, hh, fma(h, h, -hh));  // log2(e) in two parts
  c.scale = cfg.kernel == SPH_KERNEL_CUBIC ? -c.al / hh : c.i_0;
  c.pic = -wc.alpha * wc.co * h;  // -2 alpha c_ij h with c_ij = co / 2
  c.r02 = lj_reach(wc) * lj_reach(wc);
  c.lj_free = cfg.h_fixed > 0.0 && wc.r0 < 1.5 * h * (1.0 - 1e-9);
  return c;
}

// q = r / h_ij <= 3 as the reference decides it
static __device__ __noinline__ bool near_exact(double dx, double dy, double hij) {
  const double r = __dsqrt_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)));
  return __ddiv_rn(r, hij) <= 3.0;
}

}  // namespace sph
