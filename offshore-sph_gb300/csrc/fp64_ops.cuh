// fp64_ops.cuh -- reciprocal, square root and exponential in few FP64
// operations, and the launch constants of the FP64 pair kernels, for the
// kernels that the FP64 pipe bounds.
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

// ---------------------------------------------------------------------------
// Launch constants of the FP64 pair kernels
// ---------------------------------------------------------------------------
struct Pair64 {
  int xsph, sumdens;
  // uniform fluid h (UH)
  double h, ih, lim;           // h, 1/h, (support h)^2
  double lim_lo, lim_hi;       // Gaussian: below / above, q <= 3 is decided
  double h2;                   // cubic: d2 <= h^2 is the inner piece.  Gaussian: d2 <= h2 has no gradient
  double o_ir, o_r, o_0;       // cubic, outer piece: o_ir / r + o_r r + o_0
  double i_r, i_0;             // inner piece: i_r r + i_0.  Wendland: (i_r r + i_0) (1 + o_r r)^5
  double al;                   // normalisation of W
  double hb2, pic;             // viscosity: pic dot / ((d2 + hb2) (rho_i + rho_j))
  double r02;                  // r0^2
  int lj_free;                 // r0 < 1.5 h: the Lennard-Jones pairs all have q <= 3
};

inline Pair64 pair64_consts(const sph_config_t &cfg, const sph_wcsph_t &wc) {
  Pair64 c;
  c.xsph = wc.use_xsph != 0;
  c.sumdens = wc.use_summation_density != 0;
  const double h = cfg.h_fixed > 0.0 ? cfg.h_fixed : 1.0;
  const double ih = 1.0 / h, ih2 = ih * ih;
  c.h = h;
  c.ih = ih;
  c.h2 = h * h;
  c.o_ir = c.o_r = c.o_0 = c.i_r = c.i_0 = 0.0;
  if (cfg.kernel == SPH_KERNEL_CUBIC) {
    // al / (h r) times -0.75 (2 - q)^2 and -3 q (1 - 0.75 q) (CubicSpline.py:40-70)
    c.al = kCubicFac * ih2;
    c.lim = 4.0 * h * h;
    c.o_ir = -3.0 * c.al * ih;
    c.o_0 = 3.0 * c.al * ih2;
    c.o_r = -0.75 * c.al * ih2 * ih;
    c.i_0 = -3.0 * c.al * ih2;
    c.i_r = 2.25 * c.al * ih2 * ih;
  } else if (cfg.kernel == SPH_KERNEL_WENDLAND) {
    // al / (h r) (1 - q/2)^5 (-14/3) q (1 + 2.5 q) (Wendland.py:36-64)
    c.al = kWendFac * ih2;
    c.lim = 4.0 * h * h;
    c.o_r = -0.5 * ih;
    c.i_0 = (-14.0 / 3.0) * c.al * ih2;
    c.i_r = (-35.0 / 3.0) * c.al * ih2 * ih;
  } else {
    // -2 al / h^2 exp(-q^2) (Gaussian.py:37-59)
    c.al = kInvPi * ih2;
    c.lim = 9.0 * h * h;
    c.i_0 = -2.0 * c.al * ih2;
    c.h2 = 1e-24 * ih2;  // r h <= 1e-12: no gradient
  }
  c.lim_lo = c.lim * (1.0 - 1e-9);
  c.lim_hi = c.lim * (1.0 + 1e-9);
  c.hb2 = 0.01 * (h * h);
  c.pic = -wc.alpha * wc.co * h;  // -2 alpha c_ij h with c_ij = co / 2
  c.r02 = wc.r0 * wc.r0;
  c.lj_free = cfg.h_fixed > 0.0 && wc.r0 < 1.5 * h * (1.0 - 1e-9);
  return c;
}

// q = r / h_ij <= 3 as the reference decides it
static __device__ __noinline__ bool near_exact(double dx, double dy, double hij) {
  const double r = __dsqrt_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)));
  return __ddiv_rn(r, hij) <= 3.0;
}

}  // namespace sph
