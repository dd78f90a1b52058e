// adjoint.cu -- reverse mode of the WCSPH step (FP64 and mixed forms).
//
// The forward step with a fixed dt (src/Solver.py:370-372 timeStep path) and
// the PEC integrator (src/Integrators/PEC.py:32-89, damping 0) maps the state
// S = (x, v, rho, a, drho) of the fluid particles to S':
//   half:    x_h = x + dt/2 v,  v_h = v + dt/2 a,  rho_h = rho + dt/2 drho
//   compute: (A, D) = F(x_h, v_h, rho_h; alpha)   (src/Tools/SolverTools.py:120-175)
//   correct: x' = x + dt v_h,  v' = v + dt A,  rho' = rho + dt D,  a' = A,  drho' = D
// and adds omega * (wall load of the evaluation) to the loss.  The adjoint
// step maps the adjoint of S' back to the adjoint of S:
//   lambda_A = dt vb' + ab',  lambda_D = dt rhob' + drhob'       (k_adj_pre)
//   (xb_h, vb_h, rhob_h, alphab) = VJP of F and of the wall load  (k_pair_adjoint)
//   vb_h += dt xb';  xb = xb' + xb_h;  vb = vb' + dt/2 xb_h + vb_h;
//   ab = dt/2 vb_h;  rhob = rhob' + rhob_h;  drhob = dt/2 rhob_h  (k_adj_post)
//
// k_pair_adjoint is the hand-written vector-Jacobian product of the fused
// pair evaluation: continuity (src/Equations/Continuity.py), momentum with
// artificial viscosity (src/Equations/Momentum.py), the Tait EOS inside
// p/rho^2 (src/Equations/TaitEOS.py) and the Lennard-Jones boundary force
// (src/Equations/BoundaryForce.py).  For a fluid pair (k, j) the outputs of
// both particles enter one scalar
//   phi = lQ . (S dW) + lC (v_kj . dW),
//   lQ = -m_j lambdaA_k + m_k lambdaA_j,  lC = m_j lambdaD_k + m_k lambdaD_j,
//   S = p_k/rho_k^2 + p_j/rho_j^2 + Pi_kj,
// which is the same for (k, j) and (j, k); each thread differentiates it with
// respect to its own position, velocity and density, so the product is a
// gather over the neighbour set with no atomics.  The alpha adjoint takes
// each thread's own outputs only, so each pair counts once.
#include <math.h>

#include <type_traits>

#include "fp64_ops.cuh"
#include "pair_common.cuh"

namespace sph {

// two-warp blocks: the kernels have few warps per SM, and small blocks spread
// them evenly
constexpr int kAdjBlock = 64;
// resident blocks of the FP64 kernel: the registers' limit that measured
// fastest (40 steps of the 20K wall-load case: 9.09 ms at 6, 8.93 at 8, 8.70 at
// 10, 8.77 at 12)
constexpr int kAdjBlocks = 10;

struct AdjParams {
  double alpha, beta, co, r0, D, p1, p2, gamma, B, inv_rho0;
  int lj_42;
  double omega, wall_x, dt;
  long long n;
};

// d(p/rho^2)/drho of a fluid particle from its rho and p/rho^2
// (p = B ((rho/rho0)^gamma - 1) + Pb, src/Equations/TaitEOS.py:6-31)
__device__ __forceinline__ double dothr_drho(double rho, double othr, const AdjParams &ap) {
  if (!(rho > 0.0)) return 0.0;
  const double t = rho * ap.inv_rho0;
  double tg1;  // t^(gamma - 1)
  if (ap.gamma == 7.0) {
    const double t2 = t * t, t3 = t2 * t;
    tg1 = t3 * t3;
  } else {
    tg1 = pow(t, ap.gamma - 1.0);
  }
  const double dp = ap.B * ap.gamma * ap.inv_rho0 * tg1;
  return (dp - 2.0 * othr * rho) / (rho * rho);
}

struct AdjPtrs {
  const float4 *rec0;  // FP32 positions and signed h (prefilter)
  const double4_32a *r64a, *r64b;
  const longlong2 *fix;  // integer positions (fp64_ops.cuh)
  const int *perm, *keys_sorted;
  const int2 *meta;
  const unsigned int *cstart;
  const DevGrid *grid;
  DevCtrl *ctrl;
  const double *lax, *lay, *lad;                  // lambda_A, lambda_D (caller order)
  double *xhb, *yhb, *vxhb, *vyhb, *rhohb, *alb;  // outputs (caller order)
};

// The forward's padded FP32 reach test (kernel support for fluid, min(r0,
// 3 h_ij) for boundary): a candidate outside it contributes nothing.
struct AdjReach {
  const AdjPtrs &P;
  const DevGrid &g;
  long long k;
  int2 qref;
  bool filter;
  float4 Qi;
  float rf2, pad, r0f;
  __device__ __forceinline__ AdjReach(const AdjPtrs &P, const AdjParams &ap, const DevGrid &g, long long k, int2 qref,
                                      float support)
      : P(P), g(g), k(k), qref(qref) {
    filter = g.mode == 1 && (g.need_filter || P.ctrl->alias_count > 0);
    Qi = P.rec0[k];
    pad = g.pad_e;
    r0f = (float)ap.r0;
    const float rf = support * 1.000002f * Qi.z + pad;
    rf2 = rf * rf;
  }
  __device__ __forceinline__ float4 load(unsigned int j) const { return __ldg(P.rec0 + j); }
  __device__ __forceinline__ bool test(unsigned int j, float4 qj) const {
    if (j == (unsigned int)k) return false;
    if (filter && !in_ref_stencil(P.meta, j, g, qref)) return false;
    const float fx = Qi.x - qj.x, fy = Qi.y - qj.y;
    const float d2 = fx * fx + fy * fy;
    if (!signbit(qj.z)) return d2 <= rf2;  // every fluid h is the same
    const float rp = fminf(r0f, 1.5f * (Qi.z + fabsf(qj.z))) * 1.000002f + pad;
    return d2 <= rp * rp;
  }
};

// G lanes per query (for_neighbours).  The FP64 pipe bounds it: about 50 FP64
// operations per fluid pair, with the building blocks and launch constants of
// the forward (pair64.cu).  Listing the pairs first keeps the lanes of a warp
// together: evaluating each candidate as the walk met it ran 12.5 of 32 lanes
// on average.  22K particles, one step: 297 us so, 100 us with the pairs listed, 91
// with the forward's integer arithmetic, 82 with 10 blocks per SM, 87 with 2 - q
// formed before it is squared (ncu).
template <int KERNEL, int G>
__global__ void __launch_bounds__(kAdjBlock, kAdjBlocks) k_pair_adjoint(AdjPtrs P, AdjParams ap, Pair64 c) {
  constexpr int kCap = list_words<G>(ListCap<KERNEL>::value);
  constexpr bool gauss = KERNEL == SPH_KERNEL_GAUSSIAN;
  constexpr bool kFix = G < 8;  // integer differences, as in the forward
  __shared__ unsigned int lists[kCap * kAdjBlock / G];
  const DevGrid &g = *P.grid;
  const long long k = ((long long)blockIdx.x * kAdjBlock + threadIdx.x) / G;
  const long long kq = k < ap.n ? k : 0;
  const int i = P.perm[kq];
  const double4_32a Ak = P.r64a[kq], Bk = P.r64b[kq];
  const bool act = k < ap.n && !signbit(Bk.w);
  double gx = 0.0, gy = 0.0, gvx = 0.0, gvy = 0.0, glq = 0.0, grh = 0.0, gal = 0.0;
  const double mk = Bk.x, rhok = Bk.y, othrk = Bk.z, hk = Bk.w;
  if (G > 1 ? __any_sync(0xffffffffu, act) : act) {
    const double lAxk = P.lax[i], lAyk = P.lay[i], lDk = P.lad[i];
    const double ac = ap.alpha * 0.5 * ap.co;
    const longlong2 pk = kFix ? P.fix[kq] : longlong2();
    const int fix_s = g.fix_s;
    const bool wide = (kFix && fix_cut(pk)) || g.pad_e > 0.5f * (float)g.r_search;
    const int2 qref = P.meta[kq];
    const bool slow = qref.x >= g.ncx;
    const int W = g.mode == 0 ? 1 : (slow ? g.wide : g.wt);
    const AdjReach near(P, ap, g, kq, qref, (float)Support<KERNEL>::q);
    const Stencil sten(g, qref, P.keys_sorted[kq], W);
    for_neighbours<G, kCap, kAdjBlock>(sten, P.cstart, act, lists, near, [&](unsigned int j) {
      const double4_32a Aj = P.r64a[j], Bj = P.r64b[j];
      PairGeom geo;
      if constexpr (kFix) {
        const longlong2 pj = P.fix[j];
        geo = wide || fix_cut(pj) ? pair_geom_wide(Ak.x - Aj.x, Ak.y - Aj.y) : pair_geom(pk, pj, fix_s);
      } else {
        geo = pair_geom_fp64(Ak.x - Aj.x, Ak.y - Aj.y);
      }
      const double dx = geo.dx, dy = geo.dy, d2 = geo.d2;
      if (le_bits(d2, 1e-24)) return;  // coincident: no kernel gradient, no boundary force
      if (!signbit(Bj.w)) {
        // fluid pair: continuity + momentum with artificial viscosity.
        // dW = coef u; dci = (d coef / d r) / r
        double coef, dci;
        if constexpr (gauss) {
          if (!le_bits(d2, c.lim_lo) && (!le_bits(d2, c.lim_hi) || !near_exact(Ak.x - Aj.x, Ak.y - Aj.y, hk))) return;
          if (le_bits(d2, c.h2)) return;
          coef = c.i_0 * exp2_neg(geo.v, c.l2e);
          dci = coef * c.g_d;
        } else {
          if (!le_bits(d2, c.lim) || le_bits(d2, 1e-20)) return;
          double r, ir;
          sqrt_rsqrt64(geo.v, r, ir);
          if (KERNEL == SPH_KERNEL_CUBIC) {
            if (le_bits(d2, c.h2)) {
              coef = fma(c.i_r, r, c.i_0);
              dci = c.i_r * ir;
            } else {
              // o_t t^2 / r, t = 2 - r / h; its derivative -o_t (t / r) (2 / r + 1 / h)
              const double t = fma(c.o_rl, r, fma(c.o_r, r, 2.0)), A = c.o_t * ir * t;
              coef = A * t;
              dci = (A * ir) * fma(-2.0, ir, c.o_r);
            }
          } else {
            const double in = fma(c.o_rl, r, fma(c.o_r, r, 1.0)), in2 = in * in, in4 = in2 * in2;
            const double l = fma(c.i_r, r, c.i_0);
            coef = in4 * (in * l);
            dci = ir * in4 * fma(5.0 * c.o_r, l, in * c.i_r);
          }
        }
        const double mj = Bj.x;
        const int pj = P.perm[j];
        const double lAxj = P.lax[pj], lAyj = P.lay[pj], lDj = P.lad[pj];
        const double vx = Ak.z - Aj.z, vy = Ak.w - Aj.w;
        const double dot = fma(vx, dx, vy * dy);
        const double lQx = fma(mk, lAxj, -mj * lAxk), lQy = fma(mk, lAyj, -mj * lAyk);
        const double lC = fma(mk, lDj, mj * lDk);
        const double lQu = fma(lQx, dx, lQy * dy), lQdW = coef * lQu;
        double S = othrk + Bj.z;
        glq += lQdW;
        if (negative_bits(dot)) {
          const double rs = rhok + Bj.y;  // 2 rho_kj
          const double den = d2 + c.hb2;
          const double inv = rcp64(den * rs);
          const double a = dot * inv, irs = inv * den;
          double Pi, f;  // Pi, and lQdW times d Pi / d (dot)
          if (ap.beta == 0.0) {
            Pi = (-2.0 * ac * c.h) * a;
            f = lQdW * ((-2.0 * ac * c.h) * inv);
          } else {
            const double mu = c.h * (a * rs);
            Pi = 2.0 * mu * fma(ap.beta, mu, -ac) * irs;
            f = lQdW * (2.0 * c.h * fma(2.0 * ap.beta, mu, -ac) * inv);
          }
          S += Pi;
          const double c2 = 2.0 * (a * rs);  // 2 dot / (r^2 + 0.01 h^2)
          gx = fma(f, fma(-c2, dx, vx), gx);
          gy = fma(f, fma(-c2, dy, vy), gy);
          gvx = fma(f, dx, gvx);
          gvy = fma(f, dy, gvy);
          gal = fma((mj * coef) * fma(lAxk, dx, lAyk * dy), a, gal);
          grh = fma(-lQdW, Pi * irs, grh);  // d rbar / d rho_k = 1/2
        }
        // (d dW / d u)^T z = coef z + (dcoef / r) (u . z) u
        const double cq = dci * fma(S, lQu, lC * dot);
        const double lCc = lC * coef, Sc = S * coef;
        gx = fma(cq, dx, fma(Sc, lQx, fma(lCc, vx, gx)));
        gy = fma(cq, dy, fma(Sc, lQy, fma(lCc, vy, gy)));
        gvx = fma(lCc, dx, gvx);
        gvy = fma(lCc, dy, gvy);
        return;
      }
      // boundary pair: Lennard-Jones force b = D phi(r) u, phi = ((r0/r)^p1 - (r0/r)^p2) / r^2,
      // and the wall load -m_k b.x when j is on the loaded wall
      if (!le_bits(d2, c.r02)) return;
      if (!c.lj_free) {  // the neighbour test
        const double hij = 0.5 * (hk + fabs(Bj.w)), t = 3.0 * hij, t2 = t * t;
        if (!le_bits(d2, t2 * (1.0 - 1e-9)) && (!le_bits(d2, t2 * (1.0 + 1e-9)) || !near_exact(Ak.x - Aj.x, Ak.y - Aj.y, hij))) return;
      }
      const double ir2 = rcp64(d2);
      double sp1, sp2;
      if (ap.lj_42) {
        sp2 = c.r02 * ir2;
        sp1 = sp2 * sp2;
      } else {
        const double s = ap.r0 / __dsqrt_rn(d2);
        sp1 = pow(s, ap.p1);
        sp2 = pow(s, ap.p2);
      }
      const double phi = (sp1 - sp2) * ir2;
      const double dphi = fma(-ap.p1 - 2.0, sp1, (ap.p2 + 2.0) * sp2) * (ir2 * ir2);  // phi' / r
      const double zx = lAxk - ((ap.omega != 0.0 && Aj.x >= ap.wall_x) ? ap.omega * mk : 0.0), zy = lAyk;
      const double q = dphi * fma(dx, zx, dy * zy);
      gx = fma(ap.D, fma(phi, zx, q * dx), gx);
      gy = fma(ap.D, fma(phi, zy, q * dy), gy);
    });
  }
  group_sum<G>(gx);
  group_sum<G>(gy);
  group_sum<G>(gvx);
  group_sum<G>(gvy);
  group_sum<G>(glq);
  group_sum<G>(grh);
  group_sum<G>(gal);
  if (k < ap.n && threadIdx.x % G == 0) {  // non-fluid particles get zeros: no outputs, their adjoint is not used
    P.xhb[i] = gx;
    P.yhb[i] = gy;
    P.vxhb[i] = gvx;
    P.vyhb[i] = gvy;
    P.rhohb[i] = act ? fma(glq, dothr_drho(rhok, othrk, ap), grh) : 0.0;
    P.alb[i] = gal * (ap.co * c.h);  // mu cbar / rho_kj = 2 cbar h a
  }
}

// ---------------------------------------------------------------------------
// Mixed form of the adjoint pair product: the same vector-Jacobian product as
// k_pair_adjoint with the pair arithmetic in FP32 (hardware reciprocals and
// square roots) and the per-particle sums in FP32, over the FP64 records of
// the forward evaluation and the FP64 adjoint vectors.  Differences of FP64
// positions and velocities are formed in FP64 and then rounded, so large
// coordinates lose no accuracy.  The forward's q <= 3 decision is redone
// exactly where FP32 could decide it differently.
// ---------------------------------------------------------------------------
template <int KERNEL>
__device__ __forceinline__ void grad_coef_f(float r, float q, float ih, float ir, float &coef, float &dcoef) {
  coef = 0.f;
  dcoef = 0.f;
  const float ih2 = ih * ih;
  if (KERNEL == SPH_KERNEL_CUBIC) {
    if (q > 2.0f || r < 1e-10f) return;
    const float al = (float)kCubicFac * ih2;
    float g, gp;
    if (q > 1.0f) {
      const float t = 2.0f - q;
      g = -0.75f * t * t;
      gp = 1.5f * t;
    } else {
      g = -3.0f * q * (1.0f - 0.75f * q);
      gp = -3.0f + 4.5f * q;
    }
    const float a = al * ih * ir;
    coef = a * g;
    dcoef = a * (gp * ih - g * ir);
  } else if (KERNEL == SPH_KERNEL_WENDLAND) {
    if (q >= 2.0f || r < 1e-10f) return;
    const float al = (float)kWendFac * ih2;
    const float in = 1.0f - 0.5f * q, in2 = in * in, in4 = in2 * in2;
    const float g = in4 * in * (-14.0f / 3.0f) * q * (1.0f + 2.5f * q);
    const float gp = (-14.0f / 3.0f) * (in4 * in * (1.0f + 5.0f * q) - 2.5f * in4 * q * (1.0f + 2.5f * q));
    const float a = al * ih * ir;
    coef = a * g;
    dcoef = a * (gp * ih - g * ir);
  } else {
    if (!(q <= 3.0f) || !(r > 1e-12f * ih)) return;
    coef = -2.0f * (float)kInvPi * ih2 * __expf(-q * q) * ih2;
    dcoef = coef * (-2.0f * r * ih2);
  }
}

template <int KERNEL, int G>
__global__ void __launch_bounds__(kAdjBlock) k_pair_adjoint_mixed(AdjPtrs P, AdjParams ap) {
  constexpr int kCap = list_words<G>(ListCap<KERNEL>::value);
  __shared__ unsigned int lists[kCap * kAdjBlock / G];
  const DevGrid &g = *P.grid;
  const long long k = ((long long)blockIdx.x * kAdjBlock + threadIdx.x) / G;
  const long long kq = k < ap.n ? k : 0;
  const int i = P.perm[kq];
  const double4_32a Ak = P.r64a[kq], Bk = P.r64b[kq];
  const bool act = k < ap.n && !signbit(Bk.w);
  float gx = 0.f, gy = 0.f, gvx = 0.f, gvy = 0.f, grho = 0.f, gal = 0.f;
  if (G > 1 ? __any_sync(0xffffffffu, act) : act) {
    const double xk = Ak.x, yk = Ak.y, vxk = Ak.z, vyk = Ak.w;
    const double hk = Bk.w;
    const float mk = d2f_trunc(Bk.x), rhok = d2f_trunc(Bk.y), othrk = d2f_trunc(Bk.z), hkf = d2f_trunc(hk);
    const float lAxk = d2f_trunc(P.lax[i]), lAyk = d2f_trunc(P.lay[i]), lDk = d2f_trunc(P.lad[i]);
    const float dothk = d2f_trunc(dothr_drho(Bk.y, Bk.z, ap));
    const float ihk = __fdividef(1.0f, hkf);
    const float cbar = 0.5f * (float)ap.co, alpha = (float)ap.alpha, beta = (float)ap.beta;
    const float r0 = (float)ap.r0, D = (float)ap.D, p1 = (float)ap.p1, p2 = (float)ap.p2;
    const float omega_m = (float)ap.omega * mk;
    const int2 qref = P.meta[kq];
    const bool slow = qref.x >= g.ncx || !(hk > 0.0);
    const int W = g.mode == 0 ? 1 : (slow ? g.wide : g.wt);
    const AdjReach near(P, ap, g, kq, qref, (float)Support<KERNEL>::q);
    const Stencil sten(g, qref, P.keys_sorted[kq], W);
    for_neighbours<G, kCap, kAdjBlock>(sten, P.cstart, act, lists, near, [&](unsigned int j) {
      const double4_32a Aj = P.r64a[j], Bj = P.r64b[j];
      const double dxd = xk - Aj.x, dyd = yk - Aj.y;
      const float dx = d2f_trunc(dxd), dy = d2f_trunc(dyd);
      const float d2 = dx * dx + dy * dy;
      if (!(d2 > 1e-24f)) return;  // coincident: no kernel gradient, no boundary force
      const float ir = rsqrtf(d2);
      const float r = d2 * ir;
      const double hj = fabs(Bj.w);
      const float hjf = d2f_trunc(hj);
      const float hij = 0.5f * (hkf + hjf);
      const float ih = hj == hk ? ihk : (hj == 0.0 ? 2.0f * ihk : __fdividef(1.0f, hij));
      const float q = r * ih;
      bool in = q <= 3.0f;
      if (fabsf(q - 3.0f) < 1e-4f) {  // the forward's neighbour test (NNLinkedList.py:74), exactly
        const double rd = __dsqrt_rn(__dadd_rn(__dmul_rn(dxd, dxd), __dmul_rn(dyd, dyd)));
        in = __ddiv_rn(rd, __dmul_rn(0.5, __dadd_rn(hk, hj))) <= 3.0;
      }
      if (!in) return;
      if (!signbit(Bj.w)) {
        // fluid pair: continuity + momentum with artificial viscosity
        const float mj = d2f_trunc(Bj.x), rhoj = d2f_trunc(Bj.y), othrj = d2f_trunc(Bj.z);
        const float vxij = d2f_trunc(vxk - Aj.z), vyij = d2f_trunc(vyk - Aj.w);
        float coef, dcoef;
        grad_coef_f<KERNEL>(r, q, ih, ir, coef, dcoef);
        if (coef == 0.f && dcoef == 0.f) return;
        const float dWx = coef * dx, dWy = coef * dy;
        const float dot = vxij * dx + vyij * dy;
        const float irbar = __fdividef(2.0f, rhok + rhoj);
        float Pi = 0.f, dPi_dmu = 0.f, mu = 0.f, iden = 0.f, hb = 0.f;
        if (dot < 0.f) {
          hb = 0.5f * (hkf + hij);
          iden = __fdividef(1.0f, d2 + 0.01f * hb * hb);
          mu = hb * dot * iden;
          Pi = mu * (beta * mu - alpha * cbar) * irbar;
          dPi_dmu = (2.0f * beta * mu - alpha * cbar) * irbar;
        }
        const float S = othrk + othrj + Pi;
        const int pj = P.perm[j];
        const float lAxj = d2f_trunc(P.lax[pj]), lAyj = d2f_trunc(P.lay[pj]), lDj = d2f_trunc(P.lad[pj]);
        const float lQx = -mj * lAxk + mk * lAxj, lQy = -mj * lAyk + mk * lAyj;
        const float lC = mj * lDk + mk * lDj;
        const float lQdW = lQx * dWx + lQy * dWy;
        // (d dW / d u)^T z = coef z + dcoef (u . z) u / r
        const float cq = S * dcoef * (dx * lQx + dy * lQy) * ir + lC * dcoef * dot * ir;
        gx += S * coef * lQx + lC * coef * vxij + cq * dx;
        gy += S * coef * lQy + lC * coef * vyij + cq * dy;
        gvx += lC * dWx;
        gvy += lC * dWy;
        if (dot < 0.f) {
          const float f = lQdW * dPi_dmu * hb * iden;
          const float c2 = 2.0f * dot * iden;
          gx += f * (vxij - c2 * dx);
          gy += f * (vyij - c2 * dy);
          gvx += f * dx;
          gvy += f * dy;
          gal += mj * (lAxk * dWx + lAyk * dWy) * (mu * cbar * irbar);
        }
        grho += lQdW * (dothk - 0.5f * Pi * irbar);
      } else if (r <= r0 && r > 1e-12f) {
        // boundary pair: Lennard-Jones force and the wall load
        const float s = r0 * ir;
        float sp1, sp2;
        if (ap.lj_42) {
          sp2 = s * s;
          sp1 = sp2 * sp2;
        } else {
          sp1 = __powf(s, p1);
          sp2 = __powf(s, p2);
        }
        const float ir2 = ir * ir;
        const float phi = (sp1 - sp2) * ir2;
        const float dphi = ((-p1 - 2.0f) * sp1 + (p2 + 2.0f) * sp2) * ir2 * ir;
        const float zx = lAxk - ((ap.omega != 0.0 && Aj.x >= ap.wall_x) ? omega_m : 0.f), zy = lAyk;
        const float c = dphi * (dx * zx + dy * zy) * ir;
        gx += D * (phi * zx + c * dx);
        gy += D * (phi * zy + c * dy);
      }
    });
  }
  group_sum<G>(gx);
  group_sum<G>(gy);
  group_sum<G>(gvx);
  group_sum<G>(gvy);
  group_sum<G>(grho);
  group_sum<G>(gal);
  if (k >= ap.n || threadIdx.x % G != 0) return;
  P.xhb[i] = f2d(gx);
  P.yhb[i] = f2d(gy);
  P.vxhb[i] = f2d(gvx);
  P.vyhb[i] = f2d(gvy);
  P.rhohb[i] = f2d(grho);
  P.alb[i] = f2d(gal);
}

// lambda_A = dt vb' + ab', lambda_D = dt rhob' + drhob' (zero for non-fluid)
__global__ void k_adj_pre(const int8_t *__restrict__ label, long long n, double dt, const double *vxb,
                          const double *vyb, const double *rhob, const double *axb, const double *ayb,
                          const double *drhob, double *lax, double *lay, double *lad) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (!is_fluid(label[i])) {
    lax[i] = lay[i] = lad[i] = 0.0;
    return;
  }
  lax[i] = dt * vxb[i] + axb[i];
  lay[i] = dt * vyb[i] + ayb[i];
  lad[i] = dt * rhob[i] + drhob[i];
}

// the half state of step S (PEC.predict's update, src/Integrators/PEC.py:32-60)
// into the scratch particle set; m, h and label are copied
__global__ void k_adj_half(StepArgs s, StepArgs h, double dt) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s.n) return;
  const int8_t lab = s.label[i];
  const_cast<int8_t *>(h.label)[i] = lab;  // the scratch set is writable
  h.m[i] = s.m[i];
  h.h[i] = s.h[i];
  const double hdt = 0.5 * dt;
  if (is_fluid(lab)) {
    h.x[i] = s.x[i] + hdt * s.vx[i];
    h.y[i] = s.y[i] + hdt * s.vy[i];
    h.vx[i] = s.vx[i] + hdt * s.ax[i];
    h.vy[i] = s.vy[i] + hdt * s.ay[i];
    double rho = s.rho[i] + hdt * s.drho[i];
    h.rho[i] = rho;
  } else {
    h.x[i] = s.x[i];
    h.y[i] = s.y[i];
    h.vx[i] = s.vx[i];
    h.vy[i] = s.vy[i];
    h.rho[i] = s.rho[i];
  }
}

// state adjoint update of the step (see the top of the file); the *b arrays
// hold the adjoint of S' on entry and that of S on exit; alphab accumulates
__global__ void k_adj_post(const int8_t *__restrict__ label, long long n, double dt, double *xb, double *yb,
                           double *vxb, double *vyb, double *rhob, double *axb, double *ayb, double *drhob,
                           const double *xhb, const double *yhb, const double *vxhb, const double *vyhb,
                           const double *rhohb, const double *alb, double *alphab) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  alphab[i] += alb[i];
  if (!is_fluid(label[i])) return;
  const double hdt = 0.5 * dt;
  const double vhx = vxhb[i] + dt * xb[i], vhy = vyhb[i] + dt * yb[i];
  xb[i] += xhb[i];
  yb[i] += yhb[i];
  vxb[i] += hdt * xhb[i] + vhx;
  vyb[i] += hdt * yhb[i] + vhy;
  axb[i] = hdt * vhx;
  ayb[i] = hdt * vhy;
  rhob[i] += rhohb[i];
  drhob[i] = hdt * rhohb[i];
}

// Sum of v[0 .. n) in a fixed order (one block): each thread four partial sums
// over its stride, so that four loads are in flight, then shuffles.
constexpr int kSumThreads = 1024;
__global__ void __launch_bounds__(kSumThreads) k_sum_fixed(const double *__restrict__ v, long long n, double *out) {
  step_kernel_entry();
  __shared__ double red[32];
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  for (long long i = threadIdx.x; i < n; i += 4 * kSumThreads) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const long long j = i + q * kSumThreads;
      if (j < n) s[q] += v[j];
    }
  }
  double t = (s[0] + s[1]) + (s[2] + s[3]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x < 32) {
    t = red[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (threadIdx.x == 0) *out = t;
  }
}

void launch_sum_fixed(const double *v, long long n, double *out, cudaStream_t st) {
  launch_pdl(k_sum_fixed, dim3(1), dim3(kSumThreads), 0, st, v, n, out);
}

void launch_adjoint_step(const StepArgs &s, const StepArgs &h, const WsPtrs &w, const sph_config_t &cfg,
                         const sph_wcsph_t &wc, const sph_adjoint_t &adj, cudaStream_t st) {
  const long long n = s.n;
  const double dt = cfg.dt_fixed;
  const unsigned nb = nblocks(n);
  k_adj_pre<<<nb, kBlock, 0, st>>>(s.label, n, dt, adj.vxb, adj.vyb, adj.rhob, adj.axb, adj.ayb, adj.drhob, adj.lax,
                                   adj.lay, adj.lad);
  if (!adj.reuse_build) {
    k_adj_half<<<nb, kBlock, 0, st>>>(s, h, dt);
    // neighbour build and FP64 records of the half state (the forward's own passes)
    launch_bounds(h, w, cfg, wc, kStageNone, true, nullptr, nullptr, st);
    launch_build(h, w, cfg, wc, st);
    sph_config_t c64 = cfg;
    c64.precision = SPH_PREC_FP64;
    launch_records(h, w, c64, wc, true, false, false, st);
  }
  AdjPtrs P;
  P.rec0 = w.rec0;
  P.r64a = w.rec64a;
  P.fix = reinterpret_cast<const longlong2 *>(w.rec1);
  P.r64b = w.rec64b;
  P.perm = w.perm;
  P.keys_sorted = w.keys_sorted;
  P.meta = w.meta;
  P.cstart = w.cstart;
  P.grid = w.grid;
  P.ctrl = w.ctrl;
  P.lax = adj.lax;
  P.lay = adj.lay;
  P.lad = adj.lad;
  P.xhb = adj.xhb;
  P.yhb = adj.yhb;
  P.vxhb = adj.vxhb;
  P.vyhb = adj.vyhb;
  P.rhohb = adj.rhohb;
  P.alb = adj.alb;
  AdjParams ap;
  ap.alpha = wc.alpha;
  ap.beta = wc.beta;
  ap.co = wc.co;
  ap.r0 = lj_reach(wc);
  ap.D = wc.D;
  ap.p1 = wc.p1;
  ap.p2 = wc.p2;
  ap.lj_42 = (wc.p1 == 4.0 && wc.p2 == 2.0) ? 1 : 0;
  ap.gamma = wc.gamma;
  ap.B = wc.B;
  ap.inv_rho0 = 1.0 / wc.rho0;
  ap.omega = adj.omega;
  ap.wall_x = adj.wall_x;
  ap.dt = dt;
  ap.n = n;
  const Pair64 c = pair64_consts(cfg, wc);
  const int lanes = lanes_per_query(n, cfg.kernel, true, true);
  auto go = [&](auto kern, auto l) {
    constexpr int K = decltype(kern)::value, G = decltype(l)::value;
    const unsigned nbp = nblocks(n * G, kAdjBlock);
    if (cfg.precision == SPH_PREC_MIXED) k_pair_adjoint_mixed<K, G><<<nbp, kAdjBlock, 0, st>>>(P, ap);
    else k_pair_adjoint<K, G><<<nbp, kAdjBlock, 0, st>>>(P, ap, c);
  };
  auto go_lanes = [&](auto kern) {
    if (lanes == 8) go(kern, std::integral_constant<int, 8>());
    else if (lanes == 4) go(kern, std::integral_constant<int, 4>());
    else go(kern, std::integral_constant<int, 1>());
  };
  if (cfg.kernel == SPH_KERNEL_CUBIC) go_lanes(std::integral_constant<int, SPH_KERNEL_CUBIC>());
  else if (cfg.kernel == SPH_KERNEL_WENDLAND) go_lanes(std::integral_constant<int, SPH_KERNEL_WENDLAND>());
  else go_lanes(std::integral_constant<int, SPH_KERNEL_GAUSSIAN>());
  k_adj_post<<<nb, kBlock, 0, st>>>(s.label, n, dt, adj.xb, adj.yb, adj.vxb, adj.vyb, adj.rhob, adj.axb, adj.ayb,
                                    adj.drhob, adj.xhb, adj.yhb, adj.vxhb, adj.vyhb, adj.rhohb, adj.alb, adj.alphab);
}

}  // namespace sph
