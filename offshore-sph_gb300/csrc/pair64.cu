// pair64.cu -- the FP64 form of the fused pair interaction (the physics of
// pair.cu's header comment, in FP64 arithmetic).
//
// What bounds it: the FP64 pipe.  It takes 16 cycles per warp instruction
// (2 lanes per SM and cycle), so one FP64 operation costs as much issue time
// as some sixty FP32 or integer ones.  So whatever has a cheap equal goes to the
// other pipes (fp64_ops.cuh):
//   - candidates are filtered in FP32 (padded) and compared on the integer
//     pipe (positive doubles order like their bits);
//   - position differences and the squared distance come from 64-bit integer
//     positions (except for coordinates that these cut), reciprocals and square
//     roots from 64-bit fixed-point Newton steps, each rounded once.  The neighbour test q = r / h_ij <= 3
//     (NNLinkedList.py:74) is redone with correctly rounded operations where
//     an estimate could decide it differently;
//   - with a uniform fluid h (Solver(h=...)) and beta = 0, the cubic's gradient
//     factor and the viscosity's reciprocal are fixed-point too, and boundary
//     neighbours beyond the Lennard-Jones reach are not listed (without XSPH
//     they contribute nothing).
// A pair of the cubic spline so takes 11 FP64 operations instead of about 90.
// 1M-fluid dam break, pair stage: 3.67 ms at 90, 1.27 ms at 31 (Halley steps and
// launch-constant gradient polynomials in FP64), 0.65 ms now; the FP64 pipe
// is busy 63% of it and 44% of the issue slots are used.  20 steps of 3200
// fluid particles, where latency decides (several lanes per query): 2.40 ms,
// 0.71 and 0.67.
// A pair's terms are at least as close to the exact ones as the reference's
// formulas with every operation rounded to 64 bits.
#include <type_traits>

#include "fp64_ops.cuh"
#include "pair_common.cuh"

namespace sph {

struct Acc64 {
  double dd = 0.0, ax = 0.0, ay = 0.0, bx = 0.0, by = 0.0, sx = 0.0, sy = 0.0, fr = 0.0;
};

// The query's state (FP64 records).
struct Query64 {
  double x, y, vx, vy, rho, oth, h;
  longlong2 p;  // integer position
  int fix_s;
  bool wide;    // FP64 differences: its integers are cut, or their differences could wrap
};

// One listed candidate j of query q: the exact support test, then
// continuity, momentum with artificial viscosity, the Lennard-Jones boundary
// force and XSPH.  UH: every fluid h is c.h and beta = 0.
// FIX: differences from the integer positions.
template <int KERNEL, bool UH, bool FIX>
__device__ __forceinline__ void pair64(Acc64 &s, const Query64 &q, const Pair64 &c, const PairParams &pp,
                                       longlong2 pj, const double4_32a &A, const double4_32a &B) {
  constexpr bool gauss = KERNEL == SPH_KERNEL_GAUSSIAN;
  PairGeom geo;
  if constexpr (FIX) geo = q.wide || fix_cut(pj) ? pair_geom_wide(q.x - A.x, q.y - A.y) : pair_geom(q.p, pj, q.fix_s);
  else geo = pair_geom_fp64(q.x - A.x, q.y - A.y);
  const double dx = geo.dx, dy = geo.dy, d2 = geo.d2;
  const bool fluid = !signbit(B.w);
  if (fluid) {
    double coef, w = 0.0, hij = c.h, ih = c.ih;
    if constexpr (UH) {
      if constexpr (gauss) {
        if (!le_bits(d2, c.lim_lo) && (!le_bits(d2, c.lim_hi) || !near_exact(q.x - A.x, q.y - A.y, hij))) return;
        const double e = exp2_neg(geo.v, c.l2e);
        coef = le_bits(d2, c.h2) ? 0.0 : e;  // scaled in the sum
        if (c.xsph) w = c.al * e;
      } else {
        if (!le_bits(d2, c.lim)) return;  // W and its gradient are 0 at q >= 2
        const bool tiny = le_bits(d2, 1e-20);  // r < 1e-10: no gradient
        if (KERNEL == SPH_KERNEL_CUBIC) {
          coef = cubic_g(geo.v, c.ihf, c.hf);  // scaled in the sum
          if (c.xsph) {
            double r, ir;
            sqrt_rsqrt64(geo.v, r, ir);
            if (tiny) r = 0.0;
            const double qq = r * ih, t = fma(c.o_rl, r, fma(c.o_r, r, 2.0));
            w = le_bits(d2, c.h2) ? c.al * (1.0 - 1.5 * (qq * qq) * (1.0 - 0.5 * qq)) : c.al * 0.25 * (t * t * t);
          }
        } else {
          // (1 + 2.5 q) = 6 - 5 in
          const double in = wendland_in(geo.v, c.ihf), in2 = in * in;
          coef = (in2 * in2) * (in * fma(-5.0, in, 6.0));  // scaled in the sum
          if (c.xsph) {
            const double qq = fma(-2.0, in, 2.0);
            w = c.al * (in2 * in2 * in2 * ((35.0 / 12.0) * qq * qq + 3.0 * qq + 1.0));
          }
        }
        if (tiny) coef = 0.0;
      }
    } else {
      hij = half_exact(q.h + B.w);  // both positive or zero
      if (!(__double2hiint(hij) > 0)) return;  // q = r / 0
      double ihl, ih2, ih4;
      rcp_powers(hij, ih, ihl, ih2, ih4);
      if constexpr (gauss) {
        const double z = d2 * ih2;
        if (!le_bits(z, 9.0 * (1.0 - 1e-9)) && (!le_bits(z, 9.0 * (1.0 + 1e-9)) || !near_exact(q.x - A.x, q.y - A.y, hij))) return;
        const double e = exp_neg(z);
        coef = le_bits(d2, 1e-24 * ih2) ? 0.0 : (-2.0 * kInvPi) * ih4 * e;
        if (c.xsph) w = kInvPi * ih2 * e;
      } else {
        double r, ir;
        sqrt_rsqrt64(geo.v, r, ir);
        const bool tiny = le_bits(d2, 1e-20);
        if (tiny) r = 0.0;
        const double qq = r * ih;
        if (!le_bits(qq, 2.0)) return;
        const double t = fma(-r, ihl, fma(-r, ih, 2.0)), t2 = t * t;  // 2 - q
        if (KERNEL == SPH_KERNEL_CUBIC) {
          const double al = kCubicFac * ih2;
          if (le_bits(qq, 1.0)) {
            coef = (kCubicFac * ih4) * fma(2.25, qq, -3.0);
            if (c.xsph) w = al * (1.0 - 1.5 * (qq * qq) * (1.0 - 0.5 * qq));
          } else {
            coef = (-0.75 * kCubicFac) * ih4 * (hij * ir) * t2;
            if (c.xsph) w = al * 0.25 * (t2 * t);
          }
        } else {
          const double t5 = t2 * t2 * t;  // 32 (1 - q / 2)^5
          coef = (kWendFac / 32 * ih4) * t5 * fma(-35.0 / 3.0, qq, -14.0 / 3.0);
          if (c.xsph) w = (kWendFac / 64 * ih2) * (t5 * t) * ((35.0 / 12.0) * qq * qq + 3.0 * qq + 1.0);
        }
        if (tiny) coef = 0.0;
      }
    }
    const double vx = q.vx - A.z, vy = q.vy - A.w;
    const double dot = fma(vy, dy, vx * dx);
    const double mc = B.x * coef;
    s.dd = fma(mc, dot, s.dd);
    double S = q.oth + B.z;
    const double rs = q.rho + B.y;  // 2 rho_ij
    if (negative_bits(dot)) {
      if constexpr (UH) {
        const double inv = rcp_sum_prod(geo.v, c.hb2f, rs, d2, c.hb2);
        S = fma(c.pic * inv, dot, S);
      } else {
        // mu = h v.r / (r^2 + 0.01 h^2), Pi = mu (beta mu - alpha c_ij) / rho_ij
        const double hb = half_exact(q.h + hij);
        const double den = fma(0.01 * hb, hb, d2);
        const double inv = rcp64(den * rs);  // 1 / (den rs)
        const double t = 2.0 * hb * dot * inv;  // mu / rho_ij
        if (pp.beta == 0.0) S = fma(t, -0.5 * pp.alpha * pp.co, S);
        else S = fma(t, fma(pp.beta, hb * dot * (inv * rs), -0.5 * pp.alpha * pp.co), S);
      }
    }
    const double f = mc * S;
    s.ax = fma(-f, dx, s.ax);
    s.ay = fma(-f, dy, s.ay);
    if (c.xsph) {
      const double k = (-2.0 * pp.eps) * B.x * w * rcp64(rs);
      s.sx = fma(k, vx, s.sx);
      s.sy = fma(k, vy, s.sy);
    }
    return;
  }
  // a boundary neighbour: Lennard-Jones at 1e-12 < r <= r0 (the force is 0 at
  // r0), and XSPH, which takes every neighbour (a massless one adds 0)
  const bool lj = le_bits(d2, c.r02) && !le_bits(d2, 1e-24);
  const bool xs = c.xsph && (B.x != 0.0);
  if (!lj && !xs) return;
  const double hj = fabs(B.w);
  const double hij = 0.5 * (q.h + hj);
  if (!(c.lj_free && lj) || xs) {  // the neighbour test
    const double t = 3.0 * hij, t2 = t * t;
    if (!le_bits(d2, t2 * (1.0 - 1e-9)) && (!le_bits(d2, t2 * (1.0 + 1e-9)) || !near_exact(q.x - A.x, q.y - A.y, hij))) return;
    if (!(hij > 0.0)) return;
  }
  if (lj) {
    const double ir2 = rcp64(d2);
    double t;
    if (pp.lj_42) {
      const double f2 = c.r02 * ir2;
      t = fma(f2, f2, -f2);
    } else {
      const double frac = pp.r0 / __dsqrt_rn(d2);
      t = pow(frac, pp.p1) - pow(frac, pp.p2);
    }
    const double fac = pp.D * t * ir2;
    s.bx = fma(fac, dx, s.bx);
    s.by = fma(fac, dy, s.by);
    if (pp.fr && A.x >= pp.wall_x) s.fr = fma(fac, dx, s.fr);
  }
  if (xs) {
    const double r = __dsqrt_rn(d2);
    const double w = KERNEL == SPH_KERNEL_CUBIC ? cubic_w(r, hij)
                                                : (KERNEL == SPH_KERNEL_WENDLAND ? wendland_w(r, hij) : gauss_w(r, hij));
    const double k = (-2.0 * pp.eps) * B.x * w * rcp64(q.rho + B.y);
    s.sx = fma(k, q.vx - A.z, s.sx);
    s.sy = fma(k, q.vy - A.w, s.sy);
  }
}

// ---------------------------------------------------------------------------
// The kernel: G lanes per query (for_neighbours).
// ---------------------------------------------------------------------------
template <int KERNEL, bool UH>
struct Near64 {
  const float4 *rec0;
  const int2 *meta;
  const DevGrid &g;
  float4 Qi;
  int2 qref;
  unsigned int k;
  float rf2, r0f, pad;
  bool filter, xsph;
  __device__ __forceinline__ float4 load(unsigned int j) const { return __ldg(rec0 + j); }
  __device__ __forceinline__ bool test(unsigned int j, float4 qj) const {
    if (j == k) return false;  // the particle itself contributes zero
    if (filter && !in_ref_stencil(meta, j, g, qref)) return false;
    const float dx = Qi.x - qj.x, dy = Qi.y - qj.y;
    const float d2 = dx * dx + dy * dy;
    if (UH && !signbit(qj.z)) return d2 <= rf2;
    const float hij = 0.5f * (Qi.z + fabsf(qj.z));
    float reach = (float)Support<KERNEL>::q * 1.000002f * hij;
    if (signbit(qj.z)) {
      const float lj = fminf(r0f, 3.0f * hij) * 1.000002f;
      reach = xsph ? fmaxf(reach, lj) : lj;
    }
    const float rp = reach + pad;
    return d2 <= rp * rp;
  }
};

template <int KERNEL, bool UH, int G>
__global__ void __launch_bounds__(kPairBlock, G == 8 ? 4 : kPair64Blocks)
    k_pair64(StepArgs a, PairPtrs P, PairParams pp, Pair64 c, double *dt_out, double *dt_hist) {
  step_kernel_entry();
  // Integer differences save FP64 issue time and lengthen a pair's chain: not
  // where a query's latency is the time (20 steps of 3200 fluid particles 672
  // us without, 690 with; 4 steps of 1M: 3737 and 3515)
  constexpr bool kFix = G < 8;
  constexpr int kCap = list_words<G>(ListCap<KERNEL>::value);
  __shared__ unsigned int lists[kCap * kPairBlock / G];
  const DevGrid &g = *P.grid;
  const int tid = threadIdx.x;
  const int gl = tid % G;
  const long long k = ((long long)blockIdx.x * kPairBlock + tid) / G;
  unsigned long long ea = kEncMaxId;
  bool act = k < pp.n;
  const float4 Qi = act ? P.rec0[k] : make_float4(0.f, 0.f, -1.f, 0.f);  // x_hi, y_hi, h (signed), m
  const float hif = Qi.z;
  act = act && !signbit(hif);
  if (G > 1 ? __any_sync(0xffffffffu, act) : act) {
    const bool filter = g.mode == 1 && (g.need_filter || P.ctrl->alias_count > 0);
    const long long kq = act ? k : 0;
    const int i = P.perm[kq];
    const int2 qref = P.meta[kq];
    const int qkey = P.keys_sorted[kq];
    const bool slow = qref.x >= g.ncx || !(hif > 0.f);
    const int W = g.mode == 0 ? 1 : (slow ? g.wide : g.wt);
    const double4_32a A = P.r64a[kq], B = P.r64b[kq];
    const longlong2 *fix = reinterpret_cast<const longlong2 *>(P.rec1);
    const Query64 q = {A.x, A.y, A.z, A.w, B.y, B.z, B.w, fix[kq], g.fix_s,
                       (kFix && fix_cut(fix[kq])) || g.pad_e > 0.5f * (float)g.r_search};
    Acc64 s;
    // the FP32 test: the padded reach of the pair's h (kernel support; a
    // boundary neighbour without XSPH: the Lennard-Jones reach min(r0, 3 h_ij))
    const float SK = (float)Support<KERNEL>::q * 1.000002f;
    const float r0f = (float)pp.r0, pad = g.pad_e;
    const float rf = SK * hif + pad, rf2 = rf * rf;
    const Near64<KERNEL, UH> near{P.rec0, P.meta, g, Qi, qref, (unsigned int)kq, rf2, r0f, pad, filter, c.xsph != 0};
    const Stencil sten(g, qref, qkey, W);
    for_neighbours<G, kCap, kPairBlock>(sten, P.cstart, act, lists, near, [&](unsigned int j) {
      pair64<KERNEL, UH, kFix>(s, q, c, pp, kFix ? fix[j] : longlong2(), P.r64a[j], P.r64b[j]);
    });
    if (UH) {
      s.dd *= c.scale;
      s.ax *= c.scale;
      s.ay *= c.scale;
    }
    s.ax += s.bx;
    s.ay += s.by;
    group_sum<G>(s.dd);
    group_sum<G>(s.ax);
    group_sum<G>(s.ay);
    if (c.xsph) {
      group_sum<G>(s.sx);
      group_sum<G>(s.sy);
    }
    if (pp.fr) group_sum<G>(s.fr);
    if (act && gl == 0) {
      // the reference's set always holds the particle itself, except for the
      // slow queries, whose set size is counted exactly
      if (!slow || exact_count(a, P.perm, g, qref, qkey, W, g.mode == 1, P.meta, P.cstart, q.x, q.y, q.h) > 0) {
        const double axf = s.ax, ayf = s.ay - 9.81;
        a.drho[i] = c.sumdens ? 0.0 : s.dd;
        if (c.xsph || pp.write_xsph || slow || P.ctrl->xsph_left) {
          a.xsphx[i] = c.xsph ? q.vx + s.sx : 0.0;
          a.xsphy[i] = c.xsph ? q.vy + s.sy : 0.0;
        }
        ea = enc_d(accel2(axf, ayf));
        a.ax[i] = axf;
        a.ay[i] = ayf;
        if (pp.fr) pp.fr[i] = -B.x * s.fr;
      } else {
        ea = enc_d(accel2(a.ax[i], a.ay[i]));  // keeps its previous values (SolverTools.py:150-153)
        if (pp.fr) pp.fr[i] = 0.0;
        if (!c.xsph && pp.write_xsph) P.ctrl->xsph_left = 1u;
      }
    }
  }
  if (pp.do_dt) timestep_epilogue(P.ctrl, ea, pp.co, pp.cfl_c, pp.cfl_f, dt_out, dt_hist);
}

template <int KERNEL, bool UH>
static void pair64_launch(const StepArgs &a, const WsPtrs &w, const PairParams &pp, const Pair64 &c, double *dt_out,
                          double *dt_hist, cudaStream_t st) {
  auto go = [&](auto lanes) {
    constexpr int G = decltype(lanes)::value;
    launch_pdl(k_pair64<KERNEL, UH, G>, dim3(nblocks(a.n * G, kPairBlock)), dim3(kPairBlock), 0, st, a, pair_ptrs(w), pp,
               c, dt_out, dt_hist);
  };
  const int lanes = lanes_per_query(a.n, KERNEL, UH);
  if (lanes == 8) go(std::integral_constant<int, 8>());
  else if (lanes == 4) go(std::integral_constant<int, 4>());
  else go(std::integral_constant<int, 1>());
}

void launch_pair64(const StepArgs &a, const WsPtrs &w, const sph_config_t &cfg, const sph_wcsph_t &wc,
                   PairParams pp, double *dt_out, double *dt_hist, cudaStream_t st) {
  pp.r0 = lj_reach(wc);
  const Pair64 c = pair64_consts(cfg, wc);
  const bool uh = cfg.h_fixed > 0.0 && wc.beta == 0.0;
  auto go = [&](auto kern) {
    constexpr int K = decltype(kern)::value;
    if (uh) pair64_launch<K, true>(a, w, pp, c, dt_out, dt_hist, st);
    else pair64_launch<K, false>(a, w, pp, c, dt_out, dt_hist, st);
  };
  if (cfg.kernel == SPH_KERNEL_CUBIC) go(std::integral_constant<int, SPH_KERNEL_CUBIC>());
  else if (cfg.kernel == SPH_KERNEL_WENDLAND) go(std::integral_constant<int, SPH_KERNEL_WENDLAND>());
  else go(std::integral_constant<int, SPH_KERNEL_GAUSSIAN>());
}

}  // namespace sph
