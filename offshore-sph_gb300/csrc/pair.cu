// pair.cu -- the fused pair interaction of the WCSPH step, mixed form (the
// FP64 form's kernel is in pair64.cu).
//
// One thread per cell-sorted fluid particle i evaluates in one pass
// everything _loop computes per particle (src/Tools/SolverTools.py:143-173):
// the kernel value and gradient (src/Kernels/CubicSpline.py,
// src/Kernels/Gaussian.py), continuity (src/Equations/Continuity.py),
// momentum with artificial viscosity and gravity (src/Equations/Momentum.py,
// src/Methods/WCSPH.py:151-169), the Lennard-Jones boundary force
// (src/Equations/BoundaryForce.py) and XSPH (src/Equations/XSPH.py).  The
// TimeStep of the next step (src/Equations/TimeStep.py:7-91) is fused into
// the epilogue.
//
// Each thread alternates two phases so that the expensive physics runs over
// dense lists instead of sparse, divergent candidate loops:
//   1. walk the stencil rows with one 16-byte load and a conservative FP32
//      radius test per candidate (hi parts of the positions, padded by their
//      truncation bound) and append the survivors to a per-thread list in
//      shared memory;
//   2. evaluate the pair physics over the list, after the exact test.
// Phase 2 runs in FP32 on double-float differences of the FP64 state.
#include <math.h>

#include <type_traits>

#include "fp64_ops.cuh"
#include "pair_common.cuh"

namespace sph {

// ---------------------------------------------------------------------------
// Mixed-form pair physics, shared by the tile kernel and the global-path
// kernel so that both give bit-identical sums for the same candidate order.
// ---------------------------------------------------------------------------
struct MixedAcc {
  float fd = 0.f, fax = 0.f, fay = 0.f, fbx = 0.f, fby = 0.f, fsx = 0.f, fsy = 0.f;
};

// two FP32 operations in one instruction, each rounded as its scalar form
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n add.rn.ftz.f32x2 z, x, y;\n"
      " mov.b64 {%0, %1}, z;\n}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  float2 d;
  asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n sub.rn.ftz.f32x2 z, x, y;\n"
      " mov.b64 {%0, %1}, z;\n}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }
// differences of the double-float positions and velocities
__device__ __forceinline__ float2 diff_pos(float4 Qi, float4 Ri, float4 qj, float4 rj) {
  return add2(sub2(lo2(Qi), lo2(qj)), sub2(lo2(Ri), lo2(rj)));
}
__device__ __forceinline__ float2 diff_vel(float4 Vi, float4 vj) {
  return add2(sub2(lo2(Vi), lo2(vj)), sub2(hi2(Vi), hi2(vj)));
}

// One FLUID neighbour j of fluid query i under a uniform fluid h and beta = 0
// (see UniformQ): the same equations as mixed_pair's fluid branch with the
// per-pair h arithmetic taken out.
template <int KERNEL, bool XSPH, bool SUMDENS>
__device__ __forceinline__ void mixed_fluid_uh(MixedAcc &acc, const MixedConsts &c, const UniformQ &u, float4 Qi,
                                               float4 Ri, float4 Vi, float4 qj, float4 rj, const float4 *vjp) {
  const float2 d = diff_pos(Qi, Ri, qj, rj);
  const float dx = d.x, dy = d.y;
  const float d2 = dx * dx + dy * dy;
  if (d2 > u.lim) return;
  const float2 v = diff_vel(Vi, *vjp);
  const float vxij = v.x, vyij = v.y;
  // 1/r, and 0 below r = 1e-10 (d2 = 1e-20), where the kernel gradient of
  // the 2h kernels is taken as 0: the guard on the gradient folds into it
  const bool g2h = KERNEL == SPH_KERNEL_CUBIC || KERNEL == SPH_KERNEL_WENDLAND;
  const float inv_r = d2 >= (g2h ? 1e-20f : 0.f) && d2 > 0.f ? rsqrtf(d2) : 0.f;
  const float r = d2 * inv_r;
  const float q = r * u.inv_h;
  float w = 0.f, coef;
  if (KERNEL == SPH_KERNEL_CUBIC) {
    const float t2 = fmaxf(2.0f - q, 0.f);
    const bool outer = q > 1.0f;
    if (XSPH) w = outer ? u.al * 0.25f * (t2 * t2 * t2) : u.al * (1.0f - 1.5f * (q * q) * (1.0f - 0.5f * q));
    const float g = outer ? u.g0 * (t2 * t2) : q * fmaf(u.g1, q, u.g2);
    coef = g * inv_r;
  } else if (KERNEL == SPH_KERNEL_WENDLAND) {
    const float inner = fmaxf(1.0f - 0.5f * q, 0.f);
    const float i2 = inner * inner, i5 = i2 * i2 * inner;
    if (XSPH) w = u.al * (i5 * inner) * ((35.0f / 12.0f) * q * q + 3.0f * q + 1.0f);
    coef = i5 * q * fmaf(u.g1, q, u.g0) * inv_r;
  } else {
    const float e = __expf(-q * q);
    if (XSPH) w = u.al * e;
    coef = r * u.h > 1e-12f ? u.g0 * e : 0.f;
  }
  const float dwx = coef * dx, dwy = coef * dy;
  const float mj = qj.w;
  if (!SUMDENS) acc.fd = fmaf(mj, vxij * dwx + vyij * dwy, acc.fd);
  const float dot = vxij * dx + vyij * dy;
  const float rs = Ri.z + rj.z;  // 2 rho_ij
  const float PI = dot < 0.f ? u.pic * dot * __fdividef(1.0f, (d2 + u.hb2) * rs) : 0.f;
  const float fac = mj * (Ri.w + rj.w + PI);
  acc.fax = fmaf(-fac, dwx, acc.fax);
  acc.fay = fmaf(-fac, dwy, acc.fay);
  if (XSPH) {
    const float fx = -c.eps * mj * w * __fdividef(2.0f, rs);
    acc.fsx = fmaf(fx, vxij, acc.fsx);
    acc.fsy = fmaf(fx, vyij, acc.fsy);
  }
}

// One boundary neighbour j without XSPH: the Lennard-Jones force alone
// (BoundaryForce.py:6-42), at r <= min(r0, 3 h_ij).
__device__ __forceinline__ void mixed_boundary(MixedAcc &acc, const MixedConsts &c, float4 Qi, float4 Ri, float4 qj,
                                               float4 rj) {
  const float2 d = diff_pos(Qi, Ri, qj, rj);
  const float d2 = d.x * d.x + d.y * d.y;
  const float hij = 0.5f * (Qi.z + fabsf(qj.z));
  if (d2 > fminf(c.r02f, 9.0f * (hij * hij)) || !(d2 > 1e-24f)) return;
  const float ir2 = __fdividef(1.0f, d2);
  const float f2 = c.r02f * ir2;
  const float fac = c.D * (f2 * f2 - f2) * ir2;
  acc.fbx = fmaf(fac, d.x, acc.fbx);
  acc.fby = fmaf(fac, d.y, acc.fby);
}

// One candidate j of query i: the exact support test, then continuity,
// momentum with artificial viscosity, the Lennard-Jones boundary force and
// XSPH.  Qi/qj: x_hi, y_hi, h (sign bit: non-fluid), m; Ri/rj: x_lo, y_lo,
// rho, p / rho^2; Vi and *vjp: vx_hi, vy_hi, vx_lo, vy_lo (read only when the
// pair is inside the support).
template <int KERNEL, bool XSPH, bool SUMDENS>
__device__ __forceinline__ void mixed_pair(MixedAcc &acc, const MixedConsts &c, float4 Qi, float4 Ri, float4 Vi,
                                           float4 qj, float4 rj, const float4 *vjp) {
  const bool jf = !signbit(qj.z);
  if (!XSPH && !jf) {
    mixed_boundary(acc, c, Qi, Ri, qj, rj);
    return;
  }
  const float hif = Qi.z;
  const float2 d = diff_pos(Qi, Ri, qj, rj);
  const float dx = d.x, dy = d.y;
  const float d2 = dx * dx + dy * dy;
  const float hij = 0.5f * (hif + fabsf(qj.z));
  const float h2 = hij * hij;
  float lim = c.KC * h2;
  if (!jf) lim = fmaxf(lim, fminf(c.r02f, 9.0f * h2));
  if (d2 > lim) return;
  const float2 v = diff_vel(Vi, *vjp);
  const float vxij = v.x, vyij = v.y;
  const float inv_h = __fdividef(1.0f, hij);
  const float inv_r = d2 > 0.f ? rsqrtf(d2) : 0.f;
  const float r = d2 * inv_r;
  const float q = r * inv_h;
  float w, coef;
  if (KERNEL == SPH_KERNEL_CUBIC) {
    const float al = (float)kCubicFac * inv_h * inv_h;
    const float t2 = fmaxf(2.0f - q, 0.f);
    const bool outer = q > 1.0f;
    w = outer ? al * 0.25f * (t2 * t2 * t2) : al * (1.0f - 1.5f * (q * q) * (1.0f - 0.5f * q));
    const float gq = outer ? -0.75f * (t2 * t2) : -3.0f * q * (1.0f - 0.75f * q);
    coef = r >= 1e-10f ? al * gq * inv_h * inv_r : 0.f;
  } else if (KERNEL == SPH_KERNEL_WENDLAND) {
    const float al = (float)kWendFac * inv_h * inv_h;
    const float inner = fmaxf(1.0f - 0.5f * q, 0.f);
    const float i2 = inner * inner, i5 = i2 * i2 * inner;
    w = al * (i5 * inner) * ((35.0f / 12.0f) * q * q + 3.0f * q + 1.0f);
    const float gq = i5 * (-14.0f / 3.0f) * q * (1.0f + 2.5f * q);
    coef = r >= 1e-10f ? al * gq * inv_h * inv_r : 0.f;
  } else {
    const float ac = (float)kInvPi * inv_h * inv_h;
    const float e = __expf(-q * q);
    w = ac * e;
    coef = r * hij > 1e-12f ? -2.0f * ac * e * inv_h * inv_h : 0.f;
  }
  const float dwx = coef * dx, dwy = coef * dy;
  const float mj = qj.w;
  if (jf) {
    if (!SUMDENS) acc.fd = fmaf(mj, vxij * dwx + vyij * dwy, acc.fd);
    const float dot = vxij * dx + vyij * dy;
    const float hb = 0.5f * (hif + hij);
    const float mu = hb * dot * __fdividef(1.0f, d2 + 0.01f * hb * hb);
    const float PI = dot < 0.f ? mu * (c.beta * mu - c.alpha * 0.5f * c.co) * __fdividef(2.0f, Ri.z + rj.z) : 0.f;
    const float fac = mj * (Ri.w + rj.w + PI);
    acc.fax = fmaf(-fac, dwx, acc.fax);
    acc.fay = fmaf(-fac, dwy, acc.fay);
  } else if (d2 <= c.r02f && d2 > 1e-24f) {
    const float ir2 = __fdividef(1.0f, d2);
    const float f2 = c.r02f * ir2;
    const float fac = c.D * (f2 * f2 - f2) * ir2;
    acc.fbx = fmaf(fac, dx, acc.fbx);
    acc.fby = fmaf(fac, dy, acc.fby);
  }
  if (XSPH) {
    const float fac = -c.eps * mj * w * __fdividef(2.0f, Ri.z + rj.z);
    acc.fsx = fmaf(fac, vxij, acc.fsx);
    acc.fsy = fmaf(fac, vyij, acc.fsy);
  }
}

// One list entry j of query i: with a uniform fluid h and beta = 0 (UH), fluid
// neighbours take the fast path and the rest (boundary particles) the general
// one.
template <int KERNEL, bool XSPH, bool SUMDENS, bool UH>
__device__ __forceinline__ void mixed_entry(MixedAcc &acc, const MixedConsts &c, const UniformQ &u, float4 Qi,
                                            float4 Ri, float4 Vi, float4 qj, float4 rj, const float4 *vjp) {
  if (UH && !signbit(qj.z))
    mixed_fluid_uh<KERNEL, XSPH, SUMDENS>(acc, c, u, Qi, Ri, Vi, qj, rj, vjp);
  else
    mixed_pair<KERNEL, XSPH, SUMDENS>(acc, c, Qi, Ri, Vi, qj, rj, vjp);
}

// Writes the derivatives of particle i (gravity on y) and returns its encoded
// a^2 for the TimeStep reduction.
template <bool XSPH, bool SUMDENS>
__device__ __forceinline__ unsigned long long mixed_store(const MixedAcc &acc, const StepArgs &a, int i,
                                                          int write_xsph) {
  const float axs = acc.fax + acc.fbx, ays = acc.fay + acc.fby;
  a.ax[i] = f2d(axs);
  a.ay[i] = f2d(ays) - 9.81;
  a.drho[i] = SUMDENS ? 0.0 : f2d(acc.fd);
  if (XSPH) {
    a.xsphx[i] = a.vx[i] + f2d(acc.fsx);
    a.xsphy[i] = a.vy[i] + f2d(acc.fsy);
  } else if (write_xsph) {
    a.xsphx[i] = 0.0;
    a.xsphy[i] = 0.0;
  }
  const float ayg = ays - 9.81f;
  return enc_d(f2d(axs * axs + ayg * ayg));
}

// Global-path evaluation of query slot k (all candidate records read from
// global memory); returns the encoded a^2 of a fluid query, else the max
// identity.  lists: the block's per-thread candidate lists.
template <int KERNEL, bool XSPH, bool SUMDENS, bool UH>
__device__ __forceinline__ unsigned long long pair_query(const StepArgs &a, const PairPtrs &P, const PairParams &pp,
                                                         const DevGrid &g, bool filter, long long k,
                                                         unsigned int (*lists)[kPairBlock], int cell0 = 0) {
  // cell0: global id of grid g's first cell (batched form)
  const unsigned int *cst = P.cstart + cell0;
  constexpr int kListCap = ListCap<KERNEL>::value;
  const int tid = threadIdx.x;
  unsigned long long ea = kEncMaxId;
  const float SK = (float)Support<KERNEL>::q * 1.000002f;  // support / h, padded
  const float r0f = (float)pp.r0;
  const float pad = g.pad_e;
  {
    const float4 Qi = P.rec0[k];  // x_hi, y_hi, h (signed), m
    const float hif = Qi.z;
    if (!signbit(hif)) {
      const int i = P.perm[k];
      const int2 qref = P.meta[k];
      const int qkey = P.keys_sorted[k] - cell0;
      const bool slow = qref.x >= g.ncx || !(hif > 0.f);
      const int W = g.mode == 0 ? 1 : (slow ? g.wide : g.wt);
      const float4 Ri = P.rec1[k], Vi = P.rec2[k];  // x_lo, y_lo, rho, p / rho^2; velocities
      MixedAcc acc;
      const MixedConsts &mc = pp.mc;
      const UniformQ &uq = pp.u;

      // ---- phase 2: pair physics over the list
      auto physics = [&](int cnt) {
        for (int t = 0; t < cnt; t++) {
          const unsigned int j = lists[t][tid];
          mixed_entry<KERNEL, XSPH, SUMDENS, UH>(acc, mc, uq, Qi, Ri, Vi, P.rec0[j], P.rec1[j], P.rec2 + j);
        }
      };

      // ---- phase 1: padded FP32 radius test, append to this thread's list
      const Stencil sten(g, qref, qkey, W);
      int nl = 0;
      for_stencil(sten, cst, [&](unsigned int j) {
        if (j == (unsigned int)k) return;  // the particle itself contributes zero
        if (filter && !in_ref_stencil(P.meta, j, g, qref)) return;
        const float4 qj = P.rec0[j];
        const float dx = Qi.x - qj.x, dy = Qi.y - qj.y;
        const float d2 = dx * dx + dy * dy;
        const float hij = 0.5f * (hif + fabsf(qj.z));
        float reach = SK * hij;
        if (signbit(qj.z)) {
          const float lj = fminf(r0f, 3.0f * hij) * 1.000002f;
          reach = XSPH ? fmaxf(reach, lj) : lj;
        }
        const float rp = reach + pad;
        if (d2 <= rp * rp) {
          lists[nl][tid] = j;
          if (++nl == kListCap) {
            physics(nl);
            nl = 0;
          }
        }
      });
      physics(nl);

      // the reference's set always holds the particle itself, except for the
      // slow queries, whose set size is counted exactly
      const bool any = !slow || exact_count(a, P.perm, g, qref, qkey, W, g.mode == 1, P.meta, cst, a.x[i], a.y[i],
                                            a.h[i]) > 0;
      if (any) {
        ea = mixed_store<XSPH, SUMDENS>(acc, a, i, pp.write_xsph || slow);
      } else {
        ea = enc_d(accel2(a.ax[i], a.ay[i]));  // keeps its previous values (SolverTools.py:150-153)
        if (!XSPH && pp.write_xsph) P.ctrl->xsph_left = 1u;
      }
    }
  }
  return ea;
}

// The queries the tile kernel left over (slot ranges of at most kPairBlock
// slots), on the global path; the last block resets the list and, when asked,
// finishes the TimeStep reduction.
constexpr int kListBlocks = 6;
template <int KERNEL, bool XSPH, bool SUMDENS, bool UH>
__global__ void __launch_bounds__(kPairBlock, kListBlocks)
    k_pair_list(StepArgs a, PairPtrs P, PairParams pp, const int2 *__restrict__ fb, double *dt_out,
                double *dt_hist) {
  step_kernel_entry();
  __shared__ unsigned int lists[ListCap<KERNEL>::value][kPairBlock];
  const unsigned long long both = *(volatile unsigned long long *)&P.ctrl->fb_count;
  const unsigned int cnt = (unsigned int)both;
  // xsph_left, which is set in other steps only
  const bool left = !XSPH && !pp.write_xsph && (both >> 32) != 0ull;
  // only the blocks that have entries take part (at least block 0, which
  // finishes the TimeStep when the list is empty); the rest leave at once.
  // A block that starts after the last participant emptied the list reads
  // 0 and leaves too: the list is emptied only once every participant,
  // itself included, has read the count.
  const unsigned int parts = !left && cnt < gridDim.x ? (cnt > 0u ? cnt : 1u) : gridDim.x;
  if (blockIdx.x >= parts) return;
  if (left)
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < pp.n; k += (long long)gridDim.x * blockDim.x)
      if (!signbit(P.rec0[k].z) && P.rec0[k].z > 0.f && P.meta[k].x < P.grid->ncx) {
        a.xsphx[P.perm[k]] = 0.0;
        a.xsphy[P.perm[k]] = 0.0;
      }
  unsigned long long ea = kEncMaxId;
  if (blockIdx.x < cnt) {
    const DevGrid g = *P.grid;
    const bool filter = g.mode == 1 && (g.need_filter || P.ctrl->alias_count > 0);
    for (unsigned int e = blockIdx.x; e < cnt; e += gridDim.x) {
      const int2 r = fb[e];
      if ((int)threadIdx.x < r.y) {
        const unsigned long long q =
            pair_query<KERNEL, XSPH, SUMDENS, UH>(a, P, pp, g, filter, r.x + threadIdx.x, lists);
        ea = q > ea ? q : ea;
      }
    }
  }
  __syncthreads();
  // the last participant empties the fallback list (with the TimeStep
  // epilogue when there is one)
  if (pp.do_dt) {
    timestep_epilogue(P.ctrl, ea, pp.co, pp.cfl_c, pp.cfl_f, dt_out, dt_hist, &P.ctrl->fb_count, parts);
  } else if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&P.ctrl->fb_done, 1u) == parts - 1) {
      P.ctrl->fb_count = 0;
      P.ctrl->fb_done = 0;
    }
  }
}

// ---------------------------------------------------------------------------
// Summation density (SolverTools.py:129-140, SummationDensity.py:5-13):
// rho_i = sum over fluid neighbours (itself included) of m_j W(r, h_ij).
// ---------------------------------------------------------------------------
template <int KERNEL, bool MIXED>
__global__ void __launch_bounds__(kPairBlock) k_sumdens(StepArgs a, PairPtrs P, long long n) {
  const DevGrid g = *P.grid;
  const bool filter = g.mode == 1 && (g.need_filter || P.ctrl->alias_count > 0);
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const float4 Qi = P.rec0[k];
  const float hif = Qi.z;
  if (signbit(hif)) return;
  const int2 qref = P.meta[k];
  const int qkey = P.keys_sorted[k];
  const bool slow = qref.x >= g.ncx || !(hif > 0.f);
  const int W = g.mode == 0 ? 1 : (slow ? g.wide : g.wt);
  double xi = 0, yi = 0, hi = 0;
  float4 Ri = make_float4(0, 0, 0, 0);
  if (MIXED) {
    Ri = P.rec1[k];
  } else {
    const double4_32a A = P.r64a[k], B = P.r64b[k];
    xi = A.x; yi = A.y; hi = B.w;
  }
  const float KC = (float)(Support<KERNEL>::q * Support<KERNEL>::q);
  const float SK = (float)Support<KERNEL>::q * 1.000002f;
  double rho = 0.0;
  float rhof = 0.f;
  const Stencil sten(g, qref, qkey, W);
  for_stencil(sten, P.cstart, [&](unsigned int j) {
      if (filter && !in_ref_stencil(P.meta, j, g, qref)) return;
      const float4 qj = P.rec0[j];
      if (signbit(qj.z)) return;  // SummationDensity.py: fluid neighbours only
      const float hij = 0.5f * (hif + fabsf(qj.z));
      if (MIXED) {
        const float4 rj = P.rec1[j];
        const float dx = (Qi.x - qj.x) + (Ri.x - rj.x);
        const float dy = (Qi.y - qj.y) + (Ri.y - rj.y);
        const float d2 = dx * dx + dy * dy;
        if (d2 > KC * hij * hij) return;
        const float q = sqrtf(d2) / hij;
        float w;
        if (KERNEL == SPH_KERNEL_CUBIC) {
          const float al = (float)kCubicFac / (hij * hij);
          const float t = fmaxf(2.0f - q, 0.f);
          w = q > 1.0f ? al * 0.25f * t * t * t : al * (1.0f - 1.5f * q * q * (1.0f - 0.5f * q));
        } else if (KERNEL == SPH_KERNEL_WENDLAND) {
          const float inner = fmaxf(1.0f - 0.5f * q, 0.f), i2 = inner * inner;
          w = (float)kWendFac / (hij * hij) * (i2 * i2 * i2) * ((35.0f / 12.0f) * q * q + 3.0f * q + 1.0f);
        } else {
          w = (float)kInvPi / (hij * hij) * __expf(-q * q);
        }
        rhof += qj.w * w;
      } else {
        const float dx = Qi.x - qj.x, dy = Qi.y - qj.y;
        const float rp = SK * hij + g.pad_e;
        if (dx * dx + dy * dy > rp * rp) return;
        const double4_32a A = P.r64a[j], B = P.r64b[j];
        const double ddx = xi - A.x, ddy = yi - A.y;
        const double r = __dsqrt_rn(__dadd_rn(__dmul_rn(ddx, ddx), __dmul_rn(ddy, ddy)));
        const double h = __dmul_rn(0.5, __dadd_rn(hi, fabs(B.w)));
        if (__ddiv_rn(r, h) <= 3.0)
          rho += B.x * (KERNEL == SPH_KERNEL_CUBIC ? cubic_w(r, h)
                                                   : (KERNEL == SPH_KERNEL_WENDLAND ? wendland_w(r, h) : gauss_w(r, h)));
      }
   });
  a.rho[P.perm[k]] = MIXED ? f2d(rhof) : rho;
}

// ---------------------------------------------------------------------------
// Neighbour-set export (NNLinkedList.near for every particle, FP64 exact):
// count pass (idx == nullptr) or fill pass.  Reads the caller's arrays.
// Each list comes out in the reference's order (NNLinkedList.py:50-78): the
// 3x3 stencil cells with the x shift outer and the y shift inner, and inside
// a cell its linked list, head-insert order, i.e. descending index.
// ---------------------------------------------------------------------------
// Sort key of member j in the list of a query whose raw reference cell is
// qref: the stencil position of j's storage cell (an x-overflow particle is
// stored in the aliased cell), then descending index.  Smaller comes first.
__device__ __forceinline__ unsigned long long ref_order_key(const int2 *__restrict__ refcell, long long ncx,
                                                            int2 qref, long long j) {
  const int2 rc = refcell[j];
  int sx, sy;
  storage_cell(rc.x, rc.y, ncx, sx, sy);
  const unsigned p = (unsigned)((sx - qref.x + 1) * 3 + (sy - qref.y + 1));  // 0..8 for members
  return ((unsigned long long)p << 32) | (unsigned long long)(0xffffffffu - (unsigned)j);
}

// insertion sort of idx[0..cnt) (and the parallel arrays, when given) into
// the reference's order
__device__ void sort_ref_order(int64_t *idx, double *a0, double *a1, double *a2, long long cnt,
                               const int2 *__restrict__ refcell, long long ncx, int2 qref) {
  for (long long s = 1; s < cnt; s++) {
    const int64_t v = idx[s];
    const unsigned long long kv = ref_order_key(refcell, ncx, qref, v);
    double b0 = 0, b1 = 0, b2 = 0;
    if (a0) {
      b0 = a0[s];
      b1 = a1[s];
      b2 = a2[s];
    }
    long long t = s - 1;
    while (t >= 0 && ref_order_key(refcell, ncx, qref, idx[t]) > kv) {
      idx[t + 1] = idx[t];
      if (a0) {
        a0[t + 1] = a0[t];
        a1[t + 1] = a1[t];
        a2[t + 1] = a2[t];
      }
      t--;
    }
    idx[t + 1] = v;
    if (a0) {
      a0[t + 1] = b0;
      a1[t + 1] = b1;
      a2[t + 1] = b2;
    }
  }
}

__global__ void __launch_bounds__(kPairBlock)
    k_nn_export(const double *__restrict__ x, const double *__restrict__ y, const double *__restrict__ h,
                long long n, const int *__restrict__ perm, const int *__restrict__ keys_sorted,
                const int2 *__restrict__ meta, const int2 *__restrict__ refcell,
                const unsigned int *__restrict__ cstart, const DevGrid *__restrict__ gp, int64_t *counts,
                const int64_t *offsets, int64_t *idx) {
  const DevGrid g = *gp;
  long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int i = perm[k];
  const double xi = x[i], yi = y[i], hi = h[i];
  const int2 qref = meta[k];
  const int qkey = keys_sorted[k];
  const int W = g.mode == 1 ? g.wide : 1;
  const bool filter = g.mode == 1;
  long long cnt = 0;
  const long long base = idx ? offsets[i] : 0;
  const Stencil sten(g, qref, qkey, W);
  for_stencil(sten, cstart, [&](unsigned int j) {
      if (filter && !in_ref_stencil(meta, j, g, qref)) return;
      const int pj = perm[j];
      const double dx = xi - x[pj], dy = yi - y[pj];
      const double d2 = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
      const double r = __dsqrt_rn(d2);
      const double hij = __dmul_rn(0.5, __dadd_rn(hi, h[pj]));
      const double q = __ddiv_rn(r, hij);
      if (q <= 3.0) {
        if (idx) idx[base + cnt] = pj;
        cnt++;
      }
   });
  if (!idx) {
    counts[i] = cnt;
    return;
  }
  sort_ref_order(idx + base, nullptr, nullptr, nullptr, cnt, refcell, g.ncx, qref);
}

// ---------------------------------------------------------------------------
// Tile kernel (mixed form).  A block takes one tile of 2^ts x 2^ts cells at a
// time and stages the records of the tile and its W-cell halo in shared
// memory: a table of the (2^ts + 2W)^2 halo cells (counts -> exclusive scan ->
// shared-memory offsets, cells row-major, so each stencil row of a query is
// one contiguous shared-memory range), then the records row by row.  Its
// queries walk their stencils in shared memory, with 16-bit list entries.
// The candidate order (rows, then cells by x, then slot) is the global
// path's, so both give the same sums.
// Left to the global path, through the fallback list: tiles whose halo does
// not fit, queries whose own cell is not in their stencil or whose h is not
// positive, and every query when candidates need the reference-stencil filter
// or the halo table does not fit (wide stencils).
// Blocks are persistent and claim one tile at a time from the list of
// non-empty tiles the neighbour build writes, the next claim overlapping the
// current tile.
// ---------------------------------------------------------------------------
constexpr int kTileThreads = 256;   // threads of a tile block (8 warps)
static_assert(kTileThreads >= 16 * 16, "a sparse unit's slots fit one per thread");
constexpr int kHaloCellsMax = 400;  // (16 + 2 * 2)^2: 16x16 tiles with a 5x5 stencil
constexpr int kHaloScanPer = (kHaloCellsMax + 31) / 32;
#ifndef SPH_TILE_UNROLL_PAIRS
#define SPH_TILE_UNROLL_PAIRS 1
#endif
#ifndef SPH_TILE_UNROLL_CANDS
#define SPH_TILE_UNROLL_CANDS 2
#endif
// resident tile blocks per SM (registers and shared memory allow three for
// the 32-entry lists of the 2h kernels, two for the Gaussian's 64)
template <int KERNEL>
struct TileBlocks {
  static constexpr int value = ListCap<KERNEL>::value == 32 ? 3 : 2;
};
constexpr bool kSplitTail = true;  // the last tiles of a launch as half-tile units
constexpr int kTileUnrollPairs = SPH_TILE_UNROLL_PAIRS;  // ILP over list entries
constexpr int kTileUnrollCands = SPH_TILE_UNROLL_CANDS;  // ILP over stencil candidates
constexpr int kHaloCap = SPH_HALO_CAP;  // particles of one halo in shared memory
static_assert(kHaloCap <= 65535, "list entries are 16-bit");
static_assert(kHaloCellsMax <= 65535, "query map entries are 16-bit halo cells");

__device__ __forceinline__ void fb_push(DevCtrl *ctrl, int2 *fb, unsigned int fb_cap, unsigned int s,
                                        unsigned int len) {
  const unsigned int e = atomicAdd(&ctrl->fb_count, 1u);
  if (e < fb_cap) fb[e] = make_int2((int)s, (int)len);
}

// Geometry and constants of the grid a tile belongs to.
struct TileGeom {
  int ts, ntlx, ntx, nty, W, T, HW, HC;
  int cell0;  // global id of the grid's first cell (batched form; 0 otherwise)
  long long ncx;
  float r0f, pad, hmaxf;
  float rb2;  // squared, padded Lennard-Jones reach
};

__device__ __forceinline__ TileGeom tile_geom(const DevGrid &g, double r0, int cell0) {
  TileGeom tg;
  tg.ts = g.ts;
  tg.ntlx = g.ntlx;
  tg.ntx = g.ntx;
  tg.nty = g.nty;
  tg.W = g.mode == 0 ? 1 : g.wt;
  tg.T = 1 << g.ts;
  tg.HW = tg.T + 2 * tg.W;
  tg.HC = tg.HW * tg.HW;
  tg.cell0 = cell0;
  tg.ncx = g.ncx;
  tg.r0f = (float)r0;
  tg.pad = g.pad_e;
  tg.hmaxf = g.hmaxf;
  const float rb = fminf(tg.r0f, 3.0f * tg.hmaxf) * 1.000002f + tg.pad;
  tg.rb2 = rb * rb;
  return tg;
}

// shared memory of the tile kernels (dynamic: above the 48 KB static limit)
template <int KERNEL>
struct TileShared {
  float4 h0[kHaloCap], h1[kHaloCap], h2[kHaloCap];  // rec0, rec1, rec2 of the halo
  unsigned short lists[ListCap<KERNEL>::value][kTileThreads];
  unsigned int hoff[kHaloCellsMax + 1];  // shared-memory offset of each halo cell, then the total
  unsigned int hgs[kHaloCellsMax];       // its first sorted slot
  unsigned short qmap[kHaloCap];         // halo cell of each query of the tile
  long long s_tile[2];                   // this and the next claimed work unit (-1: none left)
  int s_inst[2];                         // their instances (batched form)
  unsigned long long red[kTileThreads / 32];
};

// One tile: stage its halo, run its queries.  Returns this thread's largest
// encoded a^2 over its queries.  All threads of the block call it together.
//   1. halo table: every halo cell's first sorted slot and count;
//   2. warp 0: exclusive scan of the counts (shared-memory offsets); then
//      every warp copies halo rows into shared memory (a row is at most three
//      runs of consecutive slots) and the threads map each query of the tile
//      to its halo cell;
//   3. each query walks its stencil rows.
// TSC / WC: the tile shift and stencil half-width as compile-time constants
// (the own grid's 16x16 tiles with a 5x5 stencil), so that the halo
// coordinate arithmetic has no integer division; 0 takes them from tg.
// UH: every fluid particle has the same h (UniformQ).
// part: 0 the whole tile; 1 and 2 its first and second half of cell rows;
// 3 to 6 its four quarters (the kernel's last tiles are split so that its
// final round of work is short).  wall: it holds boundary particles.
template <int KERNEL, bool XSPH, bool SUMDENS, bool UH, int TSC, int WC>
__device__ __forceinline__ unsigned long long tile_process(const StepArgs &a, const PairPtrs &P, const TileGeom &tg,
                                                           const PairParams &pp, int t, int part, bool wall,
                                                           TileShared<KERNEL> &sm, DevCtrl *ctrl, int2 *fb,
                                                           unsigned int fb_cap) {
  constexpr int kListCap = ListCap<KERNEL>::value;
  const int tid = threadIdx.x;
  const int ts = TSC ? TSC : tg.ts;
  const int W = TSC ? WC : tg.W;
  const int T = 1 << ts, HW = T + 2 * W;
  const int rows = part == 0 ? T : (part <= 2 ? T >> 1 : T >> 2);
  const int row0 = part == 2 ? T >> 1 : (part >= 3 ? (part - 3) * (T >> 2) : 0);
  const int HWy = rows + 2 * W, HC = HW * HWy;
  const int ntlx = tg.ntlx;
  float4 *h0 = sm.h0, *h1 = sm.h1, *h2 = sm.h2;
  unsigned int *hoff = sm.hoff, *hgs = sm.hgs;
  const unsigned int *cst = P.cstart + tg.cell0;  // this grid's cells
  unsigned long long ea = kEncMaxId;
  const unsigned int tb = (unsigned int)t << (2 * ts);  // the tile's first cell (row-major inside)
  const unsigned int qs = __ldg(&cst[tb + row0 * T]), qe = __ldg(&cst[tb + (row0 + rows) * T]);
  const int ox = (t % ntlx) * T - W, oy = (t / ntlx) * T + row0 - W;
  // 1. halo table: counts and first slots
  for (int c = tid; c < HC; c += kTileThreads) {
    const int x = ox + c % HW, y = oy + c / HW;
    unsigned int gs = 0, cnt = 0;
    if (x >= 0 && x < tg.ntx && y >= 0 && y < tg.nty) {
      const int key = tiled_key(x, y, ts, ntlx);
      gs = __ldg(&cst[key]);
      cnt = __ldg(&cst[key + 1]) - gs;
    }
    hgs[c] = gs;
    hoff[c] = cnt;
  }
  __syncthreads();
  if (tid < 32) {  // 2. exclusive scan of the counts, kHaloScanPer cells per lane
    const int c0 = tid * kHaloScanPer;
    unsigned int v[kHaloScanPer], sum = 0;
#pragma unroll
    for (int u = 0; u < kHaloScanPer; u++) {
      v[u] = c0 + u < HC ? hoff[c0 + u] : 0u;
      sum += v[u];
    }
    unsigned int inc = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned int o = __shfl_up_sync(0xffffffffu, inc, d);
      if (tid >= d) inc += o;
    }
    unsigned int run = inc - sum;
#pragma unroll
    for (int u = 0; u < kHaloScanPer; u++) {
      if (c0 + u < HC) hoff[c0 + u] = run;
      run += v[u];
    }
    if (tid == 31) hoff[HC] = inc;
  }
  __syncthreads();
  const unsigned int total = hoff[HC];
  if (total == 0) {  // nothing to stage (a listed tile holds particles)
    __syncthreads();
    return ea;
  }
  if (total > (unsigned)kHaloCap) {  // halo does not fit: global path
    if (tid == 0)
      for (unsigned int s = qs; s < qe; s += kPairBlock) fb_push(ctrl, fb, fb_cap, s, min((unsigned)kPairBlock, qe - s));
    __syncthreads();
    return ea;
  }
  // 2b. the halo's records, row by row: warp w copies halo rows w, w + 8,
  // ...; a row's cells are one shared-memory range, and in global memory at
  // most three runs (the cells of one row inside one tile are consecutive
  // ids).  Each lane issues 16-byte asynchronous copies of particles of the
  // row, so that all copies of the halo are in flight together and the block
  // waits once.  (One bulk copy per run and record array would be ~180 small
  // copies per tile, whose per-copy cost dominates.)
  {
    const int warp = tid >> 5, lane = tid & 31;
    const int xa = ox > 0 ? ox : 0;
    const int xe = ox + HW < tg.ntx ? ox + HW : tg.ntx;
    for (int y = warp; y < HWy; y += kTileThreads / 32) {
      const int gy = oy + y;
      if (gy < 0 || gy >= tg.nty || xa >= xe) continue;
      const int cb = y * HW - ox;  // halo cell of grid column x: cb + x
      if (T >= W) {
        // runs [xa, x1), [x1, x2), [x2, xe) (empty when their bounds meet)
        const int x1 = min(((xa >> ts) + 1) << ts, xe);
        const int x2 = min(((x1 >> ts) + 1) << ts, xe);
        const unsigned int sA = hoff[cb + xa], sB = hoff[cb + x1], sC = hoff[cb + x2], sE = hoff[cb + xe];
        const unsigned int gA = hgs[cb + xa], gB = x1 < xe ? hgs[cb + x1] : 0u, gC = x2 < xe ? hgs[cb + x2] : 0u;
        for (unsigned int k = sA + lane; k < sE; k += 32) {
          const unsigned int src = k < sB ? gA + (k - sA) : (k < sC ? gB + (k - sB) : gC + (k - sC));
          cp_async16(h0 + k, P.rec0 + src);
          cp_async16(h1 + k, P.rec1 + src);
          cp_async16(h2 + k, P.rec2 + src);
        }
      } else {
        // tiles narrower than the stencil: the row's runs one by one
        for (int x = xa; x < xe;) {
          const int re = min(((x >> ts) + 1) << ts, xe);
          const unsigned int s0 = hoff[cb + x], e0 = hoff[cb + re], g0 = hgs[cb + x];
          for (unsigned int k = s0 + lane; k < e0; k += 32) {
            cp_async16(h0 + k, P.rec0 + g0 + (k - s0));
            cp_async16(h1 + k, P.rec1 + g0 + (k - s0));
            cp_async16(h2 + k, P.rec2 + g0 + (k - s0));
          }
          x = re;
        }
      }
    }
  }
  // query -> halo cell, for the tile's own cells (their sorted slots are the
  // tile's query range, in cell order)
  for (int c = tid; c < T * rows; c += kTileThreads) {
    const int hc = (W + (c >> ts)) * HW + W + (c & (T - 1));
    const unsigned int cnt = hoff[hc + 1] - hoff[hc], base = hgs[hc] - qs;
    for (unsigned int u = 0; u < cnt; u++) sm.qmap[base + u] = (unsigned short)hc;
  }
  cp_async_wait_all();
  __syncthreads();
  // 3. queries.  Candidate radius: the padded reach of the largest pair h
  // (every |h| <= hmaxf), so that one compare per candidate suffices; next to
  // a wall, without XSPH, boundary candidates have the Lennard-Jones reach for
  // theirs (they are several times denser than the fluid, and inside the kernel
  // support most of them do nothing)
  const MixedConsts &mc = pp.mc;
  const UniformQ uq = pp.u;  // in registers: read per pair
  auto reach2 = [&](float h) {
    const float hq = 0.5f * (h + tg.hmaxf);
    const float rq = fmaxf((float)Support<KERNEL>::q * 1.000002f * hq, fminf(tg.r0f, 3.0f * hq) * 1.000002f) + tg.pad;
    return rq * rq;
  };
  const float rq2_uh = UH ? reach2(uq.h) : 0.f;
  const unsigned int nq = qe - qs;
  for (unsigned int q = tid; q < nq; q += kTileThreads) {
    const int hc = sm.qmap[q];
    const int hx = hc % HW, hy = hc / HW;
    const unsigned int k = qs + q;
    const unsigned int sq = hoff[hc] + (k - hgs[hc]);  // the query's own shared-memory slot
    const float4 Qi = h0[sq];
    const float hif = Qi.z;
    if (signbit(hif)) continue;  // queries are fluid
    // an x-overflow alias (reference cells only) or h <= 0: global path
    if ((W == 1 && P.meta[k].x >= tg.ncx) || !(hif > 0.f)) {
      fb_push(ctrl, fb, fb_cap, k, 1u);
      continue;
    }
    const float4 Ri = h1[sq], Vi = h2[sq];
    const int i = P.perm[k];
    MixedAcc acc;
    auto physics = [&](int cnt) {
#pragma unroll kTileUnrollPairs
      for (int u = 0; u < cnt; u++) {
        const unsigned int j = sm.lists[u][tid];
        mixed_entry<KERNEL, XSPH, SUMDENS, UH>(acc, mc, uq, Qi, Ri, Vi, h0[j], h1[j], h2 + j);
      }
    };
    const float rq2 = UH ? rq2_uh : reach2(hif);
    int nl = 0;
    auto walk = [&](auto near_wall) {
      constexpr bool kWall = decltype(near_wall)::value;
      // the stencil rows' slot ranges, the query's own row as the two ranges
      // either side of its own slot (the particle itself is no candidate)
      for (int r = -W, seg = 0; r <= W; seg = 0, r++) {
        const unsigned int *row = hoff + (hy + r) * HW + hx;
        unsigned int j = row[-W];
        const unsigned int e = row[W + 1];
        unsigned int se = r == 0 ? sq : e;
        for (;;) {
          while (j < se) {
            if (nl == kListCap) {
              physics(nl);
              nl = 0;
            }
            // a chunk that cannot overflow the list: every candidate is
            // written, and kept (counted) when inside the radius
            const unsigned int ce = min(se, j + (unsigned int)(kListCap - nl));
#pragma unroll kTileUnrollCands
            for (; j < ce; j++) {
              float2 p;
              float lim = rq2;
              if (kWall) {
                const float4 p4 = h0[j];
                p = lo2(p4);
                lim = signbit(p4.z) ? tg.rb2 : rq2;
              } else {
                p = *reinterpret_cast<const float2 *>(h0 + j);
              }
              const float2 d = sub2(lo2(Qi), p);
              sm.lists[nl][tid] = (unsigned short)j;
              nl += fmaf(d.x, d.x, d.y * d.y) <= lim ? 1 : 0;
            }
          }
          if (r != 0 || seg) break;
          seg = 1;
          j = sq + 1;
          se = e;
        }
      }
    };
    if (wall && !XSPH) walk(std::true_type());
    else walk(std::false_type());
    physics(nl);
    const unsigned long long qa = mixed_store<XSPH, SUMDENS>(acc, a, i, pp.write_xsph);
    ea = qa > ea ? qa : ea;
  }
  __syncthreads();
  return ea;
}

// block-wide max of v in thread 0 (all threads call it)
template <int NT>
__device__ __forceinline__ unsigned long long block_max_u64(unsigned long long v, unsigned long long *red) {
  const unsigned long long wm = warp_max_u64(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = wm;
  __syncthreads();
  unsigned long long b = kEncMaxId;
  if (threadIdx.x == 0)
    for (int w = 0; w < NT / 32; w++) b = red[w] > b ? red[w] : b;
  __syncthreads();
  return b;
}

// the tile of a single-scene grid with the shape the grid has
template <int KERNEL, bool XSPH, bool SUMDENS, bool UH>
__device__ __forceinline__ unsigned long long tile_any(const StepArgs &a, const PairPtrs &P, const TileGeom &tg,
                                                       const PairParams &pp, int t, int part, bool wall,
                                                       TileShared<KERNEL> &sm, DevCtrl *ctrl, int2 *fb,
                                                       unsigned int fb_cap) {
  if (tg.ts == 4 && tg.W == 2)
    return tile_process<KERNEL, XSPH, SUMDENS, UH, 4, 2>(a, P, tg, pp, t, part, wall, sm, ctrl, fb, fb_cap);
  if (tg.ts == 3 && tg.W == 2)
    return tile_process<KERNEL, XSPH, SUMDENS, UH, 3, 2>(a, P, tg, pp, t, part, wall, sm, ctrl, fb, fb_cap);
  return tile_process<KERNEL, XSPH, SUMDENS, UH, 0, 0>(a, P, tg, pp, t, part, wall, sm, ctrl, fb, fb_cap);
}

template <int KERNEL, bool XSPH, bool SUMDENS, bool UH>
__global__ void __launch_bounds__(kTileThreads, TileBlocks<KERNEL>::value)
    k_pair_tiles(StepArgs a, PairPtrs P, PairParams pp, const int *__restrict__ tiles,
                 const int *__restrict__ tiles_h, unsigned int tiles_cap,
                 int2 *__restrict__ fb, unsigned int fb_cap) {
  step_kernel_entry();
  extern __shared__ __align__(128) unsigned char smem_raw[];
  TileShared<KERNEL> &sm = *reinterpret_cast<TileShared<KERNEL> *>(smem_raw);
  const int tid = threadIdx.x;
  DevCtrl *ctrl = P.ctrl;
  const DevGrid *gp = P.grid;
  const TileGeom tg = tile_geom(*gp, pp.r0, 0);
  const bool filter = gp->mode == 1 && (gp->need_filter || ctrl->alias_count > 0);
  unsigned long long ea = kEncMaxId;

  if (filter || tg.HC > kHaloCellsMax) {
    // everything on the global path, in 128-slot chunks
    if (tid == 0) {
      const long long nch = (pp.n + kPairBlock - 1) / kPairBlock;
      for (long long c = blockIdx.x; c < nch; c += gridDim.x)
        fb_push(ctrl, fb, fb_cap, (unsigned)(c * kPairBlock), (unsigned)min((long long)kPairBlock, pp.n - c * kPairBlock));
    }
  } else {
    // Work units in claim order: dense tiles with a wall along a side (their
    // own list), the other dense tiles (listed from the front of the tile
    // list), then the sparse ones (listed from its back).  Of that order, the
    // last `sq` tiles come as four quarter-tile units each and the `sh`
    // before them as two half-tile units each, so that the kernel's final
    // rounds of work are short.  A unit is encoded as 8 entry + part (part 0:
    // whole tile; 1, 2: halves; 3 to 6: quarters), -1 when none is left; an
    // entry is 2 tile + 1 when the tile holds boundary particles.
    const unsigned int nh = ctrl->tl_heavy, ntl = nh + ctrl->tl_count, nall = ntl + ctrl->tl_back;
    const unsigned int sq = (kSplitTail && tg.ts >= 2) ? min(nall, gridDim.x / 4u) : 0u;
    const unsigned int sh = (kSplitTail && tg.ts >= 1) ? min(nall - sq, gridDim.x) : 0u;
    const unsigned int nw = nall - sq - sh;  // whole-tile units
    auto tile_at = [&](unsigned int p) {
      return p < nh ? tiles_h[p] : (p < ntl ? tiles[p - nh] : tiles[tiles_cap - 1 - (p - ntl)]);
    };
    auto claim = [&](unsigned int c) -> long long {
      if (c < nw) return 8ll * tile_at(c);
      c -= nw;
      if (c < 2 * sh) return 8ll * tile_at(nw + (c >> 1)) + 1 + (int)(c & 1u);
      c -= 2 * sh;
      return c < 4 * sq ? 8ll * tile_at(nw + sh + (c >> 2)) + 3 + (int)(c & 3u) : -1;
    };
    if (tid == 0) {
      if (blockIdx.x == 0) {  // the dump cell (reference-OOB particles) is in no tile
        const unsigned int d0 = __ldg(&P.cstart[gp->ncells]), d1 = __ldg(&P.cstart[gp->ncells + 1]);
        for (unsigned int s = d0; s < d1; s += kPairBlock) fb_push(ctrl, fb, fb_cap, s, min((unsigned)kPairBlock, d1 - s));
      }
      sm.s_tile[0] = claim(atomicAdd(&ctrl->tile_next, 1u));
    }
    __syncthreads();
    for (int it = 0;; it++) {
      const long long u = sm.s_tile[it & 1];
      if (u < 0) break;
      if (tid == 0)  // claim the next unit while this one runs
        sm.s_tile[(it + 1) & 1] = claim(atomicAdd(&ctrl->tile_next, 1u));
      const unsigned long long q =
          tile_any<KERNEL, XSPH, SUMDENS, UH>(a, P, tg, pp, (int)(u >> 4), (int)u & 7, (u & 8) != 0, sm, ctrl, fb, fb_cap);
      ea = q > ea ? q : ea;
    }
  }
  // this block's max a^2 (the list kernel finishes the TimeStep reduction);
  // the last block resets the tile counter
  if (pp.do_dt) {
    const unsigned long long ba = block_max_u64<kTileThreads>(ea, sm.red);
    if (tid == 0 && ba != kEncMaxId) atomicMax(&ctrl->pd_a2max, ba);
  }
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(&ctrl->tile_done, 1u) == gridDim.x - 1) {
      ctrl->tile_next = 0;
      ctrl->tile_done = 0;
    }
  }
}

// ---------------------------------------------------------------------------
// Batched form: the tile kernel over the (instance, tile) list of all
// instances, each tile with its instance's grid and constants, and the
// fallback list with each entry's instance (see nn_build.cu).  Every instance
// has a fixed h, so the uniform-h form applies to the instances whose
// viscosity beta is 0; the others take the general per-pair form.
// ---------------------------------------------------------------------------
template <int KERNEL, bool XSPH, bool SUMDENS>
__global__ void __launch_bounds__(kTileThreads, TileBlocks<KERNEL>::value)
    k_bt_pair_tiles(StepArgs a, PairPtrs P, BatchPtrs B, int2 *__restrict__ fb, unsigned int fb_cap) {
  step_kernel_entry();
  extern __shared__ __align__(128) unsigned char smem_raw[];
  TileShared<KERNEL> &sm = *reinterpret_cast<TileShared<KERNEL> *>(smem_raw);
  const int tid = threadIdx.x;
  DevCtrl *ctrl = P.ctrl;
  // Work units as in k_pair_tiles: dense tiles from the front of the list,
  // sparse ones from its back, the last of them in quarters and halves (a tile
  // too small to split comes whole with its first part).
  const unsigned int ntl = ctrl->tl_count, nall = ntl + ctrl->tl_back;
  const unsigned int sq = min(nall, gridDim.x / 4u), sh = min(nall - sq, gridDim.x);
  const unsigned int nw = nall - sq - sh;  // whole-tile units
  auto claim = [&](int slot) {
    unsigned int c = atomicAdd(&ctrl->tile_next, 1u), p = nall, part = 0, first = 1, split = 0;
    if (c < nw) {
      p = c;
    } else if (c - nw < 2 * sh) {
      c -= nw;
      p = nw + (c >> 1);
      part = 1 + (c & 1u);
      first = !(c & 1u);
      split = 1;
    } else if (c - nw - 2 * sh < 4 * sq) {
      c -= nw + 2 * sh;
      p = nw + sh + (c >> 2);
      part = 3 + (c & 3u);
      first = !(c & 3u);
      split = 2;
    }
    int2 e = make_int2(-1, -1);
    if (p < nall) {
      e = p < ntl ? B.tiles[p] : B.tiles[B.tiles_cap - 1 - (p - ntl)];
      if (B.grids[e.x].ts < (int)split) part = first ? 0 : 7;  // 7: nothing to do
    }
    sm.s_inst[slot] = e.x;
    sm.s_tile[slot] = p < nall ? 8ll * e.y + part : -1ll;
  };
  if (tid == 0) {
    // every instance's dump cell (reference-OOB particles) is in no tile.  (One
    // block walking all instances took longer than the tiles.)
    for (int b = blockIdx.x; b < B.n_inst; b += gridDim.x) {
      const int c = B.coff[b] + B.grids[b].ncells;
      const unsigned int d0 = __ldg(&P.cstart[c]), d1 = __ldg(&P.cstart[c + 1]);
      for (unsigned int s = d0; s < d1; s += kPairBlock) fb_push(ctrl, fb, fb_cap, s, min((unsigned)kPairBlock, d1 - s));
    }
    claim(0);
  }
  __syncthreads();
  for (int it = 0;; it++) {
    const long long u = sm.s_tile[it & 1];
    const int b = sm.s_inst[it & 1];
    if (u < 0) break;
    if (tid == 0) claim((it + 1) & 1);  // the next unit while this one runs
    const int t = (int)(u >> 3), part = (int)u & 7;
    if (part == 7) {
      __syncthreads();
      continue;
    }
    const DevGrid &g = B.grids[b];
    const PairParams &pp = B.ip[b].pp;
    const TileGeom tg = tile_geom(g, pp.r0, B.coff[b]);
    const bool filter = g.mode == 1 && (g.need_filter || B.sl[b].alias_count > 0);
    if (filter || tg.HC > kHaloCellsMax) {  // this instance's tiles go to the global path
      if (tid == 0) {
        const unsigned int *cst = P.cstart + tg.cell0;
        // the unit's rows of the tile (all of them, a half, a quarter)
        const int T = 1 << tg.ts, rows = part == 0 ? T : (part <= 2 ? T >> 1 : T >> 2);
        const int c0 = (t << (2 * tg.ts)) + (part == 0 ? 0 : (part <= 2 ? part - 1 : part - 3) * rows * T);
        const unsigned int qs = __ldg(&cst[c0]), qe = __ldg(&cst[c0 + rows * T]);
        for (unsigned int s = qs; s < qe; s += kPairBlock) fb_push(ctrl, fb, fb_cap, s, min((unsigned)kPairBlock, qe - s));
      }
      __syncthreads();
      continue;
    }
    const unsigned long long ea =
        pp.beta == 0.0 ? tile_any<KERNEL, XSPH, SUMDENS, true>(a, P, tg, pp, t, part, true, sm, ctrl, fb, fb_cap)
                       : tile_any<KERNEL, XSPH, SUMDENS, false>(a, P, tg, pp, t, part, true, sm, ctrl, fb, fb_cap);
    const unsigned long long ba = block_max_u64<kTileThreads>(ea, sm.red);
    if (tid == 0 && ba != kEncMaxId) atomicMax(&B.sl[b].pd_a2max, ba);
  }
  if (tid == 0) {
    __threadfence();
    if (atomicAdd(&ctrl->tile_done, 1u) == gridDim.x - 1) {
      ctrl->tile_next = 0;
      ctrl->tile_done = 0;
    }
  }
}

template <int KERNEL, bool XSPH, bool SUMDENS>
__global__ void __launch_bounds__(kPairBlock, kListBlocks)
    k_bt_pair_list(StepArgs a, PairPtrs P, BatchPtrs B, const int2 *__restrict__ fb) {
  step_kernel_entry();
  __shared__ unsigned int lists[ListCap<KERNEL>::value][kPairBlock];
  __shared__ unsigned long long red[kPairBlock / 32];
  const unsigned int cnt = *(volatile unsigned int *)&P.ctrl->fb_count;
  for (unsigned int e = blockIdx.x; e < cnt; e += gridDim.x) {
    const int2 r = fb[e];
    const int b = B.inst[P.perm[r.x]];  // an entry lies in one instance
    const DevGrid &g = B.grids[b];
    const PairParams &pp = B.ip[b].pp;
    const bool filter = g.mode == 1 && (g.need_filter || B.sl[b].alias_count > 0);
    unsigned long long ea = kEncMaxId;
    if ((int)threadIdx.x < r.y)
      ea = pp.beta == 0.0
               ? pair_query<KERNEL, XSPH, SUMDENS, true>(a, P, pp, g, filter, r.x + threadIdx.x, lists, B.coff[b])
               : pair_query<KERNEL, XSPH, SUMDENS, false>(a, P, pp, g, filter, r.x + threadIdx.x, lists, B.coff[b]);
    const unsigned long long ba = block_max_u64<kPairBlock>(ea, red);
    if (threadIdx.x == 0 && ba != kEncMaxId) atomicMax(&B.sl[b].pd_a2max, ba);
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&P.ctrl->fb_done, 1u) == gridDim.x - 1) {
      P.ctrl->fb_count = 0;
      P.ctrl->fb_done = 0;
    }
  }
}

// ---------------------------------------------------------------------------
// Probes: NNLinkedList.nearPos (src/Tools/NNLinkedList.py:41-84) at arbitrary
// points, on the table of the last build, and the pressure interpolation the
// reference's ice-coupling example composes from it (Shepard-normalised
// summation density + Tait EOS, examples/IceBreak.py:253-285,
// src/Equations/Shepard.py, src/Equations/SummationDensity.py).
// ---------------------------------------------------------------------------
// Raw reference cell (qref) of point (x, y), its own-grid cell key (clamped
// binning; mode 1) and the stencil half-width W that covers q <= 3 for a
// point with smoothing length h: r <= 1.5 (h + hmax).
__device__ __forceinline__ int probe_cell(const DevGrid &g, double x, double y, double h, int2 &qref, int &W) {
  const long long cx = ref_cell(x, g.xmin, g.cs, g.inv_cs, g.xminf, g.inv_csf);
  const long long cy = ref_cell(y, g.ymin, g.cs, g.inv_cs, g.yminf, g.inv_csf);
  qref = make_int2(sat_i32(cx), sat_i32(cy));
  if (g.mode == 0) {
    W = 1;
    return 0;
  }
  const float tx = fminf(fmaxf((d2f_trunc(x) - g.oxf) * g.inv_ctf, 0.f), g.txmaxf);
  const float ty = fminf(fmaxf((d2f_trunc(y) - g.oyf) * g.inv_ctf, 0.f), g.tymaxf);
  const int kx = min(max((int)floorf(tx), 0), g.ntx - 1), ky = min(max((int)floorf(ty), 0), g.nty - 1);
  // in FP32, rounded up (a wider stencil has the same members)
  const float reach = 1.5f * (d2f_trunc(h) + g.hmaxf) * 1.00001f;
  const float wd = ceilf(reach * g.inv_ctf * 1.00001f) + 1.0f;
  W = !(wd >= 1.0f) ? 1 : (wd > 1024.0f ? 1024 : (int)wd);
  return tiled_key(kx, ky, g.ts, g.ntlx);
}

__global__ void __launch_bounds__(kPairBlock)
    k_nn_probe(const double *__restrict__ px, const double *__restrict__ py, const double *__restrict__ ph,
               long long np, const double *__restrict__ x, const double *__restrict__ y,
               const double *__restrict__ h, const int *__restrict__ perm, const int2 *__restrict__ meta,
               const int2 *__restrict__ refcell, const unsigned int *__restrict__ cstart,
               const DevGrid *__restrict__ gp, int64_t *counts, const int64_t *offsets, int64_t *idx,
               double *hij_out, double *q_out, double *r_out) {
  const DevGrid g = *gp;
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= np) return;
  const double xi = px[k], yi = py[k], hi = ph[k];
  int2 qref;
  int W;
  const int qkey = probe_cell(g, xi, yi, hi, qref, W);
  const bool filter = g.mode == 1;
  long long cnt = 0;
  const long long base = idx ? offsets[k] : 0;
  const Stencil sten(g, qref, qkey, W);
  for_stencil(sten, cstart, [&](unsigned int j) {
    if (filter && !in_ref_stencil(meta, j, g, qref)) return;
    const int pj = perm[j];
    const double dx = xi - x[pj], dy = yi - y[pj];
    const double r = __dsqrt_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)));
    const double hij = __dmul_rn(0.5, __dadd_rn(hi, h[pj]));
    const double q = __ddiv_rn(r, hij);
    if (q <= 3.0) {
      if (idx) {
        idx[base + cnt] = pj;
        hij_out[base + cnt] = hij;
        q_out[base + cnt] = q;
        r_out[base + cnt] = r;
      }
      cnt++;
    }
  });
  if (!idx) {
    counts[k] = cnt;
    return;
  }
  sort_ref_order(idx + base, hij_out + base, q_out + base, r_out + base, cnt, refcell, g.ncx, qref);
}

// Every slot j of the stencil, spread over the lanes of a warp (all call it
// with the same stencil; pre: 33 words of shared memory of the warp's own).
// Up to 32 rows at a time: lane r loads row r's bounds, so a probe waits once
// for all of them, and the lanes then share the rows' candidates as one
// range: visit(j, valid), called by all lanes together.  Columns over several
// tiles go by whole rows per lane: lone(j), called by each lane for itself.
template <class F, class G>
__device__ __forceinline__ void warp_stencil(const Stencil &sten, const unsigned int *__restrict__ cstart,
                                             unsigned int *pre, F &&visit, G &&lone) {
  const int lane = threadIdx.x & 31;
  if (sten.multi) {
    const int m = (1 << sten.ts) - 1;
    for (int yy = sten.y0 + lane; yy <= sten.y1; yy += 32) {
      const unsigned int *c = cstart + sten.rowpart(yy);
      for (int xs = sten.x0; xs <= sten.x1; xs = (xs | m) + 1) {
        const unsigned int e = __ldg(c + Stencil::colpart(min(sten.x1, xs | m), sten.ts) + 1);
        for (unsigned int j = __ldg(c + Stencil::colpart(xs, sten.ts)); j < e; j++) lone(j);
      }
    }
    return;
  }
  for (int y0 = sten.y0; y0 <= sten.y1; y0 += 32) {
    const int yy = y0 + lane;
    unsigned int s0 = 0, e0 = 0, jump = 0, len = 0;
    if (yy <= sten.y1) {
      const unsigned int *c = cstart + sten.rowpart(yy);
      s0 = __ldg(c + sten.ca);
      e0 = __ldg(c + sten.cb);
      const unsigned int s1 = __ldg(c + sten.cc), e1 = __ldg(c + sten.cd);
      jump = s1 - e0;
      len = (e0 - s0) + (e1 - s1);
    }
    unsigned int inc = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    __syncwarp();
    pre[lane + 1] = inc;
    if (lane == 0) pre[0] = 0;
    __syncwarp();
    const unsigned int total = pre[32];
    for (unsigned int t0 = 0; t0 < total; t0 += 32) {
      const unsigned int t = t0 + lane;
      int r = 0;  // the row of candidate t: the last whose prefix is <= t
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        if (pre[r + o] <= t) r += o;
      const unsigned int rs0 = __shfl_sync(0xffffffffu, s0, r), re0 = __shfl_sync(0xffffffffu, e0, r);
      const unsigned int rj = __shfl_sync(0xffffffffu, jump, r);
      const unsigned int j = rs0 + (t - pre[r]);
      visit(j >= re0 ? j + rj : j, t < total);
    }
  }
}

// rho = sum_fluid m_j W(r_j, hk) / sum_{fluid, rho_j >= 1e-3} W(r_j, hk) m_j / rho_j over
// the nearPos set of (x, y, h_search); p = B ((rho / rho0)^gamma - 1).
// One warp per point: a probe has some 140 candidates, and walking them in
// one thread was a serial chain of loads and FP64 square roots and divisions.
// The FP64 pipe then bounds it, so the candidates first pass a test of 4 FP64
// operations (the rest of it in FP32, padded), and the members that are left,
// compacted into a list, take one round or two of the rest.  The q <= 3
// decision takes the correctly rounded operations within 1e-9 of the edge.
// 2000 points in a 200K-particle column: 757 us with a thread per point, 60
// with a warp each and one pow per point, 38 so (ncu, cold caches).
constexpr int kProbeBlock = 256;
template <int KERNEL>
__global__ void __launch_bounds__(kProbeBlock)
    k_probe_density(const double *__restrict__ px, const double *__restrict__ py, const double *__restrict__ ph,
                    const double *__restrict__ hk, long long np, StepArgs a, const int *__restrict__ perm,
                    const int2 *__restrict__ meta, const unsigned int *__restrict__ cstart,
                    const DevGrid *__restrict__ gp, double rho0, double B, double gamma, double *rho_out,
                    double *p_out) {
  constexpr int kList = 64;
  __shared__ unsigned int pre_all[kProbeBlock / 32][33];
  __shared__ int list_all[kProbeBlock / 32][kList];
  const DevGrid &g = *gp;
  __shared__ double rho_all[kProbeBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long k0 = (long long)blockIdx.x * (kProbeBlock / 32);
  const long long k = k0 + warp < np ? k0 + warp : np - 1;  // the last block's spare warps repeat the last point
  int *list = list_all[warp];
  const double xi = px[k], yi = py[k], hi = ph[k], hw = hk[k];
  const float hif = d2f_trunc(hi);
  const double ihw = 1.0 / hw;
  const double al = (KERNEL == SPH_KERNEL_CUBIC ? kCubicFac : (KERNEL == SPH_KERNEL_WENDLAND ? kWendFac : kInvPi)) /
                    (hw * hw);
  int2 qref;
  int W;
  const int qkey = probe_cell(g, xi, yi, hi, qref, W);
  const bool filter = g.mode == 1;
  double shep = 0.0, sum = 0.0;
  unsigned int nf = 0;
  // r <= 3 h_ij up to the padding; a negative h_ij (a negative search length)
  // has every particle inside
  auto close = [&](unsigned int j, int &pj) {
    if (filter && !in_ref_stencil(meta, j, g, qref)) return false;
    pj = perm[j];
    const double xj = a.x[pj], yj = a.y[pj];
    const float s = hif + d2f_trunc(a.h[pj]);
    if (!is_fluid(a.label[pj])) return false;  // Shepard and SummationDensity take fluid only
    const double dx = xi - xj, dy = yi - yj;
    const float d2 = d2f_trunc(fma(dx, dx, dy * dy));
    return hif < 0.f || !(d2 > 2.25f * 1.00001f * (s * s));
  };
  auto member = [&](int pj) {
    const double xj = a.x[pj], yj = a.y[pj], hj = a.h[pj], m = a.m[pj], rho = a.rho[pj];
    const double dx = xi - xj, dy = yi - yj;
    const double d2 = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
    const double hij = __dmul_rn(0.5, __dadd_rn(hi, hj));
    const double t = 9.0 * hij * hij;
    if (!(d2 < t * (1.0 - 1e-9)) && !(__ddiv_rn(__dsqrt_rn(d2), hij) <= 3.0)) return;
    double r = 0.0, ir;
    if (d2 > 0.0) sqrt_rsqrt64(quad64(d2), r, ir);
    // W(r, hw) (CubicSpline.py:12-36, Wendland.py:10-34, Gaussian.py:16-24)
    const double q = r * ihw;
    double w = 0.0;
    if (KERNEL == SPH_KERNEL_CUBIC) {
      const double c = 2.0 - q;
      if (q <= 1.0) w = al * (1.0 - 1.5 * (q * q) * (1.0 - 0.5 * q));
      else if (!(q > 2.0)) w = al * 0.25 * (c * c * c);
    } else if (KERNEL == SPH_KERNEL_WENDLAND) {
      const double c = 1.0 - 0.5 * q, c2 = c * c;
      if (!(q >= 2.0)) w = al * (c2 * c2 * c2 * ((35.0 / 12.0) * q * q + 3.0 * q + 1.0));
    } else if (fabs(q) < 3.0 * (1.0 - 1e-9) || r / hw <= 3.0) {
      w = al * (q < 0.0 ? exp(-q * q) : exp_neg(q * q));
    }
    const double mw = m * w;
    if (!(rho < 1e-3)) shep = rho < 1e300 ? fma(mw, rcp64(rho), shep) : shep + mw / rho;
    sum += mw;
    nf++;
  };
  int nl = 0;
  auto members = [&]() {
    __syncwarp();
    for (int t = lane; t < nl; t += 32) member(list[t]);
    nl = 0;
    __syncwarp();
  };
  const Stencil sten(g, qref, qkey, W);
  warp_stencil(
      sten, cstart, pre_all[warp],
      [&](unsigned int j, bool valid) {
        int pj = 0;
        const bool in = valid && close(j, pj);
        const unsigned int b = __ballot_sync(0xffffffffu, in);
        if (in) list[nl + __popc(b & ((1u << lane) - 1u))] = pj;
        nl += __popc(b);
        if (nl > kList - 32) members();
      },
      [&](unsigned int j) {
        int pj;
        if (close(j, pj)) member(pj);
      });
  members();
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    shep += __shfl_xor_sync(0xffffffffu, shep, o);
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
  }
  nf = __reduce_add_sync(0xffffffffu, nf);
  if (lane == 0) rho_all[warp] = nf ? sum / shep : 0.0;  // an empty sum without fluid neighbours
  __syncthreads();
  // the EOS of the block's points side by side: one pow for the block
  if (threadIdx.x < kProbeBlock / 32 && k0 + threadIdx.x < np) {
    const double rho = rho_all[threadIdx.x];
    rho_out[k0 + threadIdx.x] = rho;
    p_out[k0 + threadIdx.x] = (pow(rho / rho0, gamma) - 1.0) * B;
  }
}

void launch_nn_probe(const StepArgs &a, const WsPtrs &w, long long np, const double *px, const double *py,
                     const double *ph, int64_t *counts, const int64_t *offsets, int64_t *idx, double *hij, double *q,
                     double *r, cudaStream_t st) {
  k_nn_probe<<<nblocks(np, kPairBlock), kPairBlock, 0, st>>>(px, py, ph, np, a.x, a.y, a.h, w.perm, w.meta,
                                                              w.refcell, w.cstart, w.grid, counts, offsets, idx,
                                                              hij, q, r);
}

void launch_probe_density(const StepArgs &a, const WsPtrs &w, int kernel, long long np, const double *px,
                          const double *py, const double *ph, const double *hk, double rho0, double B, double gamma,
                          double *rho, double *p, cudaStream_t st) {
  const unsigned nb = nblocks(np * 32, kProbeBlock);
  if (kernel == SPH_KERNEL_CUBIC)
    k_probe_density<SPH_KERNEL_CUBIC><<<nb, kProbeBlock, 0, st>>>(px, py, ph, hk, np, a, w.perm, w.meta, w.cstart,
                                                                  w.grid, rho0, B, gamma, rho, p);
  else if (kernel == SPH_KERNEL_WENDLAND)
    k_probe_density<SPH_KERNEL_WENDLAND><<<nb, kProbeBlock, 0, st>>>(px, py, ph, hk, np, a, w.perm, w.meta, w.cstart,
                                                                     w.grid, rho0, B, gamma, rho, p);
  else
    k_probe_density<SPH_KERNEL_GAUSSIAN><<<nb, kProbeBlock, 0, st>>>(px, py, ph, hk, np, a, w.perm, w.meta, w.cstart,
                                                                     w.grid, rho0, B, gamma, rho, p);
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
int sm_count() {
  static int cache[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 152;
  if (!cache[dev]) {
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    cache[dev] = v > 0 ? v : 152;
  }
  return cache[dev];
}

// Dynamic shared memory of a tile kernel: allowed above 48 KB once per device
// and kernel (the attribute belongs to the kernel function on a device).
// `done` is the calling launcher's own flag array: every tile kernel
// instantiation has the same function type, so the flag cannot live here.
template <typename K>
static size_t tile_smem(K kern, size_t bytes, bool (&done)[64]) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !done[dev]) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (dev >= 0 && dev < 64) done[dev] = true;
  }
  return bytes;
}

template <int KERNEL, bool XSPH, bool SUMDENS, bool UH>
static void mixed_pair_launch(const StepArgs &a, const WsPtrs &w, const PairParams &pp, double *dt_out,
                              double *dt_hist, cudaStream_t st) {
  // persistent tile kernel, then the global path over what it left
  const int sms = sm_count();
  auto tk = k_pair_tiles<KERNEL, XSPH, SUMDENS, UH>;
  static bool done[64] = {false};  // this instantiation's attribute, per device
  const size_t smem = tile_smem(tk, sizeof(TileShared<KERNEL>), done);
  launch_pdl(tk, dim3(sms * TileBlocks<KERNEL>::value), dim3(kTileThreads), smem, st, a, pair_ptrs(w), pp, w.tiles,
             w.tiles_h, (unsigned)(w.max_cells + 1), w.fb, (unsigned)w.fb_cap);
  launch_pdl(k_pair_list<KERNEL, XSPH, SUMDENS, UH>, dim3(sms * kListBlocks), dim3(kPairBlock), 0, st, a,
             pair_ptrs(w), pp, w.fb, dt_out, dt_hist);
}

template <int KERNEL, bool XSPH, bool SUMDENS>
static void pair_dispatch(const StepArgs &a, const WsPtrs &w, const sph_config_t &cfg, const PairParams &pp,
                          double *dt_out, double *dt_hist, cudaStream_t st) {
  // a fixed h makes every fluid record's h the same (the uniform-h form,
  // taken when the viscosity's beta is 0)
  if (cfg.h_fixed > 0.0 && pp.beta == 0.0) mixed_pair_launch<KERNEL, XSPH, SUMDENS, true>(a, w, pp, dt_out, dt_hist, st);
  else mixed_pair_launch<KERNEL, XSPH, SUMDENS, false>(a, w, pp, dt_out, dt_hist, st);
}

void launch_pair(const StepArgs &a, const WsPtrs &w, const sph_config_t &cfg, const sph_wcsph_t &wc,
                 double *dt_out, double *dt_hist, cudaStream_t st, const WallLoad *wall, bool write_state) {
  PairParams pp = pair_params(a, cfg, wc, dt_out != nullptr || dt_hist != nullptr);
  pp.write_xsph = write_state ? 1 : 0;
  if (wall) {
    pp.wall_x = wall->wall_x;
    pp.fr = wall->fr;
  }
  if (cfg.precision != SPH_PREC_MIXED) {
    launch_pair64(a, w, cfg, wc, pp, dt_out, dt_hist, st);
    return;
  }
  const bool xs = wc.use_xsph != 0, sd = wc.use_summation_density != 0;
  auto go = [&](auto kern) {
    constexpr int K = decltype(kern)::value;
    if (xs) sd ? pair_dispatch<K, true, true>(a, w, cfg, pp, dt_out, dt_hist, st)
               : pair_dispatch<K, true, false>(a, w, cfg, pp, dt_out, dt_hist, st);
    else sd ? pair_dispatch<K, false, true>(a, w, cfg, pp, dt_out, dt_hist, st)
            : pair_dispatch<K, false, false>(a, w, cfg, pp, dt_out, dt_hist, st);
  };
  if (cfg.kernel == SPH_KERNEL_CUBIC) go(std::integral_constant<int, SPH_KERNEL_CUBIC>());
  else if (cfg.kernel == SPH_KERNEL_WENDLAND) go(std::integral_constant<int, SPH_KERNEL_WENDLAND>());
  else go(std::integral_constant<int, SPH_KERNEL_GAUSSIAN>());
}

void launch_sumdens(const StepArgs &a, const WsPtrs &w, const sph_config_t &cfg, const sph_wcsph_t &wc,
                    cudaStream_t st) {
  const unsigned nb = nblocks(a.n, kPairBlock);
  const bool mixed = cfg.precision == SPH_PREC_MIXED;
  const PairPtrs P = pair_ptrs(w);
  auto go = [&](auto kern) {
    constexpr int K = decltype(kern)::value;
    if (mixed) k_sumdens<K, true><<<nb, kPairBlock, 0, st>>>(a, P, a.n);
    else k_sumdens<K, false><<<nb, kPairBlock, 0, st>>>(a, P, a.n);
  };
  if (cfg.kernel == SPH_KERNEL_CUBIC) go(std::integral_constant<int, SPH_KERNEL_CUBIC>());
  else if (cfg.kernel == SPH_KERNEL_WENDLAND) go(std::integral_constant<int, SPH_KERNEL_WENDLAND>());
  else go(std::integral_constant<int, SPH_KERNEL_GAUSSIAN>());
  (void)wc;
}

void launch_nn_count(const StepArgs &a, const WsPtrs &w, int64_t *counts, const int64_t *offsets, int64_t *idx,
                     cudaStream_t st) {
  k_nn_export<<<nblocks(a.n, kPairBlock), kPairBlock, 0, st>>>(a.x, a.y, a.h, a.n, w.perm, w.keys_sorted, w.meta,
                                                               w.refcell, w.cstart, w.grid, counts, offsets, idx);
}

template <int KERNEL, bool XSPH, bool SUMDENS>
static void bt_pair_dispatch(const StepArgs &a, const WsPtrs &w, const BatchPtrs &B, int tile_blocks,
                             cudaStream_t st) {
  const int sms = sm_count();
  if (tile_blocks < 1 || tile_blocks > TileBlocks<KERNEL>::value) tile_blocks = TileBlocks<KERNEL>::value;
  auto tk = k_bt_pair_tiles<KERNEL, XSPH, SUMDENS>;
  static bool done[64] = {false};  // this instantiation's attribute, per device
  const size_t smem = tile_smem(tk, sizeof(TileShared<KERNEL>), done);
  launch_pdl(tk, dim3(sms * tile_blocks), dim3(kTileThreads), smem, st, a, pair_ptrs(w), B, w.fb, (unsigned)w.fb_cap);
  launch_pdl(k_bt_pair_list<KERNEL, XSPH, SUMDENS>, dim3(sms * kListBlocks), dim3(kPairBlock), 0, st, a, pair_ptrs(w),
             B, w.fb);
}

void launch_bt_pair(const StepArgs &a, const WsPtrs &w, const BatchPtrs &B, int kernel, bool xsph, int tile_blocks,
                    cudaStream_t st) {
  (void)xsph;  // the batched form has no XSPH
  if (kernel == SPH_KERNEL_CUBIC) bt_pair_dispatch<SPH_KERNEL_CUBIC, false, false>(a, w, B, tile_blocks, st);
  else if (kernel == SPH_KERNEL_WENDLAND) bt_pair_dispatch<SPH_KERNEL_WENDLAND, false, false>(a, w, B, tile_blocks, st);
  else bt_pair_dispatch<SPH_KERNEL_GAUSSIAN, false, false>(a, w, B, tile_blocks, st);
}

}  // namespace sph
