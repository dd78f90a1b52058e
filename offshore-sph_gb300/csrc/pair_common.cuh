// pair_common.cuh -- what the pair kernels of both precision forms share:
// their pointers and parameters, the exact neighbour count of the queries
// that can have an empty set, and the TimeStep epilogue.
#pragma once

#include "sph_internal.cuh"

namespace sph {

constexpr int kPairBlock = 128;
constexpr int kPair64Blocks = 5;  // resident blocks per SM of the FP64 kernel (registers)
// per-thread neighbour-list capacity: above the typical number of pairs inside
// the support (about 21 for the cubic spline at h = 1.3 dx, 43 for the
// Gaussian cut at 3h), so that the mid-walk flush -- which runs divergently --
// stays rare
template <int KERNEL>
struct ListCap {
  static constexpr int value = Support<KERNEL>::q == 2 ? 32 : 64;
};

struct PairPtrs {
  const float4 *rec0, *rec1, *rec2;
  const double4_32a *r64a, *r64b;
  const int *perm, *keys_sorted;
  const int2 *meta;
  const unsigned int *cstart;
  const DevGrid *grid;
  DevCtrl *ctrl;
};

inline PairPtrs pair_ptrs(const WsPtrs &w) {
  PairPtrs P;
  P.rec0 = w.rec0; P.rec1 = w.rec1; P.rec2 = w.rec2; P.r64a = w.rec64a; P.r64b = w.rec64b;
  P.perm = w.perm; P.keys_sorted = w.keys_sorted; P.meta = w.meta; P.cstart = w.cstart;
  P.grid = w.grid; P.ctrl = w.ctrl;
  return P;
}

// The FP32 constants of pp (alpha, beta, ... set) for a kernel and a fixed h
// (h <= 0: none, the uniform-h constants are not used).
inline void mixed_constants(PairParams &pp, int kernel, double h_fixed) {
  MixedConsts &c = pp.mc;
  const float support = kernel == SPH_KERNEL_GAUSSIAN ? 3.f : 2.f;
  c.KC = support * support;  // (support / h)^2
  const float r0f = (float)pp.r0;
  c.r02f = r0f * r0f;
  c.co = (float)pp.co;
  c.alpha = (float)pp.alpha;
  c.beta = (float)pp.beta;
  c.eps = (float)pp.eps;
  c.D = (float)pp.D;
  UniformQ &u = pp.u;
  const float h = h_fixed > 0.0 ? (float)h_fixed : 1.f;
  u.h = h;
  u.lim = c.KC * (h * h);
  u.inv_h = 1.0f / h;
  u.al = (float)(kernel == SPH_KERNEL_CUBIC ? kCubicFac : (kernel == SPH_KERNEL_WENDLAND ? kWendFac : kInvPi)) * u.inv_h *
         u.inv_h;
  const float alh = u.al * u.inv_h;
  if (kernel == SPH_KERNEL_CUBIC) {
    // dW/dr / r = al/h (-0.75 (2 - q)^2) / r (q > 1), al/h q (2.25 q - 3) / r (q <= 1)
    u.g0 = -0.75f * alh;
    u.g1 = 2.25f * alh;
    u.g2 = -3.0f * alh;
  } else if (kernel == SPH_KERNEL_WENDLAND) {
    // dW/dr / r = al/h (1 - q/2)^5 q (-14/3 - 35/3 q) / r
    u.g0 = (-14.0f / 3.0f) * alh;
    u.g1 = (-35.0f / 3.0f) * alh;
    u.g2 = 0.f;
  } else {
    // dW/dr / r = -2 al / h^2 exp(-q^2)
    u.g0 = -2.0f * alh * u.inv_h;
    u.g1 = u.g2 = 0.f;
  }
  u.hb2 = 0.01f * (h * h);
  u.pic = -2.0f * (c.alpha * 0.5f * c.co) * h;
}

inline PairParams pair_params(const StepArgs &a, const sph_config_t &cfg, const sph_wcsph_t &wc, bool do_dt) {
  PairParams pp;
  pp.write_xsph = 1;
  pp.wall_x = 0.0;
  pp.fr = nullptr;
  pp.alpha = wc.alpha; pp.beta = wc.beta; pp.co = wc.co; pp.eps = wc.epsilon;
  pp.r0 = wc.r0; pp.D = wc.D; pp.p1 = wc.p1; pp.p2 = wc.p2;
  pp.lj_42 = (wc.p1 == 4.0 && wc.p2 == 2.0) ? 1 : 0;
  pp.cfl_c = cfg.cfl_c; pp.cfl_f = cfg.cfl_f;
  pp.do_dt = do_dt ? 1 : 0;
  pp.n = a.n;
  mixed_constants(pp, cfg.kernel, cfg.h_fixed);
  return pp;
}

// Entries of a query's list for G lanes per query, cap being one thread's: a
// round adds up to G entries, and the list is evaluated early when another
// round might not fit.
template <int G>
constexpr int list_words(int cap) {
  return G == 1 ? cap : (G == 32 ? 3 * cap : cap + cap / 2);
}

// The neighbours of a query, for the kernels whose work per pair is long: the
// candidates of its stencil that near accepts are listed first, in candidate
// order, and pair(j) then runs over the list, so that the lanes of a warp run
// the long part together.  near.load(j) reads what near.test(j, record)
// decides on.  G lanes share a query (all lanes of the warp call this; act: the
// query exists): they test G candidates at a time, append by ballot, and take
// every G-th entry each, so a query's sums depend on G and its candidate order
// alone.  G = 1 is one query per thread.
// With G lanes the scene is small and latency is the time: the lanes load the
// stencil rows' bounds together and walk the rows as one range, two rounds of
// candidate loads in flight.  Row by row, the walk took 11.4K of the 27K cycles
// of a block of the FP64 kernel (3200-particle tank, G = 8).
// lists: CAP * BLOCK / G words of shared memory of the block.
template <int G, int CAP, int BLOCK, class Near, class Pair>
__device__ __forceinline__ void for_neighbours(const Stencil &sten, const unsigned int *__restrict__ cstart, bool act,
                                               unsigned int *lists, const Near &near, Pair &&pair) {
  const int tid = threadIdx.x;
  if constexpr (G == 1) {
    if (!act) return;
    auto physics = [&](int cnt) {
      for (int t = 0; t < cnt; t++) pair(lists[t * BLOCK + tid]);
    };
    int nl = 0;
    for_stencil(sten, cstart, [&](unsigned int j) {
      if (near.test(j, near.load(j))) {
        lists[nl * BLOCK + tid] = j;
        if (++nl == CAP) {
          physics(nl);
          nl = 0;
        }
      }
    });
    physics(nl);
  } else {
    constexpr unsigned int full = 0xffffffffu;
    const int gl = tid % G, lane = tid & 31;
    unsigned int *list = lists + tid / G * CAP;
    const unsigned int gmask = (G == 32 ? full : ((1u << (G % 32)) - 1u)) << (lane & ~(G - 1));
    const unsigned int below = gmask & ((1u << lane) - 1u);
    int nl = 0;
    auto physics = [&]() {
      for (int t = gl; t < nl; t += G) pair(list[t]);
    };
    auto append = [&](unsigned int j, bool keep) {
      const unsigned int b = __ballot_sync(full, keep) & gmask;
      if (keep) list[nl + __popc(b & below)] = j;
      nl += __popc(b);
      if (__any_sync(full, nl > CAP - G)) {  // no room for another round
        __syncwarp();
        if (nl > CAP - G) {
          physics();
          nl = 0;
        }
        __syncwarp();
      }
    };
    const int nr = act ? max(sten.y1 - sten.y0 + 1, 0) : 0;
    if (!__any_sync(full, nr > G || (act && sten.multi))) {
      // lane r holds row r: candidates [first, last) of the flat range are
      // slots base + t, from e0 on moved by jump (the second tile segment)
      unsigned int s0 = 0, e0 = 0, jump = 0, len = 0;
      if (gl < nr) {
        const unsigned int *c = cstart + sten.rowpart(sten.y0 + gl);
        s0 = __ldg(c + sten.ca);
        e0 = __ldg(c + sten.cb);
        const unsigned int s1 = __ldg(c + sten.cc), e1 = __ldg(c + sten.cd);
        jump = s1 - e0;
        len = (e0 - s0) + (e1 - s1);
      }
      unsigned int last = len;
#pragma unroll
      for (int o = 1; o < G; o <<= 1) {
        const unsigned int v = __shfl_up_sync(full, last, o, G);
        if (gl >= o) last += v;
      }
      const unsigned int base = s0 - (last - len), total = __shfl_sync(full, last, G - 1, G);
      const int rows = (int)__reduce_max_sync(full, (unsigned)nr);
      auto slot = [&](unsigned int t) {
        int r = 0;
        for (int q = 0; q < rows - 1; q++) r += t >= __shfl_sync(full, last, q, G) ? 1 : 0;
        const unsigned int j = __shfl_sync(full, base, r, G) + t;
        const unsigned int e = __shfl_sync(full, e0, r, G), s = __shfl_sync(full, jump, r, G);
        return j >= e ? j + s : j;
      };
      for (unsigned int t0 = 0; __any_sync(full, t0 < total); t0 += 2 * G) {
        const unsigned int ta = t0 + gl, tb = ta + G;
        const unsigned int ja = slot(ta), jb = slot(tb);
        float4 qa = make_float4(0.f, 0.f, 0.f, 0.f), qb = qa;
        if (ta < total) qa = near.load(ja);
        if (tb < total) qb = near.load(jb);
        append(ja, ta < total && near.test(ja, qa));
        append(jb, tb < total && near.test(jb, qb));
      }
    } else {
      // wide stencils (queries whose own cell is not in theirs) or columns
      // over several tiles: row by row, tile by tile
      const int rows = (int)__reduce_max_sync(full, (unsigned)nr);
      const int m = (1 << sten.ts) - 1;
      for (int r = 0; r < rows; r++) {
        const bool on = r < nr;
        const unsigned int *c = cstart + (on ? sten.rowpart(sten.y0 + r) : 0);
        for (int xs = sten.x0; __any_sync(full, on && xs <= sten.x1); xs = (xs | m) + 1) {
          unsigned int j = 0, e = 0;
          if (on && xs <= sten.x1) {
            j = __ldg(c + Stencil::colpart(xs, sten.ts));
            e = __ldg(c + Stencil::colpart(min(sten.x1, xs | m), sten.ts) + 1);
          }
          for (j += gl; __any_sync(full, j - gl < e); j += G)
            append(j, j < e && near.test(j, near.load(j)));
        }
      }
    }
    __syncwarp();
    physics();
  }
}

// sum over the G lanes of a query
template <int G, class T>
__device__ __forceinline__ void group_sum(T &v) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
}

// Lanes per query of the FP64 kernels for n particles, and of the adjoint's.
// Sharing a query divides the length of a thread's chain of dependent operations
// and costs issue time (short groups, the final sums).  Pair stage in us with 1 and
// 4 lanes, by sizes in waves of one query per thread (97,280 on 152 SMs); a tank's
// walls count as queries, which end at once:
//
//   lattice  cubic, fixed h  Wendland, fixed h  cubic, computed h  Gaussian
//   0.05         56  28            57  29             75  31          91  34
//   0.12         55  31            56  32             76  40          91  38
//   0.49         65  60            72  70            110 101         109  88
//   0.52         64  76            71  88            110 116         109 108
//   1.02        117 124           140 146            214 195         220 174
//   1.25        125 136           152 158            231 230         242 201
//   1.5         131 162           165 187            256 270         250 237
//   2.25        188 236           235 276            372 391         363 344
//   3.9         272 403           352 475            603 652         533 570
//   tank
//   0.97         81 108           101 126            171 192         156 178
//   1.07        117 123           138 141            222 204         227 190
//   1.2         131 131           173 154            275 235         274 216
//   1.4         136 154           179 181            288 278         280 252
//   1.75        141 183           182 214            301 329         286 302
//   2.25        189 232           247 272            375 418         406 381
//
// With 8 lanes: cubic, fixed h 18, 41 and 97 at 0.05, 0.125 and 0.5.  So G = 8
// where the GPU is idle and the chain is the time, G = 4 up to half a wave, and
// from there on G = 1 where the last wave is full enough: always with the cubic
// at a fixed h, whose pairs are short; the Gaussian's long pairs are worth sharing
// while the last wave is at most half full, up to 4 waves, those of a computed h
// in the first three eighths of the second wave, and Wendland's at a fixed h in
// the first quarter.  The adjoint (cubic, FP64: 204
// and 207 us at 1.03 waves, 263 and 282 at 1.46; mixed 123 and 161 at 1.46) does
// not share, but for the Gaussian's: mixed, 217 and 178 us at 1.0 waves, 318 and
// 303 at 1.8, 418 and 417 at 2.6, its FP64 form within 3%.
inline int lanes_per_query(long long n, int kernel = SPH_KERNEL_CUBIC, bool uniform_h = true, bool adjoint = false) {
  const long long wave = (long long)sm_count() * kPairBlock * kPair64Blocks;
  if (n < wave / 8) return 8;
  if (n < wave / 2) return 4;
  if (n <= wave || n >= 4 * wave) return 1;
  if (kernel == SPH_KERNEL_GAUSSIAN) return adjoint || n % wave <= wave / 2 ? 4 : 1;
  if (adjoint || (kernel == SPH_KERNEL_CUBIC && uniform_h)) return 1;
  return n <= wave + (uniform_h ? 2 : 3) * wave / 8 ? 4 : 1;
}

// Exact size of the reference's neighbour set of a query whose own cell is
// not in its stencil (x-overflow alias) or whose h is not positive; those are
// the only queries that can have an empty set (src/Tools/SolverTools.py:150-153).
static __device__ int exact_count(const StepArgs &a, const int *__restrict__ perm, const DevGrid &g, int2 qref, int qkey,
                           int W, bool filter, const int2 *__restrict__ meta, const unsigned int *__restrict__ cstart,
                           double xi, double yi, double hi) {
  const Stencil sten(g, qref, qkey, W);
  int cnt = 0;
  for_stencil(sten, cstart, [&](unsigned int j) {
    if (filter && !in_ref_stencil(meta, j, g, qref)) return;
    const int pj = perm[j];
    const double dx = xi - a.x[pj], dy = yi - a.y[pj];
    const double r = __dsqrt_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)));
    const double q = __ddiv_rn(r, __dmul_rn(0.5, __dadd_rn(hi, a.h[pj])));
    if (q <= 3.0) cnt++;
  });
  return cnt;
}

// TimeStep epilogue: the block's max a^2 over fluid; the last block computes
// {dt, dt_courant, dt_force} (TimeStep.py:7-56) from the min h the records
// pass gathered, and resets the slots.
__device__ __forceinline__ void timestep_epilogue(DevCtrl *ctrl, unsigned long long ea, double co, double cfl_c,
                                                  double cfl_f, double *dt_out, double *dt_hist,
                                                  unsigned int *zero_on_last = nullptr,
                                                  unsigned int nblocks = 0 /* 0: every block of the grid */) {
  __shared__ unsigned long long red[kPairBlock / 32];
  __shared__ bool last;
  const unsigned int nb = nblocks ? nblocks : gridDim.x;
  const unsigned long long wm = warp_max_u64(ea);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = wm;
  __syncthreads();
  unsigned long long ba = kEncMaxId;
  if (threadIdx.x == 0) {
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) ba = red[w] > ba ? red[w] : ba;
    if (nb == 1) {
      last = true;
    } else {
      if (ba != kEncMaxId) atomicMax(&ctrl->pd_a2max, ba);
      __threadfence();
      last = atomicAdd(&ctrl->done_pair, 1u) == nb - 1;
    }
  }
  __syncthreads();
  if (last && threadIdx.x == 0) {
    unsigned long long eh, ea2;
    unsigned int cnt;
    if (nb == 1) {
      // the only block: the other contributions came from kernels that
      // completed before this one started, so plain loads see them (one
      // round trip instead of a fence and a chain of returning atomics)
      eh = __ldcg(&ctrl->pd_hmin);
      ea2 = __ldcg(&ctrl->pd_a2max);
      cnt = __ldcg(&ctrl->pd_nfluid);
      ea2 = ba > ea2 ? ba : ea2;
    } else {
      // every other block has added its share (and fenced): L2 loads see it
      __threadfence();
      eh = __ldcg(&ctrl->pd_hmin);
      ea2 = __ldcg(&ctrl->pd_a2max);
      cnt = __ldcg(&ctrl->pd_nfluid);
      ctrl->done_pair = 0u;
    }
    ctrl->pd_hmin = kEncMinId;
    ctrl->pd_a2max = kEncMaxId;
    ctrl->pd_nfluid = 0u;
    if (zero_on_last) *zero_on_last = 0u;
    const double min_h = dec_d(eh);
    const double max_a2 = dec_d(ea2);
    const double max_c = co;  // compute_speed_of_sound gives co to every particle (WCSPH.py:110-129)
    double dc = __ddiv_rn(__dmul_rn(cfl_c, min_h), max_c);
    double df = max_a2 < 1e-12 ? 1e10 : __dmul_rn(cfl_f, __dsqrt_rn(__ddiv_rn(min_h, max_a2)));
    double dt = (df < dc) ? df : dc;  // Python min(c, f) keeps c on ties
    unsigned st = 0;
    if (cnt == 0) {
      st |= SPH_STATUS_NO_FLUID;
      dt = dc = df = nan("");
    }
    if (dt < 1e-6) st |= SPH_STATUS_SMALL_DT;
    if (st) atomicOr(&ctrl->status, st);
    if (dt_out) {
      dt_out[0] = dt;
      dt_out[1] = dc;
      dt_out[2] = df;
    }
    if (dt_hist) {
      dt_hist[0] = dt;
      dt_hist[1] = dc;
      dt_hist[2] = df;
    }
  }
}

// a^2 as TimeStep.computeVars forms it (no contraction)
__device__ __forceinline__ double accel2(double ax, double ay) {
  return __dadd_rn(__dmul_rn(ax, ax), __dmul_rn(ay, ay));
}

}  // namespace sph
