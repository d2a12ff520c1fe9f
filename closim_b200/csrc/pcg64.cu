// PCG of the FP64 path (pcg.ts:11-95) with the Newton epilogue
// (newton.ts:152-179), one persistent launch. Compiled with -fmad=false: every
// element result, vertex sum and dot product has the reference's rounding.
//
// The solve is bound by latency: a sheet's vectors fit on chip, and an
// iteration is a chain of dependent phases. So each CTA owns a contiguous range
// of vertices for the whole solve and keeps their vectors in shared memory; it
// evaluates every triangle incident to them (the finite-difference HVP's two
// gradients, one thread each) into shared memory, so the vertex sums need no
// barrier across CTAs; and the dot products, which the reference adds left to
// right, are ordered sums (ordered_sum.cuh) spread over the CTAs: every CTA
// publishes the stages of its own range, and after a barrier every CTA walks
// all of them. A stage needs an approximate start; those of |r|^2, r.z and
// |p|^2 come from recurrences in alpha and beta over sums published one phase
// earlier, so each costs one barrier. Sheets up to kPcg64SingleN vertices run in
// one CTA, which adds the terms one by one, sheets up to kPcg64ClusterN in one
// 16-CTA cluster (hardware barrier), larger ones on the whole grid.
// On a B200 against one-thread chains on a cooperative grid, us per iteration: 41 x 9
// strip (Jacobi) 43 -> 32, 64 x 64 drape Jacobi 202 -> 45, Schwarz 409 -> 84, 121 x 121 drape
// Jacobi 645 -> 69, Schwarz 1,100 -> 104, the same bits. A dot
// product now costs its stages (4,500-8,500 cycles), one or two barriers (3,000-6,500
// each) and a walk over all stages (4,000-20,000); Schwarz adds the domains' substitution
// chains, 54,000 of 175,000 cycles at 64 x 64.
#include <cooperative_groups.h>

#include <algorithm>
#include <map>
#include <mutex>

#include "contact.cuh"
#include "pcg64.cuh"
#include "schwarz64.cuh"
#include "setup.hpp"

namespace cg = cooperative_groups;

namespace cs {

namespace {

struct Args {
  Dev d;
  Pcg64Plan P;
  int maxIters;
  double tol;
};

enum Kind { D_PAP = 0, D_RR, D_RZ, D_PP };
enum Row { W_PAP = 0, W_RR, W_RAP, W_APAP, W_RZ, W_ZAP, W_ADA, W_ZZ, W_ZP, W_PP, W_MAX };

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Segment `r` of this CTA: the lane's chunk [l0, l0 + cnt) of the nt local terms.
struct Chunk {
  int l0, cnt;
};
__device__ __forceinline__ Chunk seg_chunk(const Pcg64Plan& P, int r, int nt) {
  const int lane = threadIdx.x & 31;
  Chunk c;
  c.l0 = min(nt, (r * 32 + lane) * P.K);
  c.cnt = min(P.K, nt - c.l0);
  return c;
}

// The functions below are called from several places of a kernel whose loop body
// is run through once per iteration: inlined, the body outgrew the instruction
// cache and every phase waited for its code.

// Approximate sum of a row's segments before `seg` (every lane gets it).
__device__ __noinline__ double seg_before(const double* row, int seg) {
  const int lane = threadIdx.x & 31;
  double s = 0;
  for (int i = lane; i < seg; i += 32) s += __ldcg(row + i);
  return wsum(s);
}

// The same for three rows (`stride` apart) combined with weights, their loads in flight together.
__device__ __noinline__ double seg_before3(const double* row, size_t stride, int seg, double w1, double w2) {
  const int lane = threadIdx.x & 31;
  double s = 0;
  for (int i = lane; i < seg; i += 32) {
    const double a = __ldcg(row + i), b = __ldcg(row + stride + i), c = __ldcg(row + 2 * stride + i);
    s += a + w1 * b + w2 * c;
  }
  return wsum(s);
}

// Publishes the stages of a segment, as one map where they collapse: the first at
// `head` (contiguous over the segments, all a walk usually reads), a longer list at `out`. The
// lane's chunk of the local terms t, g0 + c.l0 its place in the whole sum, `before`
// the approximate sum before the segment (first: it begins the sum). mine: one
// warp's scratch.
__device__ __noinline__ void seg_order(OrdStage* head, OrdStage* out, const double* t, int g0, Chunk c, double before,
                                       bool first, OrdStage* mine) {
  const int lane = threadIdx.x & 31;
  if (first) {
    const int end = __shfl_sync(0xffffffffu, c.l0 + c.cnt, 31);
    ord_constant(mine, ord_seq_warp(0, end, ord_bits(0.0), [&](int j) { return t[j]; }));
  } else {
    double s = 0;
    for (int j = 0; j < c.cnt; j++) s += t[c.l0 + j];
    double inc = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double a = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += a;
    }
    double ex = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane == 0) ex = 0.0;
    ord_warp_stages<0>([&](int j) { return t[c.l0 + j]; }, g0 + c.l0, c.cnt, before + ex, mine, kPcg64Stages);
    __syncwarp();
    ord_collapse(mine);
  }
  __syncwarp();
  const int n = mine[0].count;
  if (lane < 4) reinterpret_cast<int4*>(head)[lane] = reinterpret_cast<const int4*>(mine)[lane];
  for (int i = lane; n > 1 && i < n * 4; i += 32)
    reinterpret_cast<int4*>(out)[i] = reinterpret_cast<const int4*>(mine)[i];
  __syncwarp();
}

// The exact sums of nk (1 or 2) kinds (heads h, lists st, global terms T): every thread of the CTA
// calls it, warp q walks kind q. wst holds the first stage of each segment, loaded
// together (a longer list's rest is read as it is reached), stp their steps.
__device__ __noinline__ void walk(const OrdStage* h0, const OrdStage* h1, const OrdStage* st0, const OrdStage* st1,
                                  int nk, int NS, const double* T0, const double* T1, OrdStage* wst, OrdStep* stp,
                                  double* res) {
  for (int i = threadIdx.x; i < nk * NS * 4; i += blockDim.x) {
    const int4* src = reinterpret_cast<const int4*>(i >= NS * 4 ? h1 - NS : h0);
    reinterpret_cast<int4*>(wst)[i] = __ldcg(src + i);
  }
  __syncthreads();
  const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (q < nk) {
    const OrdStage* w = wst + q * NS;
    for (int i = lane; i < NS; i += 32) stp[q * NS + i] = ord_step(w[i], i + 1 < NS ? w[i + 1].B : ord_after(w[i]));
    __syncwarp();
    const long long b = ord_walk(ord_bits(0.0), NS, w, 1, q ? st1 : st0, kPcg64Stages, stp + q * NS, q ? T1 : T0);
    if (lane == 0) res[q] = ord_dbl(b);
  }
  __syncthreads();
}

// n terms in order by one thread, sixteen loaded together.
__device__ __noinline__ double serial_sum(const double* t, int n) {
  double p = 0.0;
  int j = 0;
  for (; j + 16 <= n; j += 16) {
    double a[16];
#pragma unroll
    for (int q = 0; q < 16; q++) a[q] = t[j + q];
#pragma unroll
    for (int q = 0; q < 16; q++) p = p + a[q];
  }
  for (; j < n; j++) p = p + t[j];
  return p;
}

// The CTAs of a launch: one, one thread-block cluster, or a cooperative grid.
// (GRID_FAR: whose contact-record offsets do not fit in shared memory).
enum Shape { ONE, CLUSTER, GRID, GRID_FAR };

template <Shape SHAPE>
__global__ void __launch_bounds__(kPcg64T, 1) k_pcg64(const __grid_constant__ Args A) {
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ double res[2];
  __shared__ double red[kPcg64T / 32];
  __shared__ OrdStage mine[kPcg64T / 32][kPcg64Stages];  // per warp: stages before they are published
  __shared__ double rec32[kPcg64T / 32][96];              // per warp: 32 contact records' shares
  const Dev& d = A.d;
  const Pcg64Plan& P = A.P;
  auto barrier = [&]() {
    if constexpr (SHAPE == ONE) __syncthreads();
    else if constexpr (SHAPE == CLUSTER) cg::this_cluster().sync();
    else cg::this_grid().sync();
  };
  constexpr int T = kPcg64T, W = T / 32;
  const int b = blockIdx.x, warp = threadIdx.x >> 5;
  const int vb0 = min(d.n, b * P.nv), nOwn = min(P.nv, d.n - vb0), nt = 3 * nOwn, g0 = 3 * vb0;
  const int NS = P.NS, R = P.R;
  const bool jacobi = d.precond == 0;
  // shared memory: walk stages, then the CTA's vectors, then its element results
  OrdStage* wst = reinterpret_cast<OrdStage*>(dyn);
  constexpr uint32_t kLight = 4;  // contact records a vertex's own thread sums
  OrdStep* stp = reinterpret_cast<OrdStep*>(wst + 2 * NS);
  double* vecS = reinterpret_cast<double*>(stp + 2 * NS);
  const int len = 3 * P.nv;
  const bool vs = P.vecSmem != 0;
  double* const lx = vs ? vecS : d.dx + g0;
  double* const lr = vs ? vecS + len : d.r + g0;
  double* const lz = vs ? vecS + 2 * len : d.z + g0;
  double* const lp = vs ? vecS + 3 * len : d.p + g0;
  double* const lAp = vs ? vecS + 4 * len : d.Ap + g0;
  double* const t0 = vs ? vecS + 5 * len : d.T0 + g0;
  double* const t1 = vs ? vecS + 6 * len : d.T1 + g0;
  double* const t2 = vs ? vecS + 7 * len : d.T2 + g0;
  double* const t3 = vs ? vecS + 8 * len : d.T3 + g0;
  double* const el = P.elemSmem ? vecS + (vs ? 9 * len : 0) : P.elem + (size_t)b * P.elemStride;
  const int s0 = P.slotOff[b], nSlot = P.slotOff[b + 1] - s0;
  // this launch's contact-record offsets of the owned vertices, at the end of the
  // shared memory where they fit
  uint32_t* const cOffS = reinterpret_cast<uint32_t*>(dyn + P.smem) - (P.nv + 1);
  if (SHAPE != GRID_FAR && d.hasContact)
    for (int i = threadIdx.x; i <= nOwn; i += T) cOffS[i] = d.c.cOff[vb0 + i];
  auto cOff = [&](int lv) { return SHAPE != GRID_FAR ? cOffS[lv] : __ldg(d.c.cOff + vb0 + lv); };
  // A term in the CTA's copy and (for a walk's fallback) in memory.
  auto term = [&](double* loc, double* glob, int i, double v) {
    loc[i] = v;
    if (vs) glob[g0 + i] = v;
  };
  auto stages = [&](int kind) { return P.stages + (size_t)kind * NS * kPcg64Stages; };
  auto heads = [&](int kind) { return P.heads + (size_t)kind * NS; };
  auto order = [&](int kind, int r, const double* t, double before) {
    const int seg = b * R + r;
    seg_order(heads(kind) + seg, stages(kind) + (size_t)seg * kPcg64Stages, t, g0, seg_chunk(P, r, nt), before,
              seg == 0, mine[warp]);
  };
  auto before = [&](int row, int r) { return seg_before(P.sums + (size_t)row * NS, b * R + r); };
  auto before3 = [&](int row, int r, double w1, double w2) {
    return seg_before3(P.sums + (size_t)row * NS, NS, b * R + r, w1, w2);
  };
  auto walk1 = [&](int kind, const double* T0) {
    walk(heads(kind), nullptr, stages(kind), nullptr, 1, NS, T0, nullptr, wst, stp, res);
  };
  auto walk2 = [&](int k0, int k1, const double* T0, const double* T1) {
    walk(heads(k0), heads(k1), stages(k0), stages(k1), 2, NS, T0, T1, wst, stp, res);
  };
  // A lone CTA holds all terms: its first two warps add one sum each (ta, tb) in order.
  constexpr bool single = SHAPE == ONE;
  auto serial = [&](const double* ta, const double* tb) {
    __syncthreads();
    if ((threadIdx.x & 31) == 0 && warp < (tb ? 2 : 1)) res[warp] = serial_sum(warp ? tb : ta, nt);
    __syncthreads();
  };
  // Warps q * R .. q * R + R - 1 order the segments of the q-th pending sum.
  auto segment = [&](int q) { return warp - q * R; };

  // ---- init: r = filter(b), z = M^-1 r, p = z (pcg.ts:27-55) ----
  for (int i = threadIdx.x; i < nt; i += T) {
    const int g = g0 + i;
    const double bi = -d.g[g];
    const bool pin = d.pinned[g / 3];
    const double ri = pin ? 0.0 : bi;
    term(t0, d.T0, i, bi * bi);
    term(t1, d.T1, i, ri * ri);
    lr[i] = ri;
    lx[i] = 0;
    if (!jacobi) d.r[g] = ri;
    else {
      double zi = d.diag[g] > 1e-12 ? ri / d.diag[g] : ri;
      if (pin) zi = 0;
      lz[i] = zi;
    }
  }
  if (d.hasContact) {
    const Contact& c = d.c;
    for (int i = b * T + threadIdx.x, na = n_active(c); i < na; i += P.G * T) {
      const double dist = js_max(frozen_dist(c, d.x, c.active[i]), 1e-12);
      P.curv[i] = dist < c.dHat ? barrier_curvature(dist, c.dHat, c.kappa) : 0.0;
    }
  }
  // the warp's first domain's facts stay in registers for the whole solve
  const int dom0 = b + warp * P.G;
  DomLane first{-1, 0, false, false};
  if (!jacobi && dom0 < d.D) first = domain_lane(d, dom0);
  auto all_domains = [&]() {
    for (int dom = dom0; dom < d.D; dom += P.G * W)
      domain_solve(d.L + (size_t)dom * 576, d.r, d.z, d.precond == 2 ? d.dcoarse + dom * 3 : nullptr,
                   dom == dom0 ? first : domain_lane(d, dom));
  };
  if (!jacobi) {
    barrier();
    all_domains();
    barrier();
  }
  for (int i = threadIdx.x; i < nt; i += T) {
    const double zi = jacobi ? lz[i] : __ldcg(d.z + g0 + i);
    lz[i] = zi;
    lp[i] = zi;
    d.p[g0 + i] = zi;
    term(t2, d.T2, i, lr[i] * zi);
    term(t3, d.T3, i, zi * zi);
  }
  __syncthreads();
  // approximate segment sums of the four initial chains
  for (int w = warp; !single && w < R * 4; w += W) {
    const int q = w / R, r = w - q * R;
    const double* t = q == 0 ? t0 : q == 1 ? t1 : q == 2 ? t2 : t3;
    const Chunk c = seg_chunk(P, r, nt);
    double s = 0;
    for (int j = 0; j < c.cnt; j++) s += t[c.l0 + j];
    s = wsum(s);
    const int row = q == 0 ? W_PAP : q == 1 ? W_RR : q == 2 ? W_RZ : W_PP;
    if ((threadIdx.x & 31) == 0) P.sums[(size_t)row * NS + b * R + r] = s;
  }
  barrier();
  for (int w = warp; !single && w < R * 4; w += W) {
    const int q = w / R, r = w - q * R;
    const double* t = q == 0 ? t0 : q == 1 ? t1 : q == 2 ? t2 : t3;
    const int row = q == 0 ? W_PAP : q == 1 ? W_RR : q == 2 ? W_RZ : W_PP;
    order(q, r, t, before(row, r));
  }
  barrier();
  if constexpr (single) serial(t0, t1);
  else walk2(D_PAP, D_RR, d.T0, d.T1);
  const double bNorm = sqrt(res[0]);
  double residual = sqrt(res[1]);
  __syncthreads();
  if constexpr (single) serial(t2, t3);
  else walk2(D_RZ, D_PP, d.T2, d.T3);
  double rz = res[0];
  double pp = res[1];
  const double absTol = js_max(A.tol * js_max(bNorm, 1e-12), 1e-12);
  int iters = 0;
  bool done = residual < absTol;
  // the first iteration rewrites the sums and terms just read by other CTAs
  barrier();
  int k = 0;
  for (; !done && k < A.maxIters; k++) {
    // ---- Ap = M/h^2 p + membraneHvp (fem.ts:108-130) + contact HVP ----
    const double h = 1e-8 * (1 + sqrt(pp));
    for (int e = threadIdx.x; e < 2 * nSlot; e += T) {
      const int4 sl = __ldg(P.slots + s0 + (e >> 1));
      const int vi[3] = {sl.x, sl.y, sl.z};
      double q[9];
#pragma unroll
      for (int c = 0; c < 3; c++)
#pragma unroll
        for (int u = 0; u < 3; u++) {
          const double xx = __ldg(d.x + vi[c] * 3 + u), hp = h * __ldcg(d.p + vi[c] * 3 + u);
          q[c * 3 + u] = (e & 1) ? xx - hp : xx + hp;
        }
      const float4 iv = __ldg(d.inv + sl.w);
      double en, g[9], E[3];
      tri_grad<double>(q, q + 3, q + 6, iv.x, iv.y, iv.z, iv.w, __ldg(d.area + sl.w), d.mat, en, g, E);
      double* o = el + (size_t)(e >> 1) * 18 + (e & 1) * 9;
#pragma unroll
      for (int u = 0; u < 9; u++) o[u] = g[u];
    }
    if (d.hasContact) {
      // the shares of the owned vertices' contact records, one record per thread
      const Contact& c = d.c;
      for (uint32_t q = cOff(0) + threadIdx.x, q1 = cOff(nOwn); q < q1; q += T) {
        const uint32_t rec = c.cRec[q];
        const double cv = __ldcg(P.curv + (rec >> 2));
        double o[3] = {0, 0, 0};
        if (cv != 0) {
          const Frozen f = c.active[rec >> 2];
          const double g = cv * dist_jvp(f, d.p);
          if (g != 0) dist_grad_slot(f, rec & 3, g, o);
        }
        double* sh = c.recScratch + (size_t)q * 3;
        sh[0] = o[0]; sh[1] = o[1]; sh[2] = o[2];
      }
    }
    __syncthreads();
    if (d.hasContact) {
      // A vertex may sit in hundreds of contacts: a warp sums its shares in order,
      // 32 records loaded together, one lane per component (into t2, free until the update).
      for (int lv = warp; lv < nOwn; lv += W) {
        const uint32_t q0 = cOff(lv), q1 = cOff(lv + 1);
        if (q1 - q0 <= kLight) continue;
        const int lane = threadIdx.x & 31;
        const double* src = d.c.recScratch + (size_t)q0 * 3;
        const int total = (int)(q1 - q0) * 3;
        double* buf = rec32[warp];
        double nx[3], acc = 0;
#pragma unroll
        for (int u = 0; u < 3; u++) nx[u] = u * 32 + lane < total ? src[u * 32 + lane] : 0.0;
        for (int i = 0; i < total; i += 96) {
          __syncwarp();
#pragma unroll
          for (int u = 0; u < 3; u++) buf[u * 32 + lane] = nx[u];
          __syncwarp();
#pragma unroll
          for (int u = 0; u < 3; u++) nx[u] = i + 96 + u * 32 + lane < total ? src[i + 96 + u * 32 + lane] : 0.0;
          if (lane < 3) {
#pragma unroll 8
            for (int u = 0; u < 32; u++) acc += buf[u * 3 + lane];  // zeros past the end
          }
        }
        if (lane < 3) t2[lv * 3 + lane] = acc;
      }
      __syncthreads();
    }
    for (int base = 0; base < nOwn; base += T / 2) {
      const int lv = base + (threadIdx.x >> 1), sg = threadIdx.x & 1;
      const bool on = lv < nOwn;
      const int v = vb0 + lv;
      double s[3] = {0, 0, 0};
      if (on)
        for (uint32_t q = __ldg(d.memOff + v), q1 = __ldg(d.memOff + v + 1); q < q1; q++) {
          const uint32_t rec = __ldg(P.inc + q);
          const double* e = el + (size_t)(rec >> 2) * 18 + sg * 9 + (rec & 3) * 3;
          s[0] += e[0]; s[1] += e[1]; s[2] += e[2];
        }
      double o[3];
#pragma unroll
      for (int c = 0; c < 3; c++) o[c] = __shfl_xor_sync(0xffffffffu, s[c], 1);
      if (!on || sg) continue;
      double ch[3] = {0, 0, 0};
      if (d.hasContact) {
        const uint32_t q0 = cOff(lv), cnt = cOff(lv + 1) - q0;
        if (cnt > kLight) {
#pragma unroll
          for (int c = 0; c < 3; c++) ch[c] = t2[lv * 3 + c];
        } else if (cnt) {
          double r[kLight][3];
#pragma unroll
          for (int u = 0; u < (int)kLight; u++)
#pragma unroll
            for (int c = 0; c < 3; c++) r[u][c] = u < (int)cnt ? d.c.recScratch[(size_t)(q0 + u) * 3 + c] : 0.0;
#pragma unroll
          for (int u = 0; u < (int)kLight; u++) { ch[0] += r[u][0]; ch[1] += r[u][1]; ch[2] += r[u][2]; }
        }
      }
      const double M = __ldg(d.mass + v);
      const bool pin = d.pinned[v];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const int i = lv * 3 + c;
        const double Hp = (s[c] - o[c]) / (2 * h);
        double ap = M * lp[i] * d.invH2 + Hp;
        if (d.hasContact) ap += ch[c];
        if (pin) ap = 0;
        lAp[i] = ap;
        term(t0, d.T0, i, lp[i] * ap);
      }
    }
    __syncthreads();
    if (!single && warp < 3 * R) {
      // approximate sums: p.Ap, and what the starts of |r|^2 and r.z will need
      const int q = warp / R, r = segment(q);
      const Chunk c = seg_chunk(P, r, nt);
      double u0 = 0, u1 = 0, u2 = 0;
      for (int j = 0; j < c.cnt; j++) {
        const int i = c.l0 + j;
        if (q == 0) u0 += t0[i];
        else if (q == 1) {
          const double ri = lr[i], ai = lAp[i];
          u0 += ri * ri; u1 += ri * ai; u2 += ai * ai;
        } else if (jacobi) {
          const double zi = lz[i], ai = lAp[i], dg = d.diag[g0 + i];
          u0 += lr[i] * zi; u1 += zi * ai; u2 += dg > 1e-12 ? ai * ai / dg : ai * ai;
        }
      }
      u0 = wsum(u0);
      if (q) { u1 = wsum(u1); u2 = wsum(u2); }
      if ((threadIdx.x & 31) == 0) {
        double* o = P.sums + b * R + r;
        if (q == 0) o[(size_t)W_PAP * NS] = u0;
        else {
          const int row = q == 1 ? W_RR : W_RZ;
          o[(size_t)row * NS] = u0; o[(size_t)(row + 1) * NS] = u1; o[(size_t)(row + 2) * NS] = u2;
        }
      }
    }
    if constexpr (single) {
      serial(t0, nullptr);
    } else {
      barrier();
      if (warp < R)
        order(D_PAP, warp, t0, before(W_PAP, warp));
      barrier();
      walk1(D_PAP, d.T0);
    }
    const double pAp = res[0];
    if (!(pAp > 1e-30)) { iters = k; done = true; break; }
    const double alpha = rz / pAp;
    for (int i = threadIdx.x; i < nt; i += T) {
      const int g = g0 + i;
      const bool pin = d.pinned[g / 3];
      double xi = lx[i] + alpha * lp[i];
      double ri = lr[i] - alpha * lAp[i];
      if (pin) { xi = 0; ri = 0; }
      lx[i] = xi;
      lr[i] = ri;
      term(t1, d.T1, i, ri * ri);
      if (!jacobi) d.r[g] = ri;
      else {
        double zi = d.diag[g] > 1e-12 ? ri / d.diag[g] : ri;
        if (pin) zi = 0;
        lz[i] = zi;
        term(t2, d.T2, i, ri * zi);
      }
    }
    __syncthreads();
    auto direction_sums = [&](int r) {  // z.z, z.p, p.p for the start of |z + beta p|^2
      const Chunk c = seg_chunk(P, r, nt);
      double u0 = 0, u1 = 0, u2 = 0;
      for (int j = 0; j < c.cnt; j++) {
        const double zi = lz[c.l0 + j], pi = lp[c.l0 + j];
        u0 += zi * zi; u1 += zi * pi; u2 += pi * pi;
      }
      u0 = wsum(u0); u1 = wsum(u1); u2 = wsum(u2);
      if ((threadIdx.x & 31) == 0) {
        double* o = P.sums + b * R + r;
        o[(size_t)W_ZZ * NS] = u0; o[(size_t)W_ZP * NS] = u1; o[(size_t)W_PP * NS] = u2;
      }
    };
    if (!single && warp < (jacobi ? 3 * R : R)) {
      const int q = warp / R, r = segment(q);
      if (q < 2) {
        const int row = q ? W_RZ : W_RR;
        order(q ? D_RZ : D_RR, r, q ? t2 : t1, before3(row, r, -2 * alpha, alpha * alpha));
      } else {
        direction_sums(r);
      }
    }
    barrier();
    if constexpr (single) serial(t1, jacobi ? t2 : nullptr);
    else walk(heads(D_RR), heads(D_RZ), stages(D_RR), stages(D_RZ), jacobi ? 2 : 1, NS, d.T1, d.T2, wst, stp, res);
    residual = sqrt(res[0]);
    double rzNew = res[1];
    if (residual < absTol) { iters = k + 1; done = true; break; }
    if (!jacobi) {
      all_domains();
      barrier();
      for (int i = threadIdx.x; i < nt; i += T) {
        const double zi = __ldcg(d.z + g0 + i);
        lz[i] = zi;
        term(t2, d.T2, i, lr[i] * zi);
      }
      __syncthreads();
      if (!single && warp < 2 * R) {
        const int q = warp / R, r = segment(q);
        if (q == 0) {
          const Chunk c = seg_chunk(P, r, nt);
          double u = 0;
          for (int j = 0; j < c.cnt; j++) u += t2[c.l0 + j];
          u = wsum(u);
          if ((threadIdx.x & 31) == 0) P.sums[(size_t)W_RZ * NS + b * R + r] = u;
        } else {
          direction_sums(r);
        }
      }
      if constexpr (single) {
        serial(t2, nullptr);
      } else {
        barrier();
        if (warp < R)
          order(D_RZ, warp, t2, before(W_RZ, warp));
        barrier();
        walk1(D_RZ, d.T2);
      }
      rzNew = res[0];
    }
    const double beta = rzNew / rz;
    for (int i = threadIdx.x; i < nt; i += T) {
      const double pi = lz[i] + beta * lp[i];
      lp[i] = pi;
      d.p[g0 + i] = pi;
      term(t3, d.T3, i, pi * pi);
    }
    rz = rzNew;
    __syncthreads();
    if constexpr (single) {
      serial(t3, nullptr);
    } else {
      if (warp < R) order(D_PP, warp, t3, before3(W_ZZ, warp, 2 * beta, beta * beta));
      barrier();
      walk1(D_PP, d.T3);
    }
    pp = res[0];
  }
  if (!done) iters = A.maxIters;

  // ---- descent safeguard + trust region (newton.ts:152-179) ----
  // left-to-right sum of the terms in (t0, d.T0)
  auto sum0 = [&]() {
    if constexpr (single) {
      serial(t0, nullptr);
      return res[0];
    }
    __syncthreads();
    if (warp < R) {
      const Chunk c = seg_chunk(P, warp, nt);
      double u = 0;
      for (int j = 0; j < c.cnt; j++) u += t0[c.l0 + j];
      u = wsum(u);
      if ((threadIdx.x & 31) == 0) P.sums[(size_t)W_PAP * NS + b * R + warp] = u;
    }
    barrier();
    if (warp < R)
      order(D_PAP, warp, t0, before(W_PAP, warp));
    barrier();
    walk1(D_PAP, d.T0);
    return res[0];
  };
  barrier();
  for (int i = threadIdx.x; i < nt; i += T) term(t0, d.T0, i, d.g[g0 + i] * lx[i]);
  double gtdx = sum0();
  bool fallback = false;
  if (!isfinite(gtdx) || gtdx >= 0) {
    fallback = true;
    barrier();
    for (int i = threadIdx.x; i < nt; i += T) {
      const double di = -d.g[g0 + i] / d.diag[g0 + i];
      lx[i] = di;
      term(t0, d.T0, i, d.g[g0 + i] * di);
    }
    gtdx = sum0();
  }
  double mx = 0;
  for (int i = threadIdx.x; i < nt; i += T) {
    const double a = fabs(lx[i]);
    if (a > mx) mx = a;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double w = __shfl_xor_sync(0xffffffffu, mx, o);
    if (w > mx) mx = w;
  }
  if ((threadIdx.x & 31) == 0) red[warp] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < W; i++)
      if (red[i] > mx) mx = red[i];
    P.sums[(size_t)W_MAX * NS + b] = mx;
  }
  barrier();
  double maxDx = 0;
  for (int i = 0; i < P.G; i++) {
    const double w = __ldcg(P.sums + (size_t)W_MAX * NS + i);
    if (w > maxDx) maxDx = w;
  }
  const double TRUST = 0.002;
  if (maxDx > TRUST) {
    const double sc = TRUST / maxDx;
    for (int i = threadIdx.x; i < nt; i += T) d.dx[g0 + i] = lx[i] * sc;
    gtdx *= sc;
  } else if (vs) {
    for (int i = threadIdx.x; i < nt; i += T) d.dx[g0 + i] = lx[i];
  }
  if (b == 0 && threadIdx.x == 0) {
    d.scal[S_PCG_ITERS] = iters;
    d.scal[S_PCG_RES] = residual;
    d.scal[S_GTDX] = gtdx;
    d.scal[S_FALLBACK] = fallback ? 1 : 0;
    d.scal[S_MAXDX] = maxDx;
  }
}

void cluster_attr(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int cs, size_t smem) {
  cfg.gridDim = dim3(cs);
  cfg.blockDim = dim3(kPcg64T);
  cfg.dynamicSmemBytes = smem;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
}

constexpr size_t kMaxDyn = 227 * 1024 - 22 * 1024;  // beside the kernel's static shared memory

}  // namespace

// Largest cluster of the solve's CTAs (all of their shared memory) the current
// device co-schedules; 0: none. Also raises the kernels' shared-memory limit there.
int pcg64_cluster_max() {
  static std::mutex mu;
  static std::map<int, int> known;  // per device
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  const auto it = known.find(dev);
  if (it != known.end()) return it->second;
  cudaFuncSetAttribute(k_pcg64<CLUSTER>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  cudaFuncSetAttribute(k_pcg64<CLUSTER>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxDyn);
  cudaFuncSetAttribute(k_pcg64<GRID>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxDyn);
  cudaFuncSetAttribute(k_pcg64<GRID_FAR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxDyn);
  cudaFuncSetAttribute(k_pcg64<ONE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxDyn);
  int r = 0;
  for (int cs = 16; cs >= 1 && !r; cs /= 2) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cluster_attr(cfg, attr, cs, kMaxDyn);
    int nc = 0;
    if (cudaOccupancyMaxActiveClusters(&nc, k_pcg64<CLUSTER>, &cfg) == cudaSuccess && nc >= 1) r = cs;
  }
  cudaGetLastError();
  known[dev] = r;
  return r;
}

// Sheets up to kPcg64SingleN vertices run in one CTA, up to kPcg64ClusterN in one cluster,
// larger ones on the grid. The ordered sums' stages cost more than adding the terms
// one by one while there are few: us per iteration on a B200, one thread per sum on a
// cooperative grid / stages in a cluster / one CTA, Jacobi: 36 vertices 19 / 23.3 / 8.4, 81
// vertices 23 / 24.4 / 11.7, 169 vertices 31 / 26 / 18.5, 256 vertices 37 / 26 / 24.3,
// 441 vertices 48 / 28 / 47; Schwarz: 36 vertices 51 / 37 / 18, 256 vertices 111 / 46 / 49.
constexpr int kPcg64SingleN = 256;
// One vertex per thread pair of a cluster. Beyond it the FP64 arithmetic of 16 SMs
// outweighs what the cluster's barrier saves: ms of a two-step drape in a cluster / on
// the grid, Jacobi: 55 x 55 vertices 60 / 61, 64 x 64 65 / 66, 71 x 71 73 / 67, 77 x 77
// 88 / 68. (With Schwarz the grid is ahead from 2,000 vertices on: 46 x 46 64 / 62.5, 64 x 64 73 / 64.)
constexpr int kPcg64ClusterN = 4096;
// Vertices per CTA of the grid at the least: fewer CTAs mean fewer stages to walk, but
// longer ones. The same drape with 64 / 96 / 128 / 192: 71 x 71 72 / 67 / 69 / 76 ms,
// 91 x 91 89 / 79 / 78 / 83, 111 x 111 102 / 99 / 95 / 97 (Schwarz 63 / 61 / 63 / 64).
constexpr int kPcg64GridNv = 96;

void build_pcg64_plan(const HostMesh& me, int sms, int clusterMax, bool lists, Pcg64Host& out) {
  Pcg64Plan& p = out.p;
  p = Pcg64Plan{};
  p.cluster = clusterMax > 0 && me.n <= kPcg64ClusterN * clusterMax / 16 ? 1 : 0;
  if (p.cluster) {
    p.G = me.n <= kPcg64SingleN ? 1 : clusterMax;
  } else {
    p.G = std::max(1, std::min(sms, (me.n + kPcg64GridNv - 1) / kPcg64GridNv));
  }
  p.nv = (me.n + p.G - 1) / p.G;
  const int terms = 3 * p.nv;
  // fewer segments to walk against fewer terms per lane to map
  p.R = p.G <= 16 && terms > 160 ? 2 : 1;
  p.K = ((terms + p.R * 32 - 1) / (p.R * 32)) | 1;
  p.NS = p.G * p.R;
  out.slotOff.assign(1, 0);
  out.slots.clear();
  out.inc.clear();
  if (!lists) return;
  out.inc.assign(me.memRec.size(), 0);
  std::vector<int> slot(me.m, -1), used;
  int most = 0;
  for (int b = 0; b < p.G; b++) {
    const int v0 = std::min(me.n, b * p.nv), v1 = std::min(me.n, v0 + p.nv);
    used.clear();
    for (uint32_t q = me.memOff[v0]; q < me.memOff[v1]; q++) {
      const int t = (int)(me.memRec[q] >> 2);
      if (slot[t] < 0) {
        slot[t] = (int)used.size();
        used.push_back(t);
        out.slots.push_back(make_int4((int)me.idx[3 * (size_t)t], (int)me.idx[3 * (size_t)t + 1],
                                      (int)me.idx[3 * (size_t)t + 2], t));
      }
      out.inc[q] = ((uint32_t)slot[t] << 2) | (me.memRec[q] & 3u);
    }
    for (int t : used) slot[t] = -1;
    most = std::max(most, (int)used.size());
    out.slotOff.push_back((int)out.slots.size());
  }
  p.elemStride = 18 * (size_t)std::max(most, 1);
  const size_t walk = 2 * (size_t)p.NS * (sizeof(OrdStage) + sizeof(OrdStep));
  const size_t vec = 9 * (size_t)terms * 8, elem = p.elemStride * 8;
  const size_t offs = ((size_t)(p.nv + 1) * 4 + 15) & ~(size_t)15;
  p.smem = walk;
  auto fits = [&](size_t bytes) {
    if (p.smem + bytes > kMaxDyn) return 0;
    p.smem += bytes;
    return 1;
  };
  p.offSmem = fits(offs);  // up to about 6.7 million vertices
  p.vecSmem = fits(vec);
  p.elemSmem = fits(elem);
}

int launch_pcg64(const Dev& d, const Pcg64Plan& p, int maxIters, double tol, cudaStream_t s) {
  Args a{d, p, maxIters, tol};
  void* args[] = {&a};
  if (p.G == 1) return (int)cudaLaunchKernel((void*)k_pcg64<ONE>, dim3(1), dim3(kPcg64T), args, p.smem, s);
  if (p.cluster) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cluster_attr(cfg, attr, p.G, p.smem);
    cfg.stream = s;
    return (int)cudaLaunchKernelEx(&cfg, k_pcg64<CLUSTER>, a);
  }
  auto* grid = p.offSmem ? k_pcg64<GRID> : k_pcg64<GRID_FAR>;
  return (int)cudaLaunchCooperativeKernel((void*)grid, dim3(p.G), dim3(kPcg64T), args, p.smem, s);
}

}  // namespace cs
