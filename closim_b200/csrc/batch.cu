// Batched implicit step: one launch steps every sheet of a packed work list (one
// launch per size class).
//
// Each sheet is an independent scene (no coupling), so a sheet maps to one
// thread block, or one cluster of blocks (batch_class), that runs its whole
// step -- predictor and floor-CCD bisection,
// up to newtonIters Newton iterations (gradient, FP32 Jacobi-PCG with FP64 dot
// products, descent safeguard, 2 mm trust region, CCD-gated Armijo search,
// lagged-friction commit), velocity update and restitution -- with block
// or cluster barriers only: no grid-wide synchronization and no host round trip.
// The launch is persistent: groups take sheets from a work list ordered largest
// first. A sheet's PCG is a chain of short passes over its vertices, bound by the
// latency of its gathers; one SM per sheet left the batch waiting for its largest
// sheet (96 sheets of 16 to 80 vertices a side: 76 ms a step by lone blocks, 41 with
// clusters).
// The algorithm per sheet is newton.ts:27-303 with the floor-contact
// subset of contact-assembly.ts (kind 2: per-vertex barrier, lagged friction,
// floor CCD, restitution); the bending gradient is the analytic gradient of
// the hinge energy instead of its central difference (bending.ts:19-42).
// Every reduction is a fixed-order tree over the sheet's group, whose size depends
// on the sheet alone, so a sheet's result does not depend on the rest of the batch.
#include <cooperative_groups.h>

#include "adjoint_math.cuh"
#include "batch.cuh"
#include "contact_math.cuh"
#include "elem.cuh"
#include "hvp32.cuh"

namespace cs {

namespace {

namespace cg = cooperative_groups;

struct Range {
  int v0, v1, t0, t1, h0, h1;
};

constexpr int kParts = 12;  // up to three sums of four ranks

// The threads that step one sheet: a thread-block cluster (CL) or one block, which
// may reproduce the reductions of a cluster of VIRT blocks. The shape is part of the
// type: with the stride and the barriers known at compile time 148 sheets of 38
// vertices a side took 19.85 ms a step instead of 20.3.
// `first` and `stride` spread a loop over all the threads.
template <int T, bool CL, int VIRT>
struct Group {
  static_assert(VIRT == 1 || VIRT == 2 || VIRT == 4, "the shares turn by one place");
  static constexpr bool kCluster = CL;
  static constexpr int kVirt = VIRT;
  int size, rank;
  double* sm;                  // block reduction scratch (32)
  double (*part)[kParts][32];  // warp partials, two banks in turn
  double (*bank)[3][8];        // the CTAs' partials, two banks in turn
  int turn;
  __device__ __forceinline__ int first() const { return CL ? rank * T + (int)threadIdx.x : (int)threadIdx.x; }
  __device__ __forceinline__ int stride() const { return CL ? size * T : T; }
};
// Barrier over the group; what its threads wrote before is visible after.
template <class GR>
__device__ __forceinline__ void gsync(const GR& G) {
  if constexpr (GR::kCluster) cg::this_cluster().sync();
  else __syncthreads();
}
// The CTAs' values of a block reduction: each is pushed into every peer's bank,
// one cluster barrier, then all read their own bank. A bank is written again only
// after the next call's barrier, which no CTA passes before it has read.
template <class GR, class F>
__device__ __forceinline__ double gcombine(GR& G, double v, const F& op) {
  if constexpr (!GR::kCluster) return v;
  cg::cluster_group cl = cg::this_cluster();
  double* mine = G.bank[G.turn & 1][0];
  if ((int)threadIdx.x < G.size) cl.map_shared_rank(mine, threadIdx.x)[G.rank] = v;
  cl.sync();
  double r = mine[0];
  for (int q = 1; q < G.size; q++) r = op(r, mine[q]);
  G.turn++;
  return r;
}
// A thread's part of the sums of gsums: v[r][k] belongs to rank r of the cluster
// that a lone block stands in for (a rank of a real one has only its own, v[0]).
template <int K, int VIRT>
struct Shares {
  double v[VIRT][K];
};
// f(i, s) adds item i's terms to s for the thread's items of [i0, i1). Rank r of a
// cluster takes the items first + (r + j * VIRT) * stride, so a lone block that
// stands in for it walks all items in memory order and gives each in turn to the
// next rank's share: unrolled by VIRT in the short passes of the PCG (UNROLL), by
// turning the shares one place an item in the long ones, whose code would outgrow
// the instruction cache. 512 sheets of 16 to 128 vertices a side, ms a step on a B200
// (before the vector passes loaded four dofs together): 387 with a pass per rank, 386
// turning everywhere, 387 unrolled everywhere, 384 this way; 381 with one share.
template <bool UNROLL = false, int K, class GR, class F>
__device__ __forceinline__ void geach(const GR& G, Shares<K, GR::kVirt>& S, int i0, int i1, const F& f) {
  constexpr int V = GR::kVirt;
  if constexpr (UNROLL && V > 1) {
    for (int i = i0 + G.first(); i < i1; i += V * G.stride()) {
#pragma unroll
      for (int r = 0; r < V; r++)
        if (r == 0 || i + r * G.stride() < i1) f(i + r * G.stride(), S.v[r]);
    }
    return;
  }
  auto turn = [&]() {
#pragma unroll
    for (int k = 0; k < K; k++) {
      const double t = S.v[0][k];
#pragma unroll
      for (int r = 1; r < V; r++) S.v[r - 1][k] = S.v[r][k];
      S.v[V - 1][k] = t;
    }
  };
  int place = 0;
  for (int i = i0 + G.first(); i < i1; i += G.stride()) {
    f(i, S.v[0]);
    if constexpr (V > 1) {
      turn();
      place++;
    }
  }
  if constexpr (V > 1)
    for (; place & (V - 1); place++) turn();
}
// Sums over the group of the terms that `share(S)` leaves in S (by geach), with one
// block barrier (and one cluster barrier): warp trees, every warp (of a cluster:
// warp 0) adds the warps' partials with the same tree, and the CTAs' totals are
// added in rank order. A lone block that stands in for a cluster (virt > 1) does so
// with each rank's shares, so it gets the cluster's bits. Also a barrier for
// what the group's threads wrote before.
template <int K, class GR, class F>
__device__ __forceinline__ void gsums(double (&out)[K], GR& G, const F& share) {
  constexpr int V = GR::kVirt;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int turn = G.turn & 1;
  Shares<K, V> S;
#pragma unroll
  for (int r = 0; r < V; r++)
#pragma unroll
    for (int k = 0; k < K; k++) S.v[r][k] = 0;
  share(S);
#pragma unroll
  for (int r = 0; r < V; r++)
#pragma unroll
    for (int k = 0; k < K; k++) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) S.v[r][k] += __shfl_down_sync(0xffffffffu, S.v[r][k], o);
      if (lane == 0) G.part[turn][r * K + k][warp] = S.v[r][k];
    }
  G.turn++;
  __syncthreads();
  if constexpr (!GR::kCluster) {
#pragma unroll
    for (int k = 0; k < K; k++) {
      double w[V];
#pragma unroll
      for (int r = 0; r < V; r++) w[r] = lane < nw ? G.part[turn][r * K + k][lane] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < V; r++) w[r] += __shfl_down_sync(0xffffffffu, w[r], o);
      double t = w[0];
#pragma unroll
      for (int r = 1; r < V; r++) t += w[r];
      out[k] = __shfl_sync(0xffffffffu, t, 0);
    }
    return;
  }
  cg::cluster_group cl = cg::this_cluster();
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < K; k++) {
      double w = lane < nw ? G.part[turn][k][lane] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) w += __shfl_down_sync(0xffffffffu, w, o);
      w = __shfl_sync(0xffffffffu, w, 0);
      if (lane < G.size) cl.map_shared_rank(G.bank[turn][k], lane)[G.rank] = w;
    }
  }
  cl.sync();
#pragma unroll
  for (int k = 0; k < K; k++) {
    double r = G.bank[turn][k][0];
    for (int q = 1; q < G.size; q++) r += G.bank[turn][k][q];
    out[k] = r;
  }
}

template <class GR>
__device__ __forceinline__ double gmax(double v, GR& G) {
  return gcombine(G, block_max(v, G.sm), [](double a, double b) { return js_max(a, b); });
}
template <class GR>
__device__ __forceinline__ double gmin(double v, GR& G) {
  return gcombine(G, block_min(v, G.sm), [](double a, double b) { return fmin(a, b); });
}

__device__ __forceinline__ void ld3b(const double* x, int v, double o[3]) {
  o[0] = x[v * 3]; o[1] = x[v * 3 + 1]; o[2] = x[v * 3 + 2];
}

template <class GR>
__device__ __forceinline__ void enforce_pins(const BatchDev& b, const Range& R, const GR& G, double* x) {
  for (int v = R.v0 + G.first(); v < R.v1; v += G.stride())
    if (b.pinned[v])
      for (int k = 0; k < 3; k++) x[v * 3 + k] = b.pinPos[v * 3 + k];
}

// checkTrial restricted to the floor (contact-assembly.ts:489-553): the
// smallest floor distance must exceed dMin and no vertex may cross the dMin
// level during x0 -> xT.
template <class GR>
__device__ bool floor_trial_ok(const BatchDev& b, const Range& R, const double* xT, GR& G) {
  if (!b.hasFloor) return true;
  double mn = INFINITY;
  int bad = 0;
  for (int v = R.v0 + G.first(); v < R.v1; v += G.stride()) {
    const double yT = xT[v * 3 + 1] - b.floorY;
    if (yT < mn || yT != yT) mn = yT != yT ? -INFINITY : yT;
    const double y0 = b.x0[v * 3 + 1] - b.floorY;
    if (y0 - fabs(yT - y0) > b.dMin) continue;
    if (y0 > b.dMin && yT <= b.dMin && y0 > yT) {
      const double toi = (y0 - b.dMin) / (y0 - yT);
      if (toi < 1 - 1e-9) bad = 1;
    }
  }
  const double m = gmin(mn, G);
  const double anyBad = gmax((double)bad, G);
  return !(m <= b.dMin) && anyBad == 0;
}

template <class GR>
__device__ __forceinline__ void update_active(const BatchDev& b, const Range& R, const GR& G, const double* x) {
  for (int v = R.v0 + G.first(); v < R.v1; v += G.stride())
    b.act[v] = b.hasFloor && (x[v * 3 + 1] - b.floorY < b.dHat) ? 1 : 0;
}

// totalEnergy (newton.ts:76-88): inertia + membrane + bending + barrier merit.
template <class GR>
__device__ double sheet_energy(const BatchDev& b, const Range& R, const double* x, const Mat<double>& mt, double kb,
                               GR& G) {
  double out[1];
  gsums<1>(out, G, [&](Shares<1, GR::kVirt>& S) {
    geach(G, S, R.v0, R.v1, [&](int v, double (&s)[1]) {
      double e = s[0];
      const double M = b.mass[v];
      for (int k = 0; k < 3; k++) {
        const double d = x[v * 3 + k] - b.yHat[v * 3 + k];
        e += 0.5 * M * d * d * b.invH2;
      }
      if (b.act[v]) {
        const double d = fmax(x[v * 3 + 1] - b.floorY, 1e-12);
        if (d < b.dHat) e += b.kappa * barrier_value(d, b.dHat);
      }
      s[0] = e;
    });
    geach(G, S, R.t0, R.t1, [&](int t, double (&s)[1]) {
      double p0[3], p1[3], p2[3];
      ld3b(x, b.idx[t * 3], p0); ld3b(x, b.idx[t * 3 + 1], p1); ld3b(x, b.idx[t * 3 + 2], p2);
      const float4 iv = b.inv[t];
      s[0] += tri_energy<double>(p0, p1, p2, iv.x, iv.y, iv.z, iv.w, b.area[t], mt);
    });
    if (kb > 0)
      geach(G, S, R.h0, R.h1, [&](int hh, double (&s)[1]) {
        const int4 hv = b.hinge[hh];
        double q[12], gdum[12];
        ld3b(x, hv.x, q); ld3b(x, hv.y, q + 3); ld3b(x, hv.z, q + 6); ld3b(x, hv.w, q + 9);
        s[0] += bend_grad<double>(q, b.hmeta[hh * 3], b.hmeta[hh * 3 + 1], b.hmeta[hh * 3 + 2], kb, gdum);
      });
  });
  return out[0];
}

// Newton gradient at b.x into b.g (filtered), the barrier curvature added to
// the diagonal estimate; returns |g|.
template <class GR>
__device__ double sheet_gradient(const BatchDev& b, const Range& R, const Mat<double>& mt, double kb, GR& G) {
  for (int t = R.t0 + G.first(); t < R.t1; t += G.stride()) {
    double p0[3], p1[3], p2[3];
    ld3b(b.x, b.idx[t * 3], p0); ld3b(b.x, b.idx[t * 3 + 1], p1); ld3b(b.x, b.idx[t * 3 + 2], p2);
    const float4 iv = b.inv[t];
    double en, gg[9], E[3];
    tri_grad<double>(p0, p1, p2, iv.x, iv.y, iv.z, iv.w, b.area[t], mt, en, gg, E);
    for (int k = 0; k < 9; k++) b.elem[(size_t)t * 9 + k] = gg[k];
  }
  if (kb > 0)
    for (int hh = R.h0 + G.first(); hh < R.h1; hh += G.stride()) {
      const int4 hv = b.hinge[hh];
      double q[12], gg[12];
      ld3b(b.x, hv.x, q); ld3b(b.x, hv.y, q + 3); ld3b(b.x, hv.z, q + 6); ld3b(b.x, hv.w, q + 9);
      bend_grad<double>(q, b.hmeta[hh * 3], b.hmeta[hh * 3 + 1], b.hmeta[hh * 3 + 2], kb, gg);
      for (int k = 0; k < 12; k++) b.helem[(size_t)hh * 12 + k] = gg[k];
    }
  gsync(G);
  double out[1];
  gsums<1>(out, G, [&](Shares<1, GR::kVirt>& S) {
    geach(G, S, R.v0, R.v1, [&](int v, double (&sum)[1]) {
      double s[3] = {0, 0, 0};
      for (uint32_t q = b.memOff[v]; q < b.memOff[v + 1]; q++) {
        const uint32_t rec = b.memRec[q];
        const double* e = b.elem + (size_t)(rec >> 2) * 9 + (rec & 3) * 3;
        s[0] += e[0]; s[1] += e[1]; s[2] += e[2];
      }
      if (kb > 0)
        for (uint32_t q = b.hinOff[v]; q < b.hinOff[v + 1]; q++) {
          const uint32_t rec = b.hinRec[q];
          const double* e = b.helem + (size_t)(rec >> 2) * 12 + (rec & 3) * 3;
          s[0] += e[0]; s[1] += e[1]; s[2] += e[2];
        }
      if (b.act[v]) {
        // barrier (addDistGrad) and lagged friction (addFrictionForce) of the floor contact
        const double d = fmax(b.x[v * 3 + 1] - b.floorY, 1e-12);
        if (d < b.dHat) {
          s[1] += barrier_grad_scalar(d, b.dHat, b.kappa, 1);
          const double lam = b.lagOk[v] ? b.lagLam[v] : barrier_normal_force(d, b.dHat, b.kappa, 1);
          double u[3], fr[3];
          for (int k = 0; k < 3; k++) u[k] = b.x[v * 3 + k] - b.x0[v * 3 + k];
          coulomb_force(u, 0.0, 1.0, 0.0, lam, b.mu, b.eps, fr);
          for (int k = 0; k < 3; k++) s[k] -= fr[k];
          b.diag[v * 3 + 1] += barrier_curvature(d, b.dHat, b.kappa);  // addDiagEstimate (accumulates)
        }
      }
      const double M = b.mass[v];
      const bool pin = b.pinned[v];
      for (int k = 0; k < 3; k++) {
        const int i = v * 3 + k;
        double gi = M * (b.x[i] - b.yHat[i]) * b.invH2 + s[k];
        if (pin) gi = 0;
        b.g[i] = gi;
        sum[0] += gi * gi;
      }
    });
  });
  return sqrt(out[0]);
}

// FP32 state of every triangle for the matrix-free HVP (F, S, Dm^-1, s).
template <class GR>
__device__ void sheet_tristate(const BatchDev& b, const Range& R, const GR& G, const Mat<double>& m) {
  for (int t = R.t0 + G.first(); t < R.t1; t += G.stride()) {
    double x0[3], x1[3], x2[3];
    ld3b(b.x, b.idx[t * 3], x0); ld3b(b.x, b.idx[t * 3 + 1], x1); ld3b(b.x, b.idx[t * 3 + 2], x2);
    const float4 iv = b.inv[t];
    double F0[3], F1[3];
    for (int k = 0; k < 3; k++) {
      const double e1 = x1[k] - x0[k], e2 = x2[k] - x0[k];
      F0[k] = iv.x * e1 + iv.z * e2;
      F1[k] = iv.y * e1 + iv.w * e2;
    }
    const double E00 = 0.5 * (F0[0] * F0[0] + F0[1] * F0[1] + F0[2] * F0[2] - 1);
    const double E11 = 0.5 * (F1[0] * F1[0] + F1[1] * F1[1] + F1[2] * F1[2] - 1);
    const double E01 = 0.5 * (F0[0] * F1[0] + F0[1] * F1[1] + F0[2] * F1[2]);
    float* o = b.tris + (size_t)t * 16;
    for (int k = 0; k < 3; k++) { o[k] = (float)F0[k]; o[3 + k] = (float)F1[k]; }
    o[6] = (float)(m.C00 * E00 + m.C01 * E11);
    o[7] = (float)(m.C11 * E11 + m.C01 * E00);
    o[8] = (float)(2 * m.G * E01);
    o[9] = iv.x; o[10] = iv.y; o[11] = iv.z; o[12] = iv.w;
    o[13] = (float)(m.thickness * (double)b.area[t]);
    o[14] = 0.f; o[15] = 0.f;
  }
}

// Ap = (M/h^2 + H_membrane + H_floor) p in FP32; returns p.Ap (FP64). Each
// vertex adds the corner share of its incident triangles' HVP directly
// (recomputed per corner from the stored FP32 state), so no per-triangle
// result is written and read back and no barrier splits the product.
template <class GR>
__device__ double sheet_hvp(const BatchDev& b, const Range& R, float C00, float C11, float C01, float Gs,
                            GR& G) {
  const float invH2 = (float)b.invH2;
  double out[1];
  gsums<1>(out, G, [&](Shares<1, GR::kVirt>& S) {
    geach<true>(G, S, R.v0, R.v1, [&](int v, double (&s)[1]) {
      float sp[3] = {0.f, 0.f, 0.f};
      for (uint32_t q = b.memOff[v]; q < b.memOff[v + 1]; q++) {
        const uint32_t rec = __ldg(b.memRec + q);
        const uint32_t t = rec >> 2;
        const int i0 = (int)__ldg(b.idx + t * 3), i1 = (int)__ldg(b.idx + t * 3 + 1);
        const int i2 = (int)__ldg(b.idx + t * 3 + 2);
        const float3 p0 = make_float3(b.p[i0 * 3], b.p[i0 * 3 + 1], b.p[i0 * 3 + 2]);
        const float3 p1 = make_float3(b.p[i1 * 3], b.p[i1 * 3 + 1], b.p[i1 * 3 + 2]);
        const float3 p2 = make_float3(b.p[i2 * 3], b.p[i2 * 3 + 1], b.p[i2 * 3 + 2]);
        float o[3];
        // plain loads: another CTA of the group may have written the record
        tri_hvp_corner<false>(b.tris + (size_t)t * 16, p0, p1, p2, (int)(rec & 3), C00, C11, C01, Gs, o);
        sp[0] += o[0]; sp[1] += o[1]; sp[2] += o[2];
      }
      float cy = 0.f;
      if (b.act[v]) {
        const double d = fmax(b.x[v * 3 + 1] - b.floorY, 1e-12);
        if (d < b.dHat) cy = (float)(barrier_curvature(d, b.dHat, b.kappa) * (double)b.p[v * 3 + 1]);
      }
      const float M = b.mass[v];
      const bool pin = b.pinned[v];
      for (int q = 0; q < 3; q++) {
        const int i = v * 3 + q;
        float ap = M * b.p[i] * invH2 + sp[q] + (q == 1 ? cy : 0.f);
        if (pin) ap = 0.f;
        b.Ap[i] = ap;
        s[0] += (double)b.p[i] * ap;
      }
    });
  });
  return out[0];
}

// pcg.ts:11-95 (Jacobi, tolerance 1e-3) and the newton.ts:152-179 epilogue;
// the direction lands in b.dx. Returns the PCG iteration count.
template <class GR>
__device__ int sheet_pcg(const BatchDev& b, const Range& R, float C00, float C11, float C01, float Gs, GR& G,
                         double& gtdxOut) {
  double s3[3];
  gsums<3>(s3, G, [&](Shares<3, GR::kVirt>& S) {
    geach<true>(G, S, 3 * R.v0, 3 * R.v1, [&](int i, double (&s)[3]) {
      const double bi = -b.g[i];
      s[0] += bi * bi;
      const bool pin = b.pinned[i / 3];
      const float ri = pin ? 0.f : (float)bi;
      b.r[i] = ri;
      b.xs[i] = 0.f;
      s[1] += (double)ri * ri;
      const float di = pin ? 0.f : b.diag[i] > 1e-12 ? (float)(1.0 / b.diag[i]) : 1.f;
      b.dinv[i] = di;
      const float zi = ri * di;
      b.z[i] = zi;
      b.p[i] = zi;
      s[2] += (double)ri * zi;
    });
  });
  const double bNorm = sqrt(s3[0]);
  double residual = sqrt(s3[1]), rz = s3[2];
  const double absTol = fmax(1e-3 * fmax(bNorm, 1e-12), 1e-12);
  int iters = 0;
  bool done = residual < absTol;
  int k = 0;
  for (; !done && k < b.pcgMaxIters; k++) {
    const double pAp = sheet_hvp(b, R, C00, C11, C01, Gs, G);
    if (!(pAp > 1e-30)) { iters = k; done = true; break; }
    const float alpha = (float)(rz / pAp);
    double s2[2];
    gsums<2>(s2, G, [&](Shares<2, GR::kVirt>& S) {
      // Four dofs' loads in flight together, item u where geach would put it: the pass
      // is bound by their latency (512 sheets of 16 to 128 a side 384 -> 301 ms a step).
      constexpr int U = 4;
      const int i1 = 3 * R.v1, st = G.stride();
      for (int i = 3 * R.v0 + G.first(); i < i1; i += U * st) {
        float x[U], p[U], r[U], a[U], di[U];
        bool pin[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int k = i + u * st < i1 ? i + u * st : i;
          x[u] = b.xs[k]; p[u] = b.p[k]; r[u] = b.r[k]; a[u] = b.Ap[k]; di[u] = b.dinv[k];
          pin[u] = b.pinned[k / 3];
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int k = i + u * st;
          if (k < i1) {
            float xi = x[u] + alpha * p[u];
            float ri = r[u] - alpha * a[u];
            if (pin[u]) { xi = 0.f; ri = 0.f; }
            b.xs[k] = xi;
            b.r[k] = ri;
            double(&s)[2] = S.v[u % GR::kVirt];
            s[0] += (double)ri * ri;
            const float zi = ri * di[u];
            b.z[k] = zi;
            s[1] += (double)ri * zi;
          }
        }
      }
    });
    residual = sqrt(s2[0]);
    const double rzn = s2[1];
    if (residual < absTol) { iters = k + 1; done = true; break; }
    const float beta = (float)(rzn / rz);
    rz = rzn;
    for (int i = 3 * R.v0 + G.first(), st = G.stride(), i1 = 3 * R.v1; i < i1; i += 4 * st) {
      float z[4], p[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int k = i + u * st < i1 ? i + u * st : i;
        z[u] = b.z[k];
        p[u] = b.p[k];
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (i + u * st < i1) b.p[i + u * st] = z[u] + beta * p[u];
    }
    gsync(G);
  }
  if (!done) iters = b.pcgMaxIters;
  double s1[1];
  gsums<1>(s1, G, [&](Shares<1, GR::kVirt>& S) {
    geach<true>(G, S, 3 * R.v0, 3 * R.v1, [&](int i, double (&s)[1]) {
      const double di = b.xs[i];
      b.dx[i] = di;
      s[0] += b.g[i] * di;
    });
  });
  double gtdx = s1[0];
  if (!isfinite(gtdx) || gtdx >= 0) {
    gsums<1>(s1, G, [&](Shares<1, GR::kVirt>& S) {
      geach<true>(G, S, 3 * R.v0, 3 * R.v1, [&](int i, double (&s)[1]) {
        const double di = -b.g[i] / b.diag[i];
        b.dx[i] = di;
        s[0] += b.g[i] * di;
      });
    });
    gtdx = s1[0];
  }
  double mx = 0;
  for (int i = 3 * R.v0 + G.first(); i < 3 * R.v1; i += G.stride()) mx = fmax(mx, fabs(b.dx[i]));
  const double maxDx = gmax(mx, G);
  if (maxDx > 0.002) {
    const double sc = 0.002 / maxDx;
    for (int i = 3 * R.v0 + G.first(); i < 3 * R.v1; i += G.stride()) b.dx[i] *= sc;
    gtdx *= sc;
    gsync(G);
  }
  gtdxOut = gtdx;
  return iters;
}

template <class GR>
__device__ void step_sheet(const BatchDev& b, int s, GR& G) {
  const Range R{b.vStart[s], b.vStart[s + 1], b.tStart[s], b.tStart[s + 1], b.hStart[s], b.hStart[s + 1]};
  const double* mr = b.mat + (size_t)s * BM_N;
  const Mat<double> mt{mr[BM_C00], mr[BM_C11], mr[BM_C01], mr[BM_G], mr[BM_THICK]};
  const double kb = mr[BM_KB], damp = mr[BM_DAMP], beta = mr[BM_BETA];
  const float C00 = (float)mr[BM_C00], C11 = (float)mr[BM_C11], C01 = (float)mr[BM_C01], Gs = (float)mr[BM_G];
  const double h = b.h;
  // predictor y_hat = x + h v + h^2 g, initial guess y_hat with pins (newton.ts:40-51)
  for (int v = R.v0 + G.first(); v < R.v1; v += G.stride())
    for (int k = 0; k < 3; k++) {
      const int i = v * 3 + k;
      const double xv = b.x[i];
      b.x0[i] = xv;
      const double y = xv + h * b.v[i] + h * h * b.gravity[k];
      b.yHat[i] = y;
      b.x[i] = y;
    }
  gsync(G);
  enforce_pins(b, R, G, b.x);
  gsync(G);
  int rejected = 0;
  if (b.hasFloor && !floor_trial_ok(b, R, b.x, G)) {
    // bisect back along x0 -> y_hat to the largest CCD-valid fraction (newton.ts:53-72)
    double lo = 0, hi = 1;
    for (int it = 0; it < 8; it++) {
      const double mid = 0.5 * (lo + hi);
      for (int i = 3 * R.v0 + G.first(); i < 3 * R.v1; i += G.stride()) b.xt[i] = b.x0[i] + mid * (b.x[i] - b.x0[i]);
      gsync(G);
      enforce_pins(b, R, G, b.xt);
      gsync(G);
      if (floor_trial_ok(b, R, b.xt, G)) lo = mid;
      else hi = mid;
      if (hi - lo < 1e-4) break;
    }
    for (int i = 3 * R.v0 + G.first(); i < 3 * R.v1; i += G.stride()) b.x[i] = b.x0[i] + lo * (b.x[i] - b.x0[i]);
    gsync(G);
    enforce_pins(b, R, G, b.x);
    gsync(G);
  }
  update_active(b, R, G, b.x);
  gsync(G);
  double energy = sheet_energy(b, R, b.x, mt, kb, G);
  for (int v = R.v0 + G.first(); v < R.v1; v += G.stride()) {
    const double d0 = b.mass[v] * b.invH2 + beta;
    b.diag[v * 3] = d0; b.diag[v * 3 + 1] = d0; b.diag[v * 3 + 2] = d0;
  }
  gsync(G);
  double gradNorm = INFINITY;
  int used = 0, pcgTotal = 0, trials = 0, converged = 0;
  for (int ni = 0; ni < b.newtonIters; ni++) {
    used = ni + 1;
    update_active(b, R, G, b.x);
    gsync(G);
    gradNorm = sheet_gradient(b, R, mt, kb, G);
    if (!isfinite(gradNorm)) { converged = -1; break; }
    if (gradNorm < b.gradTol) { converged = 1; break; }
    sheet_tristate(b, R, G, mt);
    gsync(G);
    double gtdx;
    pcgTotal += sheet_pcg(b, R, C00, C11, C01, Gs, G, gtdx);
    double alpha = 1;
    bool accepted = false;
    for (int li = 0; li < b.lsIters; li++) {
      trials++;
      for (int i = 3 * R.v0 + G.first(); i < 3 * R.v1; i += G.stride()) b.xt[i] = b.x[i] + alpha * b.dx[i];
      gsync(G);
      enforce_pins(b, R, G, b.xt);
      gsync(G);
      if (!floor_trial_ok(b, R, b.xt, G)) { rejected++; alpha *= 0.5; continue; }
      const double eNew = sheet_energy(b, R, b.xt, mt, kb, G);
      if (!isfinite(eNew)) { rejected++; alpha *= 0.5; continue; }
      if (eNew <= energy + 1e-4 * alpha * gtdx) {
        for (int i = 3 * R.v0 + G.first(); i < 3 * R.v1; i += G.stride()) b.x[i] = b.xt[i];
        energy = eNew;
        accepted = true;
        gsync(G);
        // commit: lagged normal force of every active floor contact (contact-assembly.ts:475-485)
        for (int v = R.v0 + G.first(); v < R.v1; v += G.stride())
          if (b.act[v]) {
            const double d = fmax(b.x[v * 3 + 1] - b.floorY, 1e-12);
            if (d < b.dHat) { b.lagLam[v] = barrier_normal_force(d, b.dHat, b.kappa, 1); b.lagOk[v] = 1; }
          }
        gsync(G);
        break;
      }
      rejected++;
      alpha *= 0.5;
    }
    if (!accepted || alpha < 1e-6) break;
  }
  // velocity update, restitution-0 on floor contacts (newton.ts:222-245)
  for (int i = 3 * R.v0 + G.first(); i < 3 * R.v1; i += G.stride()) b.v[i] = ((b.x[i] - b.x0[i]) / h) * damp;
  gsync(G);
  update_active(b, R, G, b.x);
  gsync(G);
  double nf[1];
  gsums<1>(nf, G, [&](Shares<1, GR::kVirt>& S) {
    geach(G, S, R.v0, R.v1, [&](int v, double (&s)[1]) {
      if (!b.act[v]) return;
      s[0] += 1;
      if (b.v[v * 3 + 1] < 0) b.v[v * 3 + 1] = 0;
    });
  });
  enforce_pins(b, R, G, b.x);
  if (G.rank == 0 && threadIdx.x == 0) {
    double* o = b.out + (size_t)s * BO_N;
    o[BO_NEWTON] = used;
    o[BO_PCG] = pcgTotal;
    o[BO_GRADNORM] = gradNorm;
    o[BO_ENERGY] = energy;
    o[BO_CONVERGED] = converged;
    o[BO_TRIALS] = trials;
    o[BO_FLOOR] = nf[0];
    o[BO_REJECTED] = rejected;
  }
  gsync(G);
}

// 512 threads an SM at the least: 128 registers a thread.
template <int T, bool CL, int VIRT>
__global__ void __launch_bounds__(T, 512 / T) k_batch_step(BatchDev b, const int* order, int count, unsigned int* work,
                                                     int size) {
  __shared__ double sm[32];
  __shared__ double part[2][kParts][32];
  __shared__ double bank[2][3][8];
  __shared__ int sheetSh;
  const int rank = CL ? (int)cg::this_cluster().block_rank() : 0;
  Group<T, CL, VIRT> G{size, rank, sm, part, bank, 0};
  // Shared memory of a peer may be touched once every CTA of the cluster has
  // started, which co-scheduling alone does not promise.
  gsync(G);
  for (int guard = 0; guard <= count; guard++) {
    if (rank == 0 && threadIdx.x == 0) {
      const unsigned k = atomicAdd(work, 1u);
      const int sheet = k < (unsigned)count ? order[k] : -1;
      sheetSh = sheet;
      if constexpr (CL)
        for (int q = 1; q < size; q++) *cg::this_cluster().map_shared_rank(&sheetSh, q) = sheet;
    }
    gsync(G);
    const int sheet = sheetSh;
    gsync(G);
    if (sheet < 0) return;
    step_sheet(b, sheet, G);
  }
}

void launch_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int threads, int size, int ctas) {
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(threads);
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = size;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = size > 1 ? 1 : 0;
}

template <int T>
int launch_t(const BatchDev& b, const int* order, int count, unsigned int* work, int size, int virt, int ctas,
             cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  launch_config(cfg, attr, T, size, ctas);
  cfg.stream = s;
  auto* kernel = size > 1    ? k_batch_step<T, true, 1>
                 : virt == 4 ? k_batch_step<T, false, 4>
                 : virt == 2 ? k_batch_step<T, false, 2>
                             : k_batch_step<T, false, 1>;
  return (int)cudaLaunchKernelEx(&cfg, kernel, b, order, count, work, size);
}

}  // namespace

int batch_max_ctas(int threads) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaError_t e = cudaSuccess;
  if (threads == 128) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_batch_step<128, false, 1>, 128, 0);
  else if (threads == 256) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_batch_step<256, false, 1>, 256, 0);
  else e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_batch_step<512, false, 1>, 512, 0);
  if (e != cudaSuccess || per < 1) per = 1;
  return per * sms;
}

void batch_device(int& sms, int (&maxGroups)[kBatchClasses]) {
  int dev = 0;
  cudaGetDevice(&dev);
  sms = 1;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  for (int c = 0; c < kBatchClasses; c++) {
    maxGroups[c] = sms;
    if (kBatchSize[c] == 1) continue;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    launch_config(cfg, attr, 512, kBatchSize[c], sms / kBatchSize[c] * kBatchSize[c]);
    if (cudaOccupancyMaxActiveClusters(&maxGroups[c], k_batch_step<512, true, 1>, &cfg) != cudaSuccess)
      maxGroups[c] = 0;
  }
  cudaGetLastError();
}

int batch_launch_step(const BatchDev& b, const int* order, int count, unsigned int* work, int size, int virt,
                      int threads, int ctas, cudaStream_t s) {
  if (threads == 128) return launch_t<128>(b, order, count, work, size, virt, ctas, s);
  if (threads == 256) return launch_t<256>(b, order, count, work, size, virt, ctas, s);
  return launch_t<512>(b, order, count, work, size, virt, ctas, s);
}

}  // namespace cs
