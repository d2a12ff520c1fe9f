// The FP64 Schwarz preconditioner applied by one warp per domain, shared by the
// FP64 path's PCG (pcg64.cu) and the exact-Newton / adjoint PCG (adjoint.cu).
#pragma once
#include "div_rn.cuh"
#include "plain.cuh"

namespace cs {

// z = M^-1 r on one Schwarz domain (schwarz.ts:154-309, mas.ts:110-145; dcoarse: the
// two-level term) by one warp, lane = local dof, with the reference's operation order per dof. The
// forward substitution subtracts L[i][j] y_j as each y_j becomes known; the
// backward one needs the products in ascending j, so lane i restarts its chain
// at its turn. One thread per domain held a chain of 600 dependent operations
// with divisions and strided loads; this is 2 x 24 steps, about 13,000 cycles a
// domain with 16 warps on the SM.
struct DomLane {
  int gi;     // this lane's dof (-1: none)
  int dv;     // vertices of the domain
  bool pin, factored;
};
__device__ __forceinline__ DomLane domain_lane(const Dev& d, int dom) {
  const int lane = threadIdx.x & 31;
  const int start = __ldg(d.domStart + dom);
  DomLane f;
  f.dv = __ldg(d.domStart + dom + 1) - start;
  f.gi = lane < 3 * f.dv ? __ldg(d.domVerts + start + lane / 3) * 3 + lane % 3 : -1;
  f.pin = f.gi >= 0 && d.pinned[f.gi / 3];
  f.factored = d.domFlag[dom] != 0;
  return f;
}
// The same two substitutions with plain divisions, for the rare domain that
// holds a number outside div_rn_fast's range.
static __device__ __noinline__ double domain_solve_plain(const double* L, double rhs, int dw) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int row = min(lane, dw - 1);
  double s = rhs, y = 0, sol = 0;
  for (int j = 0; j < dw; j++) {
    const double yj = __shfl_sync(full, s / L[row * 24 + row], j);
    if (lane == j) y = yj;
    if (lane > j) s -= L[row * 24 + j] * yj;
  }
  for (int i = dw - 1; i >= 0; i--) {
    double acc = y;
    for (int j = i + 1; j < dw; j++) acc -= L[j * 24 + row] * __shfl_sync(full, sol, j);
    const double si = __shfl_sync(full, acc / L[row * 24 + row], i);
    if (lane == i) sol = si;
  }
  return sol;
}
static __device__ __noinline__ double domain_solve(const double* L, const double* r, double* z, const double* dcoarse,
                                          const DomLane& f) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int dv = f.dv, dw = dv * 3, gi = f.gi;
  const double rhs = gi >= 0 ? __ldcg(r + gi) : 0.0;
  double sol = 0;
  if (f.factored) {
    // column `lane` of the symmetric tile: L[lane][j] above it, L[j][lane] below
    double a[24];
#pragma unroll
    for (int j = 0; j < 24; j++) a[j] = lane < dw && j < dw ? __ldg(L + j * 24 + lane) : 0.0;
    const double diag = lane < dw ? __ldg(L + lane * 24 + lane) : 1.0;
    const double inv = 1.0 / diag;
    bool ok = div_rn_divisor(diag);
    double s = lane < dw ? rhs : 1.0, y = 1.0;
#pragma unroll
    for (int j = 0; j < 24; j++)
      if (j < dw) {
        const double t = div_rn_fast(s, diag, inv);
        ok = ok && (lane != j || div_rn_dividend(s));
        const double yj = __shfl_sync(full, t, j);
        if (lane == j) y = yj;
        if (lane > j) s -= a[j] * yj;
      }
#pragma unroll
    for (int i = 23; i >= 0; i--)
      if (i < dw) {
        double acc = y;
#pragma unroll
        for (int j = i + 1; j < 24; j++) acc -= a[j];  // products; zero past the domain
        const double t = div_rn_fast(acc, diag, inv);
        ok = ok && (lane != i || div_rn_dividend(acc));
        const double si = __shfl_sync(full, t, i);
        if (lane == i) sol = si;
        a[i] = a[i] * si;
      }
    if (!__all_sync(full, ok)) sol = domain_solve_plain(L, rhs, dw);
  } else {
    for (int j = 0; j < dw; j++) {
      const double rj = __shfl_sync(full, rhs, j);
      if (lane < dw) sol += L[lane * 24 + j] * rj;
    }
  }
  double zz = 0.0 + sol;
  if (dcoarse) {
    const double sc = 1 / sqrt((double)dv);
    const int k = lane % 3;
    double rc = 0;
    for (int l = 0; l < dv; l++) rc += __shfl_sync(full, rhs, l * 3 + k) * sc;
    if (lane < dw) {
      const double dd = dcoarse[k];
      const double cz = dd > 1e-12 ? (0.5 * rc) / dd : 0.0;
      zz += cz * sc;
    }
  }
  zz = f.pin || lane >= dw ? 0.0 : zz;
  if (lane < dw) z[gi] = zz;
  // r.z of the domain, its dofs left to right
  const double t = rhs * zz;
  double rz = 0;
#pragma unroll 8
  for (int i = 0; i < 24; i++) rz += __shfl_sync(full, t, i);
  return rz;
}

}  // namespace cs
