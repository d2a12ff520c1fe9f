// FP64 path of the implicit-Euler Newton step (compiled with -fmad=false).
//
// One thread per element over SoA mesh constants writes element-local results;
// one thread per vertex gathers them through the element-ordered CSR
// incidence, so each vertex sum adds the same terms in the same order as the
// reference's scatter (src/mesh/incidence.ts:1-7). Sums the reference
// accumulates in a loop are ordered sums (ordered_sum.cuh). The PCG solve is
// pcg64.cu's.
#include <cstdio>

#include "adjoint_math.cuh"
#include "contact.cuh"
#include <algorithm>

#include "ordered_sum.cuh"
#include "plain.cuh"

namespace cs {

static inline int nblk(int n) { return (n + kThreads - 1) / kThreads; }

__device__ __forceinline__ void load3(const double* x, int v, double o[3]) {
  o[0] = x[v * 3]; o[1] = x[v * 3 + 1]; o[2] = x[v * 3 + 2];
}

// Block size of the kernels that evaluate one ordered sum (ordered_sum.cuh).
constexpr int kOrdThreads = 1024;
#define ORD_LAUNCH(kernel, n, grid, stream, ...)                                  \
  do {                                                                            \
    if ((n) <= kOrdThreads) kernel<true><<<grid, kOrdThreads, 0, stream>>>(__VA_ARGS__); \
    else kernel<false><<<grid, kOrdThreads, 0, stream>>>(__VA_ARGS__);            \
  } while (0)

// ---- predictor (newton.ts:41-50) -------------------------------------------
// yHat = x0 + h v + h^2 g is the inertial target and, in the reference, the
// first Newton iterate. Exact-Newton mode starts from x0 + h v instead: for a
// sheet resting on a barrier, the gravity term pushes every contact vertex
// into the barrier and Newton spends its first iterations damping back out
// (on the floor drape, 10 iterations per step against 3 in free fall). The
// converged step does not depend on the first iterate.
__global__ void k_predict(Dev d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n) return;
  const double h = d.h;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const double x0 = d.x[i * 3 + k];
    d.x0[i * 3 + k] = x0;
    const double drift = x0 + h * d.v[i * 3 + k];
    const double y = drift + h * h * d.gravity[k];
    d.yHat[i * 3 + k] = y;
    d.x[i * 3 + k] = d.driftGuess ? drift : y;
  }
}

__global__ void k_pins(Dev d, double* x) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= d.npins) return;
  const int id = d.pinIds[k];
  x[id * 3] = d.pinPos[k * 3];
  x[id * 3 + 1] = d.pinPos[k * 3 + 1];
  x[id * 3 + 2] = d.pinPos[k * 3 + 2];
}

// ---- gradient (fem.ts:15-54, newton.ts:113-130) -------------------------------
__global__ void __launch_bounds__(kThreads) k_tri_grad(Dev d) {
  __shared__ double sm[32];
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  double strain = 0;
  if (t < d.m) {
    const uint32_t i0 = d.idx[t * 3], i1 = d.idx[t * 3 + 1], i2 = d.idx[t * 3 + 2];
    double p0[3], p1[3], p2[3];
    load3(d.x, i0, p0); load3(d.x, i1, p1); load3(d.x, i2, p2);
    const float4 iv = d.inv[t];
    double e, g[9], E[3];
    tri_grad<double>(p0, p1, p2, iv.x, iv.y, iv.z, iv.w, d.area[t], d.mat, e, g, E);
#pragma unroll
    for (int k = 0; k < 9; k++) d.elem[(size_t)t * 9 + k] = g[k];
    strain = js_max(js_max(fabs(E[0]), fabs(E[1])), fabs(E[2]));
  }
  const double bm = block_max(strain, sm);
  if (threadIdx.x == 0) d.part[0 * d.partStride + blockIdx.x] = bm;
}

__global__ void __launch_bounds__(kThreads) k_hinge_grad(Dev d) {
  const int hh = blockIdx.x * blockDim.x + threadIdx.x;
  if (hh >= d.hg) return;
  const int4 hv = d.hinge[hh];
  double q[12];
  load3(d.x, hv.x, q); load3(d.x, hv.y, q + 3); load3(d.x, hv.z, q + 6); load3(d.x, hv.w, q + 9);
  double out[12];
  hinge_fd_grad(q, d.hmeta[hh * 3], d.hmeta[hh * 3 + 1], d.hmeta[hh * 3 + 2], d.kb, out);
#pragma unroll
  for (int k = 0; k < 12; k++) d.helem[(size_t)hh * 12 + k] = out[k];
}

// Mixed path: the analytic gradient of the same hinge energy (bend_grad, the
// derivative of bending.ts:7-16) in place of the reference's central
// differences, which cost 24 energy evaluations per hinge.
__global__ void __launch_bounds__(kThreads) k_hinge_grad_analytic(Dev d) {
  const int hh = blockIdx.x * blockDim.x + threadIdx.x;
  if (hh >= d.hg) return;
  const int4 hv = d.hinge[hh];
  double q[12];
  load3(d.x, hv.x, q); load3(d.x, hv.y, q + 3); load3(d.x, hv.z, q + 6); load3(d.x, hv.w, q + 9);
  double out[12];
  bend_grad<double>(q, d.hmeta[hh * 3], d.hmeta[hh * 3 + 1], d.hmeta[hh * 3 + 2], d.kb, out);
#pragma unroll
  for (int k = 0; k < 12; k++) d.helem[(size_t)hh * 12 + k] = out[k];
}

// g = M (x - yHat) / h^2 + gradE (+ contact grad), pin filter, partial |g|^2.
__global__ void __launch_bounds__(kThreads) k_gather_grad(Dev d) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < d.n) {
    double s[3] = {0, 0, 0};
    for (uint32_t k = d.memOff[v]; k < d.memOff[v + 1]; k++) {
      const uint32_t rec = d.memRec[k];
      const double* e = d.elem + (size_t)(rec >> 2) * 9 + (rec & 3) * 3;
      s[0] += e[0]; s[1] += e[1]; s[2] += e[2];
    }
    if (d.kb > 0)
      for (uint32_t k = d.hinOff[v]; k < d.hinOff[v + 1]; k++) {
        const uint32_t rec = d.hinRec[k];
        const double* e = d.helem + (size_t)(rec >> 2) * 12 + (rec & 3) * 3;
        s[0] += e[0]; s[1] += e[1]; s[2] += e[2];
      }
    const double M = d.mass[v];
    const bool pin = d.pinned[v];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const int i = v * 3 + k;
      double gi = M * (d.x[i] - d.yHat[i]) * d.invH2 + s[k];
      if (d.hasContact) gi += d.cgrad[i];
      if (pin) gi = 0;
      d.g[i] = gi;
      d.T0[i] = gi * gi;
    }
  }
}

// Final reduction of the gradient pass: sqrt(sum g^2) in index order
// (newton.ts:128), max strain (order-free).
template <bool SHORT>
__global__ void __launch_bounds__(kOrdThreads) k_grad_final(Dev d, int nbT) {
  const double gs = ordered_sum<kOrdThreads / 32, SHORT>(d.T0, d.n * 3);
  if (threadIdx.x >= 32) return;
  const double ms = warp_max_partials(d.part + 0 * d.partStride, nbT);
  if (threadIdx.x == 0) {
    d.scal[S_GRADNORM] = sqrt(gs);
    d.scal[S_MAXSTRAIN] = ms;
  }
}

// ---- total energy (newton.ts:76-88; fem.ts:56-75) ------------------------------
// Per-element energy terms: inertia 0.5 m d^2 / h^2 per dof into T0, triangle
// energies then hinge energies into T1 (the order internalEnergyOnly adds them).
__global__ void __launch_bounds__(kThreads) k_energy(Dev d, const double* x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < d.n) {
    const double m = d.mass[i];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const double dd = x[i * 3 + k] - d.yHat[i * 3 + k];
      d.T0[i * 3 + k] = 0.5 * m * dd * dd / (d.h * d.h);
    }
  }
  if (i < d.m) {
    double p0[3], p1[3], p2[3];
    load3(x, d.idx[i * 3], p0); load3(x, d.idx[i * 3 + 1], p1); load3(x, d.idx[i * 3 + 2], p2);
    const float4 iv = d.inv[i];
    d.T1[i] = tri_energy<double>(p0, p1, p2, iv.x, iv.y, iv.z, iv.w, d.area[i], d.mat);
  }
  if (i < d.hg && d.kb > 0) {
    const int4 hv = d.hinge[i];
    double q[12];
    load3(x, hv.x, q); load3(x, hv.y, q + 3); load3(x, hv.z, q + 6); load3(x, hv.w, q + 9);
    d.T1[d.m + i] = hinge_energy4(q, d.hmeta[i * 3], d.hmeta[i * 3 + 1], d.hmeta[i * 3 + 2], d.kb);
  }
}

// totalEnergy (newton.ts:76-88): ((sum inertia) + internal) + merit, each sum a
// left-to-right chain; block 0 inertia, block 1 internal, block 2 merit.
template <bool SHORT>
__global__ void __launch_bounds__(kOrdThreads) k_energy_chains(Dev d, int nMerit) {
  const double* t = blockIdx.x == 0 ? d.T0 : blockIdx.x == 1 ? d.T1 : d.Tc;
  const int n = blockIdx.x == 0 ? d.n * 3 : blockIdx.x == 1 ? d.m + (d.kb > 0 ? d.hg : 0) : d.hasContact ? nMerit : 0;
  const double v = ordered_sum<kOrdThreads / 32, SHORT>(t, n);
  if (threadIdx.x == 0) d.scal[S_E_INERTIA + blockIdx.x] = v;
}
__global__ void k_energy_final(Dev d) {
  double e = d.scal[S_E_INERTIA] + d.scal[S_E_TRI];
  if (d.hasContact) e += d.scal[S_E_MERIT];
  d.scal[S_ENERGY_TRIAL] = e;
}

__global__ void k_diag_init(Dev d, double beta) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n * 3) return;
  d.diag[i] = (double)d.mass[i / 3] * d.invH2 + beta;
}

// ---- one-level additive Schwarz (schwarz.ts:154-309) ---------------------------
// Factor: one warp per domain. Lane l owns the rows of member l and adds its
// incident triangles' 9x9 rows in ascending triangle order (the reference's
// per-entry accumulation order); the Cholesky is row-parallel with each entry
// computed by one lane in the reference's sequential inner order.
constexpr int kSchwarzWarps = 4;
__global__ void __launch_bounds__(kSchwarzWarps * 32) k_schwarz_factor(Dev d) {
  __shared__ double A[kSchwarzWarps][24 * 24];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int dom = blockIdx.x * kSchwarzWarps + wib;
  if (dom >= d.D) return;
  double* a = A[wib];
  const int start = d.domStart[dom], dv = d.domStart[dom + 1] - start, dw = dv * 3;
  for (int i = lane; i < 24 * 24; i += 32) a[i] = 0;
  __syncwarp();
  if (lane < dv) {
    const int v = d.domVerts[start + lane];
    for (int k = d.v2tOff[v]; k < d.v2tOff[v + 1]; k++) {
      const int t = d.v2t[k];
      const int cvs[3] = {(int)d.idx[t * 3], (int)d.idx[t * 3 + 1], (int)d.idx[t * 3 + 2]};
      const int ci = cvs[0] == v ? 0 : cvs[1] == v ? 1 : 2;
      double p0[3], p1[3], p2[3];
      load3(d.x, cvs[0], p0); load3(d.x, cvs[1], p1); load3(d.x, cvs[2], p2);
      const float4 iv = d.inv[t];
      double h27[27];
      tri_hessian9_rows<double>(p0, p1, p2, iv.x, iv.y, iv.z, iv.w, d.area[t], d.mat, ci * 3, ci * 3 + 3, h27);
      for (int cj = 0; cj < 3; cj++) {
        int lw = -1;
        for (int q = 0; q < dv; q++)
          if (d.domVerts[start + q] == cvs[cj]) { lw = q; break; }
        if (lw < 0) continue;
        for (int aa = 0; aa < 3; aa++)
          for (int bb = 0; bb < 3; bb++) a[(lane * 3 + aa) * dw + (lw * 3 + bb)] += h27[aa * 9 + cj * 3 + bb];
      }
    }
  }
  __syncwarp();
  if (lane < dw) {
    const int v = d.domVerts[start + lane / 3];
    a[lane * dw + lane] += d.diag[v * 3 + lane % 3];
  }
  __syncwarp();
  for (int i = lane; i < dw; i += 32)
    for (int j = i + 1; j < dw; j++) {
      const double s = 0.5 * (a[i * dw + j] + a[j * dw + i]);
      a[i * dw + j] = s;
      a[j * dw + i] = s;
    }
  __syncwarp();
  double scale = 0;
  for (int i = 0; i < dw; i++) scale = js_max(scale, fabs(a[i * dw + i]));
  const double tiny = 1e-20 * (1 + scale);
  bool ok = true;
  for (int k = 0; k < dw; k++) {
    double diagk = 0;
    if (lane == 0) {
      double sum = a[k * dw + k];
      for (int s = 0; s < k; s++) sum -= a[k * dw + s] * a[k * dw + s];
      ok = sum > tiny;
      if (ok) a[k * dw + k] = sqrt(sum);
    }
    ok = __shfl_sync(0xffffffffu, ok, 0);
    __syncwarp();
    if (!ok) break;
    diagk = a[k * dw + k];
    if (lane > k && lane < dw) {
      double s2 = a[lane * dw + k];
      for (int s = 0; s < k; s++) s2 -= a[lane * dw + s] * a[k * dw + s];
      a[lane * dw + k] = s2 / diagk;
    }
    __syncwarp();
  }
  double* L = d.L + (size_t)dom * 576;
  if (ok) {
    for (int i = lane; i < dw; i += 32)
      for (int j = 0; j < 24; j++)  // the upper triangle holds L^T: a column read gives both
        L[i * 24 + j] = j >= dw ? 0.0 : j <= i ? a[i * dw + j] : a[j * dw + i];
  } else {
    for (int i = lane; i < dw; i += 32) {
      const int v = d.domVerts[start + i / 3];
      const double dd = d.diag[v * 3 + i % 3];
      for (int j = 0; j < 24; j++) L[i * 24 + j] = j == i ? (dd > 1e-12 ? 1 / dd : 0.0) : 0.0;
    }
  }
  if (lane == 0) d.domFlag[dom] = ok ? 1 : 0;
}

// Two-level Schwarz (src/solver/mas.ts buildCoarseDiag, mas.ts:57-101): the
// coarse diagonal of each domain, one thread per domain, in the reference's
// accumulation order: the domain's triangles in ascending order, their
// within-domain (ci, cj) pairs, then the Jacobi diagonal over the members.
constexpr int kCoarseTris = 96;  // triangles touching a domain of <= 8 vertices
__global__ void __launch_bounds__(kThreads) k_coarse_diag(Dev d) {
  const int dom = blockIdx.x * blockDim.x + threadIdx.x;
  if (dom >= d.D) return;
  const int start = d.domStart[dom], dv = d.domStart[dom + 1] - start;
  int tris[kCoarseTris];
  int nt = 0;
  for (int l = 0; l < dv; l++) {
    const int v = d.domVerts[start + l];
    for (int k = d.v2tOff[v]; k < d.v2tOff[v + 1]; k++) {
      const int t = d.v2t[k];
      int pos = nt;  // insertion into the sorted list, duplicates skipped
      bool dup = false;
      for (int q = 0; q < nt; q++) {
        if (tris[q] == t) { dup = true; break; }
        if (tris[q] > t) { pos = q; break; }
      }
      if (dup || nt >= kCoarseTris) continue;
      for (int q = nt; q > pos; q--) tris[q] = tris[q - 1];
      tris[pos] = t;
      nt++;
    }
  }
  auto inDom = [&](int v) {
    for (int l = 0; l < dv; l++)
      if (d.domVerts[start + l] == v) return true;
    return false;
  };
  double dc[3] = {0, 0, 0};
  for (int q = 0; q < nt; q++) {
    const int t = tris[q];
    const int cvs[3] = {(int)d.idx[t * 3], (int)d.idx[t * 3 + 1], (int)d.idx[t * 3 + 2]};
    const bool in[3] = {inDom(cvs[0]), inDom(cvs[1]), inDom(cvs[2])};
    double p0[3], p1[3], p2[3];
    load3(d.x, cvs[0], p0); load3(d.x, cvs[1], p1); load3(d.x, cvs[2], p2);
    const float4 iv = d.inv[t];
    for (int ci = 0; ci < 3; ci++) {
      if (!in[ci]) continue;
      double h27[27];  // rows ci*3 .. ci*3+2 of the 9x9 block
      tri_hessian9_rows<double>(p0, p1, p2, iv.x, iv.y, iv.z, iv.w, d.area[t], d.mat, ci * 3, ci * 3 + 3, h27);
      for (int cj = 0; cj < 3; cj++) {
        if (!in[cj]) continue;
        const double s = 1.0 / (double)dv;
        for (int a = 0; a < 3; a++) dc[a] += s * h27[a * 9 + cj * 3 + a];
      }
    }
  }
  for (int l = 0; l < dv; l++) {
    const int v = d.domVerts[start + l];
    const double s = 1.0 / (double)dv;
    for (int a = 0; a < 3; a++) dc[a] += s * d.diag[v * 3 + a];
  }
  for (int a = 0; a < 3; a++) d.dcoarse[dom * 3 + a] = dc[a];
}

// ---- standalone FD membrane HVP (fem.ts:108-130) -----------------------------------
// out = (gradM(x + h p) - gradM(x - h p)) / (2h), h = 1e-8 (1 + |p|): the same
// element and gather arithmetic as the PCG kernel's HVP phase, as plain kernels.
__global__ void k_hvp_terms(const double* p, int n3, double* T) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n3) T[i] = p[i] * p[i];
}
template <bool SHORT>
__global__ void __launch_bounds__(kOrdThreads) k_hvp_h(const double* T, int n3, double* h) {
  const double pp = ordered_sum<kOrdThreads / 32, SHORT>(T, n3);
  if (threadIdx.x == 0) *h = 1e-8 * (1 + sqrt(pp));
}
__device__ __forceinline__ void hvp_elem_tri(int t, const uint32_t* idx, const float4* inv, const float* area,
                                             const Mat<double>& mat, const double* x, const double* p, double h,
                                             double* elem) {
  const uint32_t vi[3] = {idx[t * 3], idx[t * 3 + 1], idx[t * 3 + 2]};
  double xp[9], xm[9];
#pragma unroll
  for (int c = 0; c < 3; c++)
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const double xx = x[vi[c] * 3 + q], pq = p[vi[c] * 3 + q];
      xp[c * 3 + q] = xx + h * pq;
      xm[c * 3 + q] = xx - h * pq;
    }
  const float4 iv = inv[t];
  double e, gp[9], gm[9], E[3];
  tri_grad<double>(xp, xp + 3, xp + 6, iv.x, iv.y, iv.z, iv.w, area[t], mat, e, gp, E);
  tri_grad<double>(xm, xm + 3, xm + 6, iv.x, iv.y, iv.z, iv.w, area[t], mat, e, gm, E);
  double* o = elem + (size_t)t * 18;
#pragma unroll
  for (int q = 0; q < 9; q++) { o[q] = gp[q]; o[9 + q] = gm[q]; }
}
__global__ void __launch_bounds__(kThreads) k_hvp_elem(const uint32_t* idx, const float4* inv, const float* area,
                                                       Mat<double> mat, int m, const double* x, const double* p,
                                                       const double* h, double* elem) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < m) hvp_elem_tri(t, idx, inv, area, mat, x, p, *h, elem);
}
__global__ void __launch_bounds__(kThreads) k_hvp_gather(const uint32_t* memOff, const uint32_t* memRec, int n,
                                                         const double* elem, const double* h, double* out) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n) return;
  double sp[3] = {0, 0, 0}, sn[3] = {0, 0, 0};
  for (uint32_t q = memOff[v]; q < memOff[v + 1]; q++) {
    const uint32_t rec = memRec[q];
    const double* e = elem + (size_t)(rec >> 2) * 18 + (rec & 3) * 3;
    sp[0] += e[0]; sp[1] += e[1]; sp[2] += e[2];
    sn[0] += e[9]; sn[1] += e[10]; sn[2] += e[11];
  }
  const double hh = *h;
#pragma unroll
  for (int c = 0; c < 3; c++) out[v * 3 + c] = (sp[c] - sn[c]) / (2 * hh);
}

void launch_membrane_hvp(const uint32_t* idx, const float4* inv, const float* area, const Mat<double>& mat, int n,
                         int m, const uint32_t* memOff, const uint32_t* memRec, const double* x, const double* p,
                         double* out, double* T, double* h, double* elem, cudaStream_t s) {
  k_hvp_terms<<<nblk(n * 3), kThreads, 0, s>>>(p, n * 3, T);
  ORD_LAUNCH(k_hvp_h, n * 3, 1, s, T, n * 3, h);
  k_hvp_elem<<<nblk(m), kThreads, 0, s>>>(idx, inv, area, mat, m, x, p, h, elem);
  k_hvp_gather<<<nblk(n), kThreads, 0, s>>>(memOff, memRec, n, elem, h, out);
}

// ---- material-model evaluation (material-model.ts:278-288) -------------------------
// internalEnergyOnly (fem.ts:56-75) terms: triangle energies, then hinge
// energies when kb > 0, into T1 in the order the reference adds them.
__global__ void __launch_bounds__(kThreads) k_internal_energy_terms(Dev d, const double* x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < d.m) {
    double p0[3], p1[3], p2[3];
    load3(x, d.idx[i * 3], p0); load3(x, d.idx[i * 3 + 1], p1); load3(x, d.idx[i * 3 + 2], p2);
    const float4 iv = d.inv[i];
    d.T1[i] = tri_energy<double>(p0, p1, p2, iv.x, iv.y, iv.z, iv.w, d.area[i], d.mat);
  }
  if (i < d.hg && d.kb > 0) {
    const int4 hv = d.hinge[i];
    double q[12];
    load3(x, hv.x, q); load3(x, hv.y, q + 3); load3(x, hv.z, q + 6); load3(x, hv.w, q + 9);
    d.T1[d.m + i] = hinge_energy4(q, d.hmeta[i * 3], d.hmeta[i * 3 + 1], d.hmeta[i * 3 + 2], d.kb);
  }
}
// evalInternal's gradient (fem.ts:15-54): per vertex, its triangle terms in
// ascending triangle order, then its hinge terms in hinge order (the
// reference's scatter order); no inertia, pins or contact.
__global__ void __launch_bounds__(kThreads) k_gather_internal(Dev d, double* grad) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= d.n) return;
  double s[3] = {0, 0, 0};
  for (uint32_t k = d.memOff[v]; k < d.memOff[v + 1]; k++) {
    const uint32_t rec = d.memRec[k];
    const double* e = d.elem + (size_t)(rec >> 2) * 9 + (rec & 3) * 3;
    s[0] += e[0]; s[1] += e[1]; s[2] += e[2];
  }
  if (d.kb > 0)
    for (uint32_t k = d.hinOff[v]; k < d.hinOff[v + 1]; k++) {
      const uint32_t rec = d.hinRec[k];
      const double* e = d.helem + (size_t)(rec >> 2) * 12 + (rec & 3) * 3;
      s[0] += e[0]; s[1] += e[1]; s[2] += e[2];
    }
  grad[v * 3] = s[0];
  grad[v * 3 + 1] = s[1];
  grad[v * 3 + 2] = s[2];
}
// out[0] = the internal energy chain, out[1] = max strain over the triangle
// partials (nbT of them; 0 when none were computed).
template <bool SHORT>
__global__ void __launch_bounds__(kOrdThreads) k_internal_final(Dev d, int nbT, double* out) {
  const double e = ordered_sum<kOrdThreads / 32, SHORT>(d.T1, d.m + (d.kb > 0 ? d.hg : 0));
  if (threadIdx.x >= 32) return;
  const double ms = nbT > 0 ? warp_max_partials(d.part + 0 * d.partStride, nbT) : 0.0;
  if (threadIdx.x == 0) {
    out[0] = e;
    out[1] = ms;
  }
}
// evalMembraneHvp (membrane-hvp.ts:80-108): the analytic per-triangle HVP
// (triangleHvp, membrane-hvp.ts:18-75) and the same vertex gather order.
__global__ void __launch_bounds__(kThreads) k_tri_hvp_elem(Dev d, const double* x, const double* p) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= d.m) return;
  const uint32_t i0 = d.idx[t * 3], i1 = d.idx[t * 3 + 1], i2 = d.idx[t * 3 + 2];
  double p0[3], p1[3], p2[3], v0[3], v1[3], v2[3];
  load3(x, i0, p0); load3(x, i1, p1); load3(x, i2, p2);
  load3(p, i0, v0); load3(p, i1, v1); load3(p, i2, v2);
  const float4 iv = d.inv[t];
  double o[9];
  tri_hvp<double>(p0, p1, p2, v0, v1, v2, iv.x, iv.y, iv.z, iv.w, d.area[t], d.mat, o);
#pragma unroll
  for (int k = 0; k < 9; k++) d.elem[(size_t)t * 9 + k] = o[k];
}
__global__ void __launch_bounds__(kThreads) k_gather_elem9(Dev d, double* out) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= d.n) return;
  double s[3] = {0, 0, 0};
  for (uint32_t k = d.memOff[v]; k < d.memOff[v + 1]; k++) {
    const uint32_t rec = d.memRec[k];
    const double* e = d.elem + (size_t)(rec >> 2) * 9 + (rec & 3) * 3;
    s[0] += e[0]; s[1] += e[1]; s[2] += e[2];
  }
  out[v * 3] = s[0];
  out[v * 3 + 1] = s[1];
  out[v * 3 + 2] = s[2];
}

void launch_internal_eval(const Dev& d0, const double* x, double* grad, double* out2, cudaStream_t s) {
  Dev d = d0;
  d.x = const_cast<double*>(x);
  int nbT = 0;
  if (grad) {
    k_tri_grad<<<nblk(d.m), kThreads, 0, s>>>(d);
    nbT = nblk(d.m);
    if (d.kb > 0 && d.hg > 0) k_hinge_grad<<<nblk(d.hg), kThreads, 0, s>>>(d);
    k_gather_internal<<<nblk(d.n), kThreads, 0, s>>>(d, grad);
  }
  k_internal_energy_terms<<<nblk(std::max(d.m, d.hg)), kThreads, 0, s>>>(d, x);
  ORD_LAUNCH(k_internal_final, d.m + (d.kb > 0 ? d.hg : 0), 1, s, d, nbT, out2);
}

void launch_membrane_hvp_analytic(const Dev& d, const double* x, const double* p, double* out, cudaStream_t s) {
  k_tri_hvp_elem<<<nblk(d.m), kThreads, 0, s>>>(d, x, p);
  k_gather_elem9<<<nblk(d.n), kThreads, 0, s>>>(d, out);
}

// ---- Armijo trial + velocity ----------------------------------------------------
__global__ void k_trial(Dev d, double alpha) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n * 3) return;
  d.xt[i] = d.x[i] + alpha * d.dx[i];
}

__global__ void k_velocity(Dev d, double damp) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n * 3) return;
  d.v[i] = ((d.x[i] - d.x0[i]) / d.h) * damp;
}

// ---- simulation-session hand-off -------------------------------------------------
// flag = 1 when any coordinate of x is non-finite.
__global__ void k_nonfinite(const double* x, int n3, int* flag) {
  int bad = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n3; i += gridDim.x * blockDim.x)
    if (!isfinite(x[i])) bad = 1;
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(flag, 1);
}
// stable <- x when the flag is clear (the last NaN-free state stays on the device).
__global__ void k_keep_if_finite(const double* x, double* stable, int n3, const int* flag) {
  if (*flag) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n3; i += gridDim.x * blockDim.x) stable[i] = x[i];
}

void launch_session_check(const double* x, double* stable, int n3, int* flag, cudaStream_t s) {
  cudaMemsetAsync(flag, 0, sizeof(int), s);
  const int blocks = std::min(1184, std::max(1, (n3 + kThreads - 1) / kThreads));
  k_nonfinite<<<blocks, kThreads, 0, s>>>(x, n3, flag);
  k_keep_if_finite<<<blocks, kThreads, 0, s>>>(x, stable, n3, flag);
}

// ---- launchers ------------------------------------------------------------------

void launch_predict(const Dev& d, cudaStream_t s) {
  k_predict<<<nblk(d.n), kThreads, 0, s>>>(d);
  launch_pins(d, d.x, s);
}
void launch_pins(const Dev& d, double* x, cudaStream_t s) {
  if (d.npins > 0) k_pins<<<nblk(d.npins), kThreads, 0, s>>>(d, x);
}
void launch_grad_terms(const Dev& d, cudaStream_t s, bool analyticBend) {
  k_tri_grad<<<nblk(d.m), kThreads, 0, s>>>(d);
  if (d.kb > 0 && d.hg > 0) {
    if (analyticBend) k_hinge_grad_analytic<<<nblk(d.hg), kThreads, 0, s>>>(d);
    else k_hinge_grad<<<nblk(d.hg), kThreads, 0, s>>>(d);
  }
  k_gather_grad<<<nblk(d.n), kThreads, 0, s>>>(d);
}
void launch_grad(const Dev& d, cudaStream_t s, bool analyticBend) {
  launch_grad_terms(d, s, analyticBend);
  ORD_LAUNCH(k_grad_final, d.n * 3, 1, s, d, nblk(d.m));
}
void launch_energy_terms(const Dev& d, const double* x, cudaStream_t s) {
  const int nb = nblk(std::max(std::max(d.n, d.m), d.hg));
  k_energy<<<nb, kThreads, 0, s>>>(d, x);
}
void launch_energy(const Dev& d, const double* x, cudaStream_t s) {
  launch_energy_terms(d, x, s);
  const int nMerit = d.hasContact ? d.c.nActive : 0;
  ORD_LAUNCH(k_energy_chains, std::max(std::max(d.n * 3, d.m + (d.kb > 0 ? d.hg : 0)), nMerit), 3, s, d, nMerit);
  k_energy_final<<<1, 1, 0, s>>>(d);
}
void launch_diag_init(const Dev& d, double beta, cudaStream_t s) {
  k_diag_init<<<nblk(d.n * 3), kThreads, 0, s>>>(d, beta);
}
void launch_schwarz_factor(const Dev& d, cudaStream_t s) {
  k_schwarz_factor<<<(d.D + kSchwarzWarps - 1) / kSchwarzWarps, kSchwarzWarps * 32, 0, s>>>(d);
  if (d.precond == 2) k_coarse_diag<<<nblk(d.D), kThreads, 0, s>>>(d);
}
void launch_trial(const Dev& d, double alpha, cudaStream_t s) {
  k_trial<<<nblk(d.n * 3), kThreads, 0, s>>>(d, alpha);
  launch_pins(d, d.xt, s);
}
void launch_velocity(const Dev& d, double damp, cudaStream_t s) {
  k_velocity<<<nblk(d.n * 3), kThreads, 0, s>>>(d, damp);
}

}  // namespace cs
