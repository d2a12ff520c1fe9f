// Adjoint of the implicit-Euler step through the implicit-function theorem
// (no reference counterpart; it differentiates newton.ts:27-232).
//
// A converged step satisfies g(x1; x0, v0, theta) = 0 with
//   g = M (x1 - yHat) / h^2 + grad E_membrane(x1; C00, C11, C01, G)
//       + grad E_bend(x1; k) + grad E_contact(x1),   yHat = x0 + h v0 + h^2 g_grav,
// so for a loss L(x1): H mu = dL/dx1 (H = dg/dx1, symmetric), and
//   dL/dtheta = -mu . dg/dtheta,  dL/dx0 = M mu / h^2,  dL/dv0 = M mu / h.
// H is applied matrix-free in FP64: M/h^2, the analytic membrane HVP
// (membrane-hvp.ts:18-75), the exact bending HVP (dual numbers over the
// analytic hinge gradient) and the frozen-contact barrier HVP
// (contact-assembly.ts:371-414, active set frozen at x1). Friction and the
// restitution filter are treated as constants, as the forward Newton HVP
// treats friction. Pinned dofs are filtered out of every vector.
//
// dg/dtheta: the membrane gradient is linear in (C00, C11, C01, G), so its
// derivative along C00 is the gradient evaluated with C00 = 1 and the others 0
// (likewise C11, G); the bending gradient is linear in k, so its derivative is
// the analytic hinge gradient at k = 1, the gradient the exact-Newton forward
// takes (the derivative of bending.ts:7-16).
#include <cooperative_groups.h>

#include <map>
#include <mutex>

#include "adjoint.cuh"
#include "adjoint_math.cuh"
#include "contact.cuh"
#include "schwarz64.cuh"

namespace cg = cooperative_groups;

namespace cs {

__device__ __forceinline__ void load3(const double* x, int v, double o[3]) {
  o[0] = x[v * 3]; o[1] = x[v * 3 + 1]; o[2] = x[v * 3 + 2];
}

__device__ __forceinline__ double adj_total(const Dev& d, int row, int blocks, double* bc) {
  if (threadIdx.x < 32) {
    const double s = warp_sum_partials(d.part + row * d.partStride, blocks);
    if (threadIdx.x == 0) bc[0] = s;
  }
  __syncthreads();
  const double r = bc[0];
  __syncthreads();
  return r;
}
__device__ __forceinline__ void adj_put(const Dev& d, int row, double v, double* sm) {
  const double b = block_sum(v, sm);
  if (threadIdx.x == 0) d.part[row * d.partStride + blockIdx.x] = b;
}

// Membrane HVP in FP64 (membrane-hvp.ts:18-75). With psd set, the second
// Piola stress S in the geometric term dF S is replaced by its positive part
// (negative principal stresses of a compressed triangle clamped to zero), which
// makes every element block positive semi-definite: a Newton matrix for the
// forward solve that leaves its converged solution unchanged.
__device__ __forceinline__ void mem_hvp64(const double* x0, const double* x1, const double* x2, const double* v0,
                                          const double* v1, const double* v2, double a, double b, double c, double d,
                                          double area, const Mat<double>& m, bool psd, double out[9]) {
  double F0[3], F1[3], dF0[3], dF1[3];
  for (int k = 0; k < 3; k++) {
    const double e1 = x1[k] - x0[k], e2 = x2[k] - x0[k];
    const double w1 = v1[k] - v0[k], w2 = v2[k] - v0[k];
    F0[k] = a * e1 + c * e2;
    F1[k] = b * e1 + d * e2;
    dF0[k] = a * w1 + c * w2;
    dF1[k] = b * w1 + d * w2;
  }
  const double E00 = 0.5 * (F0[0] * F0[0] + F0[1] * F0[1] + F0[2] * F0[2] - 1);
  const double E11 = 0.5 * (F1[0] * F1[0] + F1[1] * F1[1] + F1[2] * F1[2] - 1);
  const double E01 = 0.5 * (F0[0] * F1[0] + F0[1] * F1[1] + F0[2] * F1[2]);
  const double dE00 = F0[0] * dF0[0] + F0[1] * dF0[1] + F0[2] * dF0[2];
  const double dE11 = F1[0] * dF1[0] + F1[1] * dF1[1] + F1[2] * dF1[2];
  const double dE01 = 0.5 * (dF0[0] * F1[0] + F0[0] * dF1[0] + dF0[1] * F1[1] + F0[1] * dF1[1] + dF0[2] * F1[2] +
                             F0[2] * dF1[2]);
  double S00 = m.C00 * E00 + m.C01 * E11;
  double S11 = m.C11 * E11 + m.C01 * E00;
  double S01 = 2 * m.G * E01;
  if (psd) psd_stress(S00, S11, S01);
  const double dS00 = m.C00 * dE00 + m.C01 * dE11;
  const double dS11 = m.C11 * dE11 + m.C01 * dE00;
  const double dS01 = 2 * m.G * dE01;
  const double s = m.thickness * area;
  for (int k = 0; k < 3; k++) {
    const double P0 = dF0[k] * S00 + F0[k] * dS00 + dF1[k] * S01 + F1[k] * dS01;
    const double P1 = dF0[k] * S01 + F0[k] * dS01 + dF1[k] * S11 + F1[k] * dS11;
    const double g1 = s * (P0 * a + P1 * b);
    const double g2 = s * (P0 * c + P1 * d);
    out[k] = -(g1 + g2);
    out[3 + k] = g1;
    out[6 + k] = g2;
  }
}

// PCG on H mu = rhs (pcg.ts's recurrence, FP64 tree reductions), one launch of C
// CTAs. out: [iterations, final residual, |rhs|].
//
// Small sheets are bound by latency: the hinges' dual-number products and the
// domains' substitutions are long dependent chains, and every phase ends in a
// barrier. So all C CTAs share the elements and the domains (a warp each), and up
// to 16 reducing blocks run as one thread-block cluster with its hardware barrier.
// The reductions keep the shape of `blocks` blocks of kThreads, whatever C is: the
// first `blocks` CTAs hold the vectors' elements, so results do not depend on how
// the rest of the work is spread. On a B200, 19 x 16 vertices with Schwarz took
// 65 us an iteration with a thread per domain on 4 cooperative blocks, 27 us now;
// a fit's forward and backward pass 1.25 -> 0.51 s, the same bits.
template <bool CLUSTER>
__global__ void __launch_bounds__(kThreads) k_adj_pcg(AdjArgs A, int blocks) {
  __shared__ double sm[32];
  __shared__ double bc[2];
  auto barrier = [&]() {
    if constexpr (CLUSTER) cg::this_cluster().sync();
    else cg::this_grid().sync();
  };
  const Dev& d = A.d;
  const bool reducing = (int)blockIdx.x < blocks;
  const int n3 = d.n * 3;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nthAll = gridDim.x * blockDim.x;
  const int nth = blocks * blockDim.x;
  const int i0 = reducing ? tid : n3, v0 = reducing ? tid : d.n;
  const int gwarp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, nwarps = nthAll >> 5;
  auto put = [&](int row, double v) {
    if (reducing) adj_put(d, row, v, sm);
  };
  auto total = [&](int row) { return adj_total(d, row, blocks, bc); };
  // z = M^-1 r (one-level Schwarz factors, or Jacobi); this thread's share of r.z.
  // (The two-level coarse term is not applied here.)
  auto precond = [&]() {
    double rz = 0;
    if (d.precond >= 1) {
      for (int dom = gwarp; dom < d.D; dom += nwarps) {
        const double s = domain_solve(d.L + (size_t)dom * 576, A.r, A.z, nullptr, domain_lane(d, dom));
        if ((threadIdx.x & 31) == 0) A.domRz[dom] = s;
      }
      barrier();
      for (int dom = reducing ? tid : d.D; dom < d.D; dom += nth) rz += __ldcg(A.domRz + dom);
    } else {
      for (int i = i0; i < n3; i += nth) {
        const double ri = A.r[i];
        double zi = d.diag[i] > 1e-12 ? ri / d.diag[i] : ri;
        if (d.pinned[i / 3]) zi = 0;
        A.z[i] = zi;
        rz += ri * zi;
      }
    }
    return rz;
  };
  double bb = 0, rr = 0;
  for (int i = i0; i < n3; i += nth) {
    const double ri = d.pinned[i / 3] ? 0.0 : A.rhs[i];
    bb += A.rhs[i] * A.rhs[i];
    A.r[i] = ri;
    A.mu[i] = 0;
    rr += ri * ri;
  }
  barrier();
  const double rz0 = precond();
  put(0, bb);
  put(1, rr);
  put(2, rz0);
  barrier();
  for (int i = i0; i < n3; i += nth) A.p[i] = __ldcg(A.z + i);
  const double bNorm = sqrt(total(0));
  double residual = sqrt(total(1));
  double rz = total(2);
  const double absTol = fmax(A.tol * bNorm, 1e-300);
  int k = 0;
  bool done = !(residual > absTol);
  barrier();
  for (; !done && k < A.maxIters; k++) {
    // ---- H p: elements on every CTA, then the vertex sums ----
    const int nHin = A.kb > 0 ? d.hg : 0;
    // whole warps of one kind of element: hinges first, they take longest
    const int hinPad = (nHin + 31) & ~31;
    for (int e = tid; e < hinPad + d.m; e += nthAll) {
      if (e < nHin) {
        const int4 hv = __ldg(d.hinge + e);
        double q[12], v[12], o[12];
        load3(d.x, hv.x, q); load3(d.x, hv.y, q + 3); load3(d.x, hv.z, q + 6); load3(d.x, hv.w, q + 9);
        load3(A.p, hv.x, v); load3(A.p, hv.y, v + 3); load3(A.p, hv.z, v + 6); load3(A.p, hv.w, v + 9);
        bend_hvp(q, v, d.hmeta[e * 3], d.hmeta[e * 3 + 1], d.hmeta[e * 3 + 2], A.kb, o);
#pragma unroll
        for (int c = 0; c < 12; c++) A.hin12[(size_t)e * 12 + c] = o[c];
      } else if (e >= hinPad) {
        const int t = e - hinPad;
        const uint32_t t0 = __ldg(d.idx + t * 3), t1 = __ldg(d.idx + t * 3 + 1), t2 = __ldg(d.idx + t * 3 + 2);
        double x0[3], x1[3], x2[3], w0[3], w1[3], w2[3];
        load3(d.x, t0, x0); load3(d.x, t1, x1); load3(d.x, t2, x2);
        load3(A.p, t0, w0); load3(A.p, t1, w1); load3(A.p, t2, w2);
        const float4 iv = __ldg(d.inv + t);
        double o[9];
        mem_hvp64(x0, x1, x2, w0, w1, w2, iv.x, iv.y, iv.z, iv.w, d.area[t], d.mat, A.psd != 0, o);
#pragma unroll
        for (int c = 0; c < 9; c++) A.tri9[(size_t)t * 9 + c] = o[c];
      }
    }
    if (d.hasContact) contact_hvp_coeffs(d, A.p, tid, nthAll);
    barrier();
    double pAp = 0;
    for (int v = v0; v < d.n; v += nth) {
      double s[3] = {0, 0, 0};
      for (uint32_t q0 = d.memOff[v], q1 = d.memOff[v + 1]; q0 < q1; q0 += 4) {
        double e[4][3];  // four incidences in flight, added in order
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const bool on = q0 + u < q1;
          const uint32_t rec = on ? __ldg(d.memRec + q0 + u) : 0u;
#pragma unroll
          for (int c = 0; c < 3; c++) e[u][c] = on ? A.tri9[(size_t)(rec >> 2) * 9 + (rec & 3) * 3 + c] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; u++) { s[0] += e[u][0]; s[1] += e[u][1]; s[2] += e[u][2]; }
      }
      if (A.kb > 0)
        for (uint32_t q0 = d.hinOff[v], q1 = d.hinOff[v + 1]; q0 < q1; q0 += 4) {
          double e[4][3];
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const bool on = q0 + u < q1;
            const uint32_t rec = on ? __ldg(d.hinRec + q0 + u) : 0u;
#pragma unroll
            for (int c = 0; c < 3; c++) e[u][c] = on ? A.hin12[(size_t)(rec >> 2) * 12 + (rec & 3) * 3 + c] : 0.0;
          }
#pragma unroll
          for (int u = 0; u < 4; u++) { s[0] += e[u][0]; s[1] += e[u][1]; s[2] += e[u][2]; }
        }
      double ch[3] = {0, 0, 0};
      if (d.hasContact) contact_hvp_gather(d, v, ch);
      const double M = d.mass[v];
      const bool pin = d.pinned[v];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const int i = v * 3 + c;
        const double ap = pin ? 0.0 : M * A.p[i] * d.invH2 + s[c] + ch[c];
        A.Ap[i] = ap;
        pAp += A.p[i] * ap;
      }
    }
    put(3, pAp);
    barrier();
    const double pApT = total(3);
    if (!(pApT > 0)) break;  // H not positive along p: stop with the current iterate
    const double alpha = rz / pApT;
    double rrn = 0;
    for (int i = i0; i < n3; i += nth) {
      A.mu[i] += alpha * A.p[i];
      const double ri = A.r[i] - alpha * A.Ap[i];
      A.r[i] = ri;
      rrn += ri * ri;
    }
    barrier();
    const double rzn = precond();
    put(4, rrn);
    put(5, rzn);
    barrier();
    residual = sqrt(total(4));
    const double rzNew = total(5);
    if (!(residual > absTol)) { k++; done = true; break; }
    const double beta = rzNew / rz;
    rz = rzNew;
    for (int i = i0; i < n3; i += nth) A.p[i] = __ldcg(A.z + i) + beta * A.p[i];
    barrier();
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    A.out[0] = k;
    A.out[1] = residual;
    A.out[2] = bNorm;
  }
}

// Per-element terms of mu . dg/dtheta for theta = (C00, C11, G, k): four rows
// of per-triangle / per-hinge values in `terms` (stride m + hg), summed later.
__global__ void __launch_bounds__(kThreads) k_adj_theta_terms(Dev d, const double* mu, double* terms, int stride) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < d.m) {
    const uint32_t ids[3] = {d.idx[e * 3], d.idx[e * 3 + 1], d.idx[e * 3 + 2]};
    double x0[3], x1[3], x2[3];
    load3(d.x, ids[0], x0); load3(d.x, ids[1], x1); load3(d.x, ids[2], x2);
    const float4 iv = d.inv[e];
    double mu9[9];
    for (int c = 0; c < 3; c++) {
      const bool pin = d.pinned[ids[c]];
      for (int k = 0; k < 3; k++) mu9[c * 3 + k] = pin ? 0.0 : mu[ids[c] * 3 + k];
    }
    const double th = d.mat.thickness;
    const Mat<double> unit[3] = {{1, 0, 0, 0, th}, {0, 1, 0, 0, th}, {0, 0, 0, 1, th}};
    for (int j = 0; j < 3; j++) {
      double en, g[9], E[3];
      tri_grad<double>(x0, x1, x2, iv.x, iv.y, iv.z, iv.w, d.area[e], unit[j], en, g, E);
      double s = 0;
      for (int k = 0; k < 9; k++) s += mu9[k] * g[k];
      terms[(size_t)j * stride + e] = s;
    }
    terms[(size_t)3 * stride + e] = 0;
  } else if (e < d.m + d.hg) {
    const int hh = e - d.m;
    const int4 hv = d.hinge[hh];
    const int ids[4] = {hv.x, hv.y, hv.z, hv.w};
    double q[12], g[12];
    for (int c = 0; c < 4; c++) load3(d.x, ids[c], q + c * 3);
    bend_grad<double>(q, d.hmeta[hh * 3], d.hmeta[hh * 3 + 1], d.hmeta[hh * 3 + 2], 1.0, g);
    double s = 0;
    for (int c = 0; c < 4; c++) {
      if (d.pinned[ids[c]]) continue;
      for (int k = 0; k < 3; k++) s += mu[ids[c] * 3 + k] * g[c * 3 + k];
    }
    for (int j = 0; j < 3; j++) terms[(size_t)j * stride + e] = 0;
    terms[(size_t)3 * stride + e] = s;
  }
}

// Fixed-order sums of the four rows (one block per row); acc[j] -= sum.
__global__ void __launch_bounds__(1024) k_adj_theta_sum(const double* terms, int stride, int count, double* acc) {
  __shared__ double sm[32];
  double s = 0;
  for (int i = threadIdx.x; i < count; i += blockDim.x) s += terms[(size_t)blockIdx.x * stride + i];
  const double t = block_sum(s, sm);
  if (threadIdx.x == 0) acc[blockIdx.x] -= t;
}

// lambda_x0 = M mu / h^2 - (damp / h) lambda_v,  lambda_v0 = M mu / h (pins filtered);
// then the next step's total lambda_x1 = lambda_x0 + (damp / h) lambda_v0 is formed
// by the caller through adj_rhs.
__global__ void k_adj_propagate(Dev d, const double* mu, double* lamX, double* lamV, double damp) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n * 3) return;
  const int v = i / 3;
  if (d.pinned[v]) { lamX[i] = 0; lamV[i] = 0; return; }
  const double M = d.mass[v];
  const double lv = lamV[i];
  lamX[i] = M * mu[i] * d.invH2 - damp * lv / d.h;
  lamV[i] = M * mu[i] / d.h;
}

// rhs = lambda_x1 + (damp / h) lambda_v1 (v1 = damp (x1 - x0) / h).
__global__ void k_adj_rhs(Dev d, const double* lamX, const double* lamV, double damp, double* rhs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.n * 3) return;
  rhs[i] = d.pinned[i / 3] ? 0.0 : lamX[i] + damp * lamV[i] / d.h;
}

// Newton epilogue after the full-Hessian solve (newton.ts:152-179): descent
// safeguard (Jacobi-scaled steepest descent when g.dx >= 0) and the 2 mm trust
// region. One block; tree reductions. Writes the step's scalars.
__global__ void __launch_bounds__(1024) k_newton_epilogue(Dev d, const double* out3) {
  __shared__ double sm[32];
  const int n3 = d.n * 3;
  double gt = 0;
  for (int i = threadIdx.x; i < n3; i += blockDim.x) gt += d.g[i] * d.dx[i];
  double gtdx = block_sum(gt, sm);
  bool fallback = false;
  if (!isfinite(gtdx) || gtdx >= 0) {
    fallback = true;
    gt = 0;
    for (int i = threadIdx.x; i < n3; i += blockDim.x) {
      const double di = -d.g[i] / d.diag[i];
      d.dx[i] = di;
      gt += d.g[i] * di;
    }
    gtdx = block_sum(gt, sm);
  }
  double mx = 0;
  for (int i = threadIdx.x; i < n3; i += blockDim.x) mx = fmax(mx, fabs(d.dx[i]));
  const double maxDx = block_max(mx, sm);
  if (maxDx > 0.002) {
    const double sc = 0.002 / maxDx;
    for (int i = threadIdx.x; i < n3; i += blockDim.x) d.dx[i] *= sc;
    gtdx *= sc;
  }
  if (threadIdx.x == 0) {
    d.scal[S_PCG_ITERS] = out3[0];
    d.scal[S_PCG_RES] = out3[1];
    d.scal[S_GTDX] = gtdx;
    d.scal[S_FALLBACK] = fallback ? 1 : 0;
    d.scal[S_MAXDX] = maxDx;
  }
}

__global__ void k_neg_grad(Dev d, double* rhs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < d.n * 3) rhs[i] = -d.g[i];
}

int newton_exact_solve(const AdjArgs& a, int blocks, cudaStream_t s) {
  k_neg_grad<<<(a.d.n * 3 + kThreads - 1) / kThreads, kThreads, 0, s>>>(a.d, const_cast<double*>(a.rhs));
  const int rc = adj_launch_pcg(a, blocks, s);
  if (rc != 0) return rc;
  k_newton_epilogue<<<1, 1024, 0, s>>>(a.d, a.out);
  return (int)cudaGetLastError();
}

static inline int ablk(long n) { return (int)((n + kThreads - 1) / kThreads); }

namespace {

constexpr int kAdjCluster = 16;  // CTAs of the cluster launch, and the most blocks it reduces over

struct AdjDevice {
  int sms = 0, maxCtas = 0;
  bool cluster = false;
};
void adj_cluster_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr) {
  cfg.gridDim = dim3(kAdjCluster);
  cfg.blockDim = dim3(kThreads);
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kAdjCluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
}
AdjDevice adj_device() {
  static std::mutex mu;
  static std::map<int, AdjDevice> known;  // per device
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  const auto it = known.find(dev);
  if (it != known.end()) return it->second;
  AdjDevice a;
  int per = 0, nc = 0;
  cudaDeviceGetAttribute(&a.sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_adj_pcg<false>, kThreads, 0);
  a.maxCtas = std::max(1, per * a.sms);
  cudaFuncSetAttribute(k_adj_pcg<true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  adj_cluster_config(cfg, attr);
  a.cluster = cudaOccupancyMaxActiveClusters(&nc, k_adj_pcg<true>, &cfg) == cudaSuccess && nc >= 1;
  cudaGetLastError();
  known[dev] = a;
  return a;
}

}  // namespace

int adj_grid_blocks(const Dev& d) {
  const int want = ablk(std::max(std::max(d.n * 3, d.m), std::max(d.hg, d.D)));
  return std::max(1, std::min(want, std::min(adj_device().maxCtas, d.partStride)));
}

int adj_launch_pcg(const AdjArgs& a, int blocks, cudaStream_t s) {
  const AdjDevice dv = adj_device();
  AdjArgs c = a;
  if (blocks <= kAdjCluster && dv.cluster) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    adj_cluster_config(cfg, attr);
    cfg.stream = s;
    return (int)cudaLaunchKernelEx(&cfg, k_adj_pcg<true>, c, blocks);
  }
  void* args[] = {&c, &blocks};
  const int ctas = std::min(dv.maxCtas, std::max(blocks, dv.sms));
  return (int)cudaLaunchCooperativeKernel((void*)k_adj_pcg<false>, dim3(ctas), dim3(kThreads), args, 0, s);
}

void adj_theta(const Dev& d, const double* mu, double* terms, double* acc, cudaStream_t s) {
  const int stride = d.m + d.hg;
  k_adj_theta_terms<<<ablk(stride), kThreads, 0, s>>>(d, mu, terms, stride);
  k_adj_theta_sum<<<4, 1024, 0, s>>>(terms, stride, d.kb > 0 ? stride : d.m, acc);
}

void adj_propagate(const Dev& d, const double* mu, double* lamX, double* lamV, double damp, cudaStream_t s) {
  k_adj_propagate<<<ablk(d.n * 3), kThreads, 0, s>>>(d, mu, lamX, lamV, damp);
}

void adj_rhs(const Dev& d, const double* lamX, const double* lamV, double damp, double* rhs, cudaStream_t s) {
  k_adj_rhs<<<ablk(d.n * 3), kThreads, 0, s>>>(d, lamX, lamV, damp, rhs);
}

}  // namespace cs
