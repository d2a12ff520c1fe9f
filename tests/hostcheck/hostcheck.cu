// Test helper: host builds of the solver's device-side contact primitives
// (closim_b200/csrc/contact_math.cuh, jsmath.cuh), exported for CPU checks
// against the oracle. Built with -fmad=false like the FP64 device path.
#include "../../closim_b200/csrc/contact_math.cuh"
#include "../../closim_b200/csrc/adjoint_math.cuh"
#include "../../closim_b200/csrc/div_rn.cuh"
#include "../../closim_b200/csrc/ordered_sum.cuh"
#include "../../closim_b200/csrc/pcg64.cu"

template <bool SHORT>
__global__ void __launch_bounds__(1024) k_hc_ordered(const double* t, int n, double* o) {
  const double s = cs::ordered_sum<32, SHORT>(t, n);
  if (threadIdx.x == 0) *o = s;
}

extern "C" {
double hc_js_acos(double x) { return cs::js_acos(x); }
double hc_js_log(double x) { return cs::js_log(x); }
double hc_js_cbrt(double x) { return cs::js_cbrt(x); }
double hc_hypot3(double a, double b, double c) { return cs::js_hypot3(a, b, c); }
void hc_closest_vt(const double* q, double* o) {
  cs::Closest c = cs::closest_vt(q, q + 3, q + 6, q + 9);
  o[0] = c.s; o[1] = c.t; o[2] = c.dist; o[3] = c.rx; o[4] = c.ry; o[5] = c.rz;
}
void hc_closest_ee(const double* q, double* o) {
  cs::Closest c = cs::closest_ee(q, q + 3, q + 6, q + 9);
  o[0] = c.s; o[1] = c.t; o[2] = c.dist; o[3] = c.rx; o[4] = c.ry; o[5] = c.rz;
}
double hc_vt_ccd(const double* P0, const double* P1, double th) { return cs::vt_ccd(P0, P1, th); }
double hc_ee_ccd(const double* P0, const double* P1, double th) { return cs::ee_ccd(P0, P1, th); }
// The trial kernel's gated CCD: distance at P1 first, then trial_ccd.
double hc_trial_ccd(const double* P0, const double* P1, double th, int kind) {
  const double dT = kind == 0 ? cs::closest_vt(P1, P1 + 3, P1 + 6, P1 + 9).dist
                              : cs::closest_ee(P1, P1 + 3, P1 + 6, P1 + 9).dist;
  return cs::trial_ccd(kind, P0, P1, dT, th);
}
int hc_solve_cubic01(double a3, double a2, double a1, double a0, double* o) { return cs::solve_cubic01(a3, a2, a1, a0, o); }
double hc_barrier_value(double d, double dh) { return cs::barrier_value(d, dh); }
double hc_barrier_grad(double d, double dh, double k) { return cs::barrier_grad_scalar(d, dh, k, 1); }
double hc_barrier_curv(double d, double dh, double k) { return cs::barrier_curvature(d, dh, k); }
double hc_bend_grad(const double* q, const double* meta, double k, double* g) {
  return cs::bend_grad<double>(q, meta[0], meta[1], meta[2], k, g);
}
void hc_bend_hvp(const double* q, const double* v, const double* meta, double k, double* o) {
  cs::bend_hvp(q, v, meta[0], meta[1], meta[2], k, o);
}
void hc_membrane_block9(const double* x9, const double* inv4, double s, const double* C4, double* h) {
  cs::membrane_block9<double>(x9, x9 + 3, x9 + 6, inv4[0], inv4[1], inv4[2], inv4[3], s, C4[0], C4[1], C4[2], C4[3], h);
}
// Exact-Newton mode: the block with the stress's positive part, and the clamp itself.
void hc_membrane_block9_psd(const double* x9, const double* inv4, double s, const double* C4, double* h) {
  cs::membrane_block9<double>(x9, x9 + 3, x9 + 6, inv4[0], inv4[1], inv4[2], inv4[3], s, C4[0], C4[1], C4[2], C4[3], h,
                              true);
}
void hc_psd_stress(double* s3) { cs::psd_stress(s3[0], s3[1], s3[2]); }
// The chunk maps of the ordered sum (ordered_sum.cuh), walked chunk by chunk
// with starts guessed `rel` away from the true ones; covered = chunks whose map applied.
double hc_ordered_maps(const double* t, int n, double rel, int* covered) {
  long long b = cs::ord_bits(0.0);
  *covered = 0;
  for (int t0 = 0, c = 0; t0 < n; t0 += 4, c++) {
    double ch[4] = {0, 0, 0, 0};
    const int cnt = n - t0 < 4 ? n - t0 : 4;
    for (int j = 0; j < cnt; j++) ch[j] = t[t0 + j];
    cs::OrdStage s;
    cs::ord_chunk<4>([&](int j) { return ch[j]; }, cnt, cs::ord_dbl(b) * (1 + (c % 7 - 3) * rel), s);
    s.t0 = t0;
    s.t1 = t0 + cnt;
    const long long d = b - s.B;
    *covered += s.type != cs::ORD_RAW && d >= -(long long)s.r && d <= (long long)s.r;
    b = cs::ord_apply(s, b, t);
  }
  return cs::ord_dbl(b);
}
void hc_div_rn(const double* a, const double* b, int n, double* o) {
  for (int i = 0; i < n; i++) o[i] = cs::div_rn_divisor(b[i]) && cs::div_rn_dividend(a[i]) ? cs::div_rn_fast(a[i], b[i], 1.0 / b[i]) : NAN;
}
// Shared memory of the FP64 solve's launch for n vertices (no triangles) on a device
// with 148 SMs and clusters of 16; parts: 1 offsets, 2 vectors, 4 element results kept there.
int64_t hc_pcg64_smem(int n, int* parts) {
  cs::HostMesh me;
  me.n = n;
  me.memOff.assign((size_t)n + 1, 0u);
  cs::Pcg64Host h;
  cs::build_pcg64_plan(me, 148, 16, true, h);
  *parts = h.p.offSmem | (h.p.vecSmem << 1) | (h.p.elemSmem << 2);
  return (int64_t)h.p.smem;
}
// The block-wide ordered sum on the GPU; returns a cudaError_t.
int hc_gpu_ordered_sum(const double* t, int n, int brief, double* out) {
  double *dt = nullptr, *dout = nullptr;
  cudaError_t e = cudaMalloc(&dt, (size_t)(n > 0 ? n : 1) * 8);
  if (e == cudaSuccess) e = cudaMalloc(&dout, 8);
  if (e == cudaSuccess && n > 0) e = cudaMemcpy(dt, t, (size_t)n * 8, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    if (brief) k_hc_ordered<true><<<1, 1024>>>(dt, n, dout);
    else k_hc_ordered<false><<<1, 1024>>>(dt, n, dout);
    e = cudaMemcpy(out, dout, 8, cudaMemcpyDeviceToHost);
  }
  cudaFree(dt);
  cudaFree(dout);
  return (int)e;
}
}
