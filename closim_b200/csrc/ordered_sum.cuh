// Left-to-right sums of doubles, rounding for rounding, evaluated in parallel.
//
// The reference accumulates `for (i...) s += t[i]`; its rounded partial sums
// steer line searches and PCG iterations, so the FP64 path must reproduce them.
// One thread adding in order is bound by the latency of a dependent FP64 add
// (about 4 ns a term). This computes the same bits with all threads, from one
// property of round-to-nearest-even: while a partial sum stays inside one
// binade [2^e, 2^(e+1)), every addition rounds on the fixed grid ulp(e), so
// translating the start by an even number of ulps translates every later
// partial sum by the same amount. A chunk of terms therefore maps the bit
// pattern b of its start to b + d[b & 1], with the two increments d[0], d[1]
// found by adding the chunk from two neighbouring starts near an approximate
// one (a tree prefix sum). The map holds for every start of that binade that
// the chunk's path does not carry within reach of a power of two; the distance
// kept on the way is the window r it is published with. A chunk that crosses
// one power of two maps b by its residue mod 4 instead (four starts are added).
// Maps compose, so chunks merge into per-warp stages by a segmented scan, and
// one warp walks the stages with the exact running sum. A stage whose
// window does not hold the true start, or that no rule covers (several
// crossings, subnormal sums, infinities, NaN), is added term by term, so the
// result is the sequential sum's in every case.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace cs {

enum OrdType { ORD_AFFINE = 0, ORD_CROSS = 1, ORD_RAW = 2 };

struct __align__(16) OrdStage {
  long long B;      // base pattern the window is centred on
  long long R[4];   // affine: increments by parity in R[0], R[1]; cross: end pattern of start B + q
  int r;            // valid for starts within r ulps of B
  int type;
  int t0, t1;       // terms covered
  int sh;           // net binades climbed + 1, | 4 if the path goes above the start's, | 8 if below
  int count;        // first stage of a list: the list's length
};

__host__ __device__ __forceinline__ long long ord_bits(double x) {
#ifdef __CUDA_ARCH__
  return __double_as_longlong(x);
#else
  long long b;
  __builtin_memcpy(&b, &x, 8);
  return b;
#endif
}
__host__ __device__ __forceinline__ double ord_dbl(long long b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double(b);
#else
  double x;
  __builtin_memcpy(&x, &b, 8);
  return x;
#endif
}

constexpr long long kOrdM52 = (1ll << 52) - 1;
constexpr int kOrdRMax = 1 << 30;

// Distance (in ulps of b's binade) to the nearest power of two.
__host__ __device__ __forceinline__ long long ord_margin(long long b) {
  const long long f = b & kOrdM52, g = kOrdM52 + 1 - f;
  return f < g ? f : g;
}

// The map of one chunk of cnt terms t(0), t(1), ... for starts near `guess`.
// Fills B, R, r, type, sh. K > 0: cnt <= K with the loops unrolled (terms in
// registers); K = 0: any cnt.
template <int K, class F>
__host__ __device__ __forceinline__ void ord_chunk(const F& t, int cnt, double guess, OrdStage& s) {
  s.type = ORD_RAW;
  s.r = -1;
  s.sh = 1;
  s.B = ord_bits(guess);
  s.R[0] = s.R[1] = s.R[2] = s.R[3] = 0;
  const int lim = K > 0 ? K : cnt;
  const long long B = s.B & ~3ll;
  const int e = (int)((B >> 52) & 0x7ff);
  if (e < 64 || e > 0x7f0) return;
  s.B = B;
  double p0 = ord_dbl(B), p1 = ord_dbl(B | 1);
  long long m = ord_margin(B);
  bool cross = false;
#pragma unroll(K > 0 ? K : 1)
  for (int j = 0; j < lim; j++)
    if (j < cnt) {
      const double a = t(j);
      p0 = p0 + a;
      p1 = p1 + a;
      const long long b = ord_bits(p0), mm = ord_margin(b);
      m = mm < m ? mm : m;
      cross |= (b >> 52) != (B >> 52);
    }
  if (!cross) {
    const long long w = m - 8;  // the odd start's path stays within 2 ulps of the even one's
    if (w < 8) return;
    s.type = ORD_AFFINE;
    s.r = (int)(w < kOrdRMax ? w : kOrdRMax);
    s.R[0] = ord_bits(p0) - B;
    s.R[1] = ord_bits(p1) - (B | 1);
    return;
  }
  // Starts a multiple of 4 ulps apart stay an even number of ulps apart one
  // binade up and one down, so a path confined to those translates too.
  double q2 = ord_dbl(B | 2), q3 = ord_dbl(B | 3), q0 = ord_dbl(B);
  long long up = 0, down = 0;
#pragma unroll(K > 0 ? K : 1)
  for (int j = 0; j < lim; j++)
    if (j < cnt) {
      const double a = t(j);
      q0 = q0 + a;
      q2 = q2 + a;
      q3 = q3 + a;
      const long long de = (ord_bits(q0) >> 52) - (B >> 52);
      up = de > up ? de : up;
      down = de < down ? de : down;
    }
  const long long w = (m >> 1) - 32;
  if (up > 1 || down < -1 || w < 8) return;
  s.type = ORD_CROSS;
  s.r = (int)(w < kOrdRMax ? w : kOrdRMax);
  s.R[0] = ord_bits(p0);
  s.R[1] = ord_bits(p1);
  s.R[2] = ord_bits(q2);
  s.R[3] = ord_bits(q3);
  s.sh = (int)((s.R[0] >> 52) - (B >> 52)) + 1 + (up ? 4 : 0) + (down ? 8 : 0);
}

// Terms may come from other blocks of the same launch: read them from L2.
__host__ __device__ __forceinline__ double ord_load(const double* t) {
#ifdef __CUDA_ARCH__
  return __ldcg(t);
#else
  return *t;
#endif
}

// The stage applied to the exact running sum; terms it does not cover are added one by one.
__host__ __device__ __forceinline__ long long ord_raw(int t0, int t1, long long b, const double* t) {
  double p = ord_dbl(b);
  int j = t0;
  for (; j + 8 <= t1; j += 8) {  // the loads of eight terms in flight together
    double a[8];
#pragma unroll
    for (int q = 0; q < 8; q++) a[q] = ord_load(t + j + q);
#pragma unroll
    for (int q = 0; q < 8; q++) p = p + a[q];
  }
  for (; j < t1; j++) p = p + ord_load(t + j);
  return ord_bits(p);
}
__host__ __device__ __forceinline__ bool ord_covers(long long B, int r, long long b) {
  const long long dl = b - B;
  return dl >= -(long long)r && dl <= (long long)r;
}
// The map of a stage that covers b.
__host__ __device__ __forceinline__ long long ord_map(const OrdStage& s, long long b) {
  if (s.type == ORD_AFFINE) return b + ((b & 1) ? s.R[1] : s.R[0]);
  const long long dl = b - s.B;
  const int q = (int)(dl & 3);
  const long long k = dl - q;  // a multiple of 4
  const long long R = q == 0 ? s.R[0] : q == 1 ? s.R[1] : q == 2 ? s.R[2] : s.R[3];
  return R + ((k * 2) >> (s.sh & 3));
}
__host__ __device__ __forceinline__ long long ord_apply(const OrdStage& s, long long b, const double* t) {
  if (s.type == ORD_RAW || !ord_covers(s.B, s.r, b)) return ord_raw(s.t0, s.t1, b, t);
  return ord_map(s, b);
}

#ifdef __CUDACC__

__device__ __forceinline__ void ord_store(OrdStage* o, long long B, long long R0, long long R1, long long R2,
                                          long long R3, int r, int type, int t0, int t1, int sh, int count) {
  o->B = B;
  o->R[0] = R0; o->R[1] = R1; o->R[2] = R2; o->R[3] = R3;
  o->r = r; o->type = type; o->t0 = t0; o->t1 = t1; o->sh = sh; o->count = count;
}

// Terms t(j), j in [t0, t1), added to b in order by a warp: 32 loaded together,
// then handed round. (Past t1 zeros are added, which changes no sum but -0.0,
// and a sum that starts at +0.0 never becomes that.)
template <class F>
__device__ __forceinline__ long long ord_seq_warp(int t0, int t1, long long b, const F& t) {
  const int lane = threadIdx.x & 31;
  double p = ord_dbl(b);
  for (int j = t0; j < t1; j += 32) {
    const double a = j + lane < t1 ? t(j + lane) : 0.0;
    const int m = min(32, t1 - j);
#pragma unroll 1
    for (int u = 0; u < m; u += 8)
#pragma unroll
      for (int v = 0; v < 8; v++) p = p + __shfl_sync(0xffffffffu, a, u + v);
  }
  return ord_bits(p);
}
static __device__ __noinline__ long long ord_raw_warp(int t0, int t1, long long b, const double* T) {
  return ord_seq_warp(t0, t1, b, [&](int j) { return ord_load(T + j); });
}

// The published form of a known partial sum (of the segment that begins the sum).
__device__ __forceinline__ void ord_constant(OrdStage* out, long long b) {
  if ((threadIdx.x & 31) == 0) ord_store(out, ord_bits(0.0), b, b, b, b, 0, ORD_CROSS, 0, 0, 1, 1);
}

// The stages of a warp's 32 consecutive chunks (lane l: terms [t0, t0 + cnt) with
// approximate start `guess`), merged where neighbours are affine in one binade
// (at most `cap`, else one raw stage for the whole range).
template <int K, class F>
__device__ __forceinline__ void ord_warp_stages(const F& t, int t0, int cnt, double guess, OrdStage* out, int cap) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int lim = K > 0 ? K : cnt;
  OrdStage s;
  bool zero = true;
#pragma unroll(K > 0 ? K : 1)
  for (int j = 0; j < lim; j++) zero &= j >= cnt || t(j) == 0.0;
  if (__all_sync(full, zero)) {  // adding zeros changes no partial sum
    if (lane == 0) ord_store(out, ord_bits(guess) & ~3ll, 0, 0, 0, 0, kOrdRMax, ORD_AFFINE, 0, 0, 1, 1);
    return;
  }
  ord_chunk<K>(t, cnt, guess, s);
  const bool aff = s.type == ORD_AFFINE;
  const unsigned affs = __ballot_sync(full, aff);
  const int key = (int)(s.B >> 52);
  const int keyUp = __shfl_up_sync(full, key, 1);
  const bool head = lane == 0 || !aff || !((affs >> (lane - 1)) & 1u) || key != keyUp;
  const unsigned heads = __ballot_sync(full, head);
  const unsigned le = full >> (31 - lane);
  const int hl = 31 - __clz(heads & le);                            // first lane of my segment
  const unsigned above = heads & ~le;
  const int nx = above ? __ffs(above) - 1 : 32;                     // first lane after it
  const unsigned seg = (nx == 32 ? full : (1u << nx) - 1u) & ~((1u << hl) - 1u);
  long long d0 = s.R[0], d1 = s.R[1];
  bool f = head;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long a0 = __shfl_up_sync(full, d0, o), a1 = __shfl_up_sync(full, d1, o);
    const bool af = __shfl_up_sync(full, (int)f, o) != 0;
    if (lane >= o && !f) {
      const long long n0 = a0 + ((a0 & 1) ? d1 : d0), n1 = a1 + ((a1 & 1) ? d0 : d1);
      d0 = n0;
      d1 = n1;
      f = af;
    }
  }
  long long ex = __shfl_up_sync(full, d0, 1);
  if (head) ex = 0;
  const long long Bs = __shfl_sync(full, s.B, hl);
  const int ts = __shfl_sync(full, t0, hl);
  // how far this lane's base lies from where the segment's base would arrive
  long long c = Bs + ex - s.B;
  c = c < 0 ? -c : c;
  long long rr = (long long)s.r - 4 - c;
  rr = rr < -1 ? -1 : rr;
  const int rmin = __reduce_min_sync(seg, (int)rr);
  const int count = __popc(heads);
  const int t1 = t0 + cnt;
  if (count > cap) {
    const int tend = __shfl_sync(full, t1, 31), tbeg = __shfl_sync(full, t0, 0);
    if (lane == 0) ord_store(out, 0, 0, 0, 0, 0, 0, ORD_RAW, tbeg, tend, 1, 1);
    return;
  }
  if (lane == nx - 1) {
    OrdStage* o = out + __popc(heads & le) - 1;
    if (aff) ord_store(o, Bs, d0, d1, 0, 0, rmin, rmin < 0 ? ORD_RAW : ORD_AFFINE, ts, t1, 1, count);
    else ord_store(o, s.B, s.R[0], s.R[1], s.R[2], s.R[3], s.r, s.type, ts, t1, s.sh, count);
  }
}

// A list of stages that stays within one binade above and below its start's is
// itself a map by residue mod 4, valid where every stage's window is: lanes 0..3
// carry the four starts through it. out[0] then becomes that map.
static __device__ __noinline__ void ord_collapse(OrdStage* out) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int count = out[0].count, end = out[count - 1].t1;
  if (count == 1) return;
  const long long B = out[0].B & ~3ll;
  long long b = B + (lane & 3), w = kOrdRMax;
  int level = 0, flags = 0;
  bool ok = true;
  for (int j = 0; j < count; j++) {
    const OrdStage& s = out[j];
    long long c = b - s.B;
    c = c < 0 ? -c : c;
    const long long room = ((long long)s.r - c - 8) >> 1;
    w = room < w ? room : w;
    ok = ok && s.type != ORD_RAW && room >= 8;
    if (!ok) break;
    if (s.type == ORD_CROSS) {
      const int hi = level + ((s.sh & 4) ? 1 : 0), lo = level - ((s.sh & 8) ? 1 : 0);
      ok = hi <= 1 && lo >= -1;
      if (!ok) break;
      flags |= (hi > 0 ? 4 : 0) | (lo < 0 ? 8 : 0);
      level += (s.sh & 3) - 1;
    }
    b = ord_map(s, b);
  }
  const int wmin = __reduce_min_sync(full, (int)w);
  if (!__all_sync(full, ok)) return;
  const long long R0 = __shfl_sync(full, b, 0), R1 = __shfl_sync(full, b, 1), R2 = __shfl_sync(full, b, 2),
                  R3 = __shfl_sync(full, b, 3);
  const int t0 = out[0].t0;
  __syncwarp();
  if (lane == 0) ord_store(out, B, R0, R1, R2, R3, wmin, ORD_CROSS, t0, end, (level + 1) | flags, 1);
}

// A list's map for a walk in small integers: with the start written B + dl, the
// next list's start is nextB + dl', dl' = c[dl & 3] + the binade-scaled rest of
// dl. r < 0: the list is not one map, or its numbers are not small.
struct __align__(16) OrdStep {
  int c[4];
  int r, sh, pad[2];
};
__device__ __forceinline__ OrdStep ord_step(const OrdStage& s, long long nextB) {
  OrdStep o;
  o.sh = s.sh & 3;
  o.r = s.count == 1 && s.type != ORD_RAW && (s.B & 3) == 0 ? s.r : -1;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const long long e = (s.type == ORD_AFFINE ? s.B + q + s.R[q & 1] : s.R[q]) - nextB;
    if (e < -(1ll << 29) || e > (1ll << 29)) o.r = -1;
    o.c[q] = (int)e;
  }
  if (o.r > (1 << 28)) o.r = 1 << 28;
  return o;
}
// The base a walk uses behind the last list of its range.
__device__ __forceinline__ long long ord_after(const OrdStage& s) {
  return s.type == ORD_AFFINE ? s.B + s.R[0] : s.type == ORD_CROSS ? s.R[0] : s.B;
}

// The exact sum b carried through n lists by one warp: list i's first stage at
// w + i * stride (its others at more + i * moreStride), its step in st[i]. The
// dependent chain is five integer operations per list; the windows are checked
// eight lists at a time. Lists without a step, or whose window does not hold,
// are applied stage by stage.
static __device__ __noinline__ long long ord_walk(long long b, int n, const OrdStage* w, int stride,
                                                  const OrdStage* more, int moreStride, const OrdStep* st,
                                                  const double* T) {
  int i = 0;
  while (i < n) {
    const long long dl = b - w[(size_t)i * stride].B;
    int r = st[i].r;
    if (dl >= -(long long)r && dl <= (long long)r) {
      int d = (int)dl, stop = n;
      for (; i < stop;) {
        const int d0 = d;
        const int m = min(8, stop - i);
        bool ok = true;
#pragma unroll
        for (int u = 0; u < 8; u++)
          if (u < m) {
            const OrdStep& e = st[i + u];
            const int4 c = *reinterpret_cast<const int4*>(e.c);
            const int2 rs = *reinterpret_cast<const int2*>(&e.r);
            ok &= (unsigned)(d + rs.x) <= 2u * (unsigned)rs.x && rs.x >= 0;
            const int lo = (d & 1) ? c.y : c.x, hi = (d & 1) ? c.w : c.z;
            d = ((d & 2) ? hi : lo) + (((d & ~3) << 1) >> rs.y);
          }
        if (ok) {
          i += m;
          continue;
        }
        // find the list in these that is not covered: one by one up to it
        d = d0;
        while (i < stop) {
          const OrdStep& e = st[i];
          if (e.r < 0 || d < -e.r || d > e.r) {
            stop = i;
            break;
          }
          d = e.c[d & 3] + (((d & ~3) << 1) >> e.sh);
          i++;
        }
      }
      b = (i < n ? w[(size_t)i * stride].B : ord_after(w[(size_t)(n - 1) * stride])) + d;
      continue;
    }
    const OrdStage* s = w + (size_t)i * stride;
    const int count = s->count;
    for (int j = 0; j < count; j++) {
      if (s->type != ORD_RAW && ord_covers(s->B, s->r, b)) b = ord_map(*s, b);
      else b = ord_raw_warp(s->t0, s->t1, b, T);
      s = more + (size_t)i * moreStride + j + 1;
    }
    i++;
  }
  return b;
}

constexpr int kOrdK = 4;        // terms per lane and tile
constexpr int kOrdStages = 8;   // stages kept per warp and tile

template <int WARPS>
struct OrdSmem {
  OrdStage st[2][WARPS - 1][kOrdStages];
  OrdStep step[WARPS];
  double wsum[2][32];
};

// A sum of at most one term a thread, added by thread 0 from shared memory.
// Cycles of a block of 1,024 on a B200, this way / by stages: 129 terms 2,100 / 12,100, 512
// terms 5,200 / 12,100, 1,024 terms 9,700 / 12,400; by stages 2,048 terms take 13,300.
template <int WARPS>
__device__ __forceinline__ double block_short_sum(const double* t, int n) {
  __shared__ double buf[32 * WARPS];
  if ((int)threadIdx.x < n) buf[threadIdx.x] = t[threadIdx.x];
  __syncthreads();
  double p = 0.0;
  if (threadIdx.x == 0) {
    int j = 0;
    for (; j + 16 <= n; j += 16) {
      double a[16];
#pragma unroll
      for (int q = 0; q < 16; q++) a[q] = buf[j + q];
#pragma unroll
      for (int q = 0; q < 16; q++) p = p + a[q];
    }
    for (; j < n; j++) p = p + buf[j];
  }
  return p;
}

// 0.0 + t[0] + ... + t[n-1], left to right, by a block of 32 * WARPS threads
// (all of them call it; the sum is valid in thread 0). Warps 1.. turn tiles of
// terms into stages while warp 0 walks the previous tile's. The arithmetic
// is the sequential loop's bit for bit, which was bound by one dependent add per
// term; evaluating a 131 x 98 mesh's material (three sums of up to 63,000 terms
// among its kernels) went from 1.08 to 0.55 ms.
template <int WARPS>
__device__ __forceinline__ double block_ordered_sum(const double* t, int n, OrdSmem<WARPS>& sm) {
  constexpr int E = WARPS - 1;
  constexpr int kTile = E * 32 * kOrdK;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nTiles = (n + kTile - 1) / kTile;
  const int off = ((warp - 1) * 32 + lane) * kOrdK;
  double cur[kOrdK], nxt[kOrdK];
  auto load = [&](double (&d)[kOrdK], int tile) {
#pragma unroll
    for (int j = 0; j < kOrdK; j++) {
      const long i = (long)tile * kTile + off + j;
      d[j] = warp > 0 && i < n ? t[i] : 0.0;
    }
  };
  load(cur, 0);
  double approx = 0.0;           // approximate sum before the tile
  long long S = ord_bits(0.0);   // warp 0: exact sum before the walked tile
  for (int tile = 0; tile <= nTiles; tile++) {
    const int buf = tile & 1;
    double ex = 0.0;
    if (warp > 0 && tile < nTiles) {
      double s = 0.0;
#pragma unroll
      for (int j = 0; j < kOrdK; j++) s += cur[j];
      double inc = s;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double a = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += a;
      }
      ex = __shfl_up_sync(0xffffffffu, inc, 1);
      if (lane == 0) ex = 0.0;
      if (lane == 31) sm.wsum[buf][warp - 1] = inc;
    }
    __syncthreads();
    if (warp > 0 && tile < nTiles) {
      load(nxt, tile + 1);
      const double w = lane < E ? sm.wsum[buf][lane] : 0.0;
      double before = lane < warp - 1 ? w : 0.0, all = w;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        before += __shfl_xor_sync(0xffffffffu, before, o);
        all += __shfl_xor_sync(0xffffffffu, all, o);
      }
      const long i0 = (long)tile * kTile + off;
      const int t0 = (int)(i0 < n ? i0 : n);
      const int cnt = n - t0 < kOrdK ? n - t0 : kOrdK;
      if (tile == 0 && warp == 1) {
        ord_constant(sm.st[0][0], ord_raw_warp(0, min(n, 32 * kOrdK), ord_bits(0.0), t));
      } else {
        ord_warp_stages<kOrdK>([&](int j) { return cur[j]; }, t0, cnt, approx + before + ex, sm.st[buf][warp - 1],
                               kOrdStages);
        __syncwarp();
        ord_collapse(sm.st[buf][warp - 1]);
      }
      approx += all;
#pragma unroll
      for (int j = 0; j < kOrdK; j++) cur[j] = nxt[j];
    } else if (warp == 0 && tile > 0) {
      OrdStage* const w = sm.st[buf ^ 1][0];
      if (lane < E)
        sm.step[lane] = ord_step(w[lane * kOrdStages],
                                 lane + 1 < E ? w[(lane + 1) * kOrdStages].B : ord_after(w[lane * kOrdStages]));
      __syncwarp();
      S = ord_walk(S, E, w, kOrdStages, w, kOrdStages, sm.step, t);
    }
    __syncthreads();
  }
  return ord_dbl(S);
}

// The same by either way. SHORT (n <= 32 * WARPS, chosen at the launch) keeps the
// stages' code and shared memory out of the kernel. One call per kernel.
template <int WARPS, bool SHORT>
__device__ __forceinline__ double ordered_sum(const double* t, int n) {
  if constexpr (SHORT) return block_short_sum<WARPS>(t, n);
  __shared__ OrdSmem<WARPS> sm;
  return block_ordered_sum(t, n, sm);
}

#endif  // __CUDACC__

}  // namespace cs
