// Per-feature TimestepNorm and SequenceNorm with their backward, parallel over time (channels contiguous, any
// activation type).
//
// The running statistics are counts, means and squared deviations, which combine associatively, so the sequence
// is cut into segments: (1) the moments of every segment; (2) every segment combines those of the segments
// before it with the prior and walks its steps from there, with sums about the mean it starts from (they are
// as well conditioned as a step-by-step Welford update, and a step waits for nothing but two additions).
// The backward keeps no statistics of the forward: it takes the moments again.  With V = dL/dvar / n and
// U = dL/dmean / n at count n, the reverse recurrence is made of plain suffix sums (group_norm.cu):
//   b_t = -r^3 dy w (x - u) / (2 n),  a_t = -r dy w / n,  e_t = 2 (x - u_{t-1}) / n,
//   V_t = V + sum_{s >= t} b_s,  h_t = U + sum_{s > t} (a_s - e_s V_s) + a_t,  dx_t = dy r w + h_t + 2 (x - u) V_t,
// and a suffix is a total minus a prefix: one launch takes every segment's totals, the next walks forward in
// time from them.  A segment acts on (V, U) by an affine map, composed over the later segments.
// Bound: the issue slots, about 20 instructions per element and pass forward and 30 backward; HBM moves x twice
// and y once forward, x three times, dy twice and dx once backward.  B = 16, L = 4096, D = 1024, bf16: the
// walk of whole sequences (16384 chains of 4096 steps, statistics of every step saved in fp32) took 370 us
// forward and 365 us backward.  SequenceNorm needs the moments of the whole sequence only (B = 16, L = 1024, D = 256
// bf16: 403 us as one thread per column, its backward 99 us as one strided block per column).
#include <cmath>

#include "common.cuh"
#include "norm_run.cuh"
#include "scan_norm.cuh"
#include "scratch.cuh"
#include "walk.cuh"

namespace mega {

namespace {

struct SegNorm {
  ScanNormArgs a;
  int T, S;
  float* rn;               // [B][S] unmasked steps
  float *rm, *rs;          // [B][S][D] mean, squared deviations
  float *sv, *su, *sw;     // [B][S][D] backward: the segment's map
};

static MomentArgs moments_of(const SegNorm& s) {
  return {s.a.x, s.a.xsb, s.a.xsl, s.a.mask, s.a.L, s.a.D, s.T, s.S, s.rn, s.rm, s.rs};
}

struct NormLane {
  int lane, warp, d, dc, d0, left, b, seg, t0, t1;
  bool ok, active;
};
__device__ __forceinline__ NormLane norm_lane(const SegNorm& s) {
  NormLane l;
  l.lane = threadIdx.x & 31;
  l.warp = threadIdx.x >> 5;
  l.d0 = blockIdx.x * 32;
  l.left = s.a.D - l.d0;
  l.d = l.d0 + l.lane;
  l.ok = l.d < s.a.D;
  l.dc = l.ok ? l.d : s.a.D - 1;
  l.seg = blockIdx.y * kWarps + l.warp;
  l.b = blockIdx.z;
  l.active = l.seg < s.S;
  l.t0 = min(s.a.L, l.seg * s.T);
  l.t1 = min(s.a.L, l.t0 + s.T);
  return l;
}

// What a segment starts from: the prior and the segments before it.
__device__ __forceinline__ Run run_before(const SegNorm& s, const NormLane& l) {
  const float n0 = (float)s.a.prev_count[l.b];
  const size_t i = (size_t)l.b * s.a.D + l.dc;
  Run r{n0, s.a.prev_mean[i], s.a.prev_var[i] * n0};
  const float* pn = s.rn + (size_t)l.b * s.S;
  const float *pm = s.rm + (size_t)l.b * s.S * s.a.D + l.dc, *ps = s.rs + (size_t)l.b * s.S * s.a.D + l.dc;
#pragma unroll 4
  for (int k = 0; k < l.seg; ++k)
    r = combine(r, Run{__ldg(pn + k), __ldg(pm + (size_t)k * s.a.D), __ldg(ps + (size_t)k * s.a.D)});
  return r;
}

template <typename T, bool kMask>
__global__ void __launch_bounds__(kWarps * 32) norm_emit_kernel(SegNorm s) {
  extern __shared__ __align__(16) unsigned char rings[];
  const ScanNormArgs& a = s.a;
  const NormLane l = norm_lane(s);
  if (!l.active) return;
  const T* x = reinterpret_cast<const T*>(a.x) + l.b * a.xsb + l.d0;
  T* py = reinterpret_cast<T*>(a.y) + l.b * a.ysb + (long long)l.t0 * a.ysl + l.dc;
  const unsigned char* m = kMask ? a.mask + (size_t)l.b * a.L : nullptr;
  const float w = __ldg(a.gamma + l.dc), bb = __ldg(a.beta + l.dc), eps = a.eps;
  const Run in = run_before(s, l);
  Running st;
  st.start(in);
  walk<T, 1, false, kMask>(x, a.xsl, x, 0, m, l.t0, l.t1, l.left, rings + (size_t)l.warp * kRing * kTileBytes,
                           [&](int, float xv, float, bool pad) {
                             float out = 0.f;
                             if (!(kMask && pad)) {
                               float inv, r;
                               const float d = st.step(xv, eps, inv, r);
                               out = fmaf((d - st.u) * r, w, bb);
                             }
                             if (l.ok) Elem<T>::st(py, out);
                             py += a.ysl;
                           });
  if (l.seg == s.S - 1 && l.ok) {
    const size_t i = (size_t)l.b * a.D + l.d;
    const bool any = st.n > 0.f;
    const float inv = any ? 1.f / st.n : 0.f;
    a.mean_out[i] = any ? fmaf(st.s1, inv, st.c) : a.prev_mean[i];
    const float u = st.s1 * inv;
    a.var_out[i] = any ? fmaxf(fmaf(-u, u, (st.in_s + st.s2) * inv), 0.f) : a.prev_var[i];
    if (l.d == 0) a.count_out[l.b] = a.prev_count[l.b] + (long long)(st.n - (float)a.prev_count[l.b] + 0.5f);
  }
}

// The affine map of every segment, and the sums for dgamma and dbeta.
template <typename T, bool kMask>
__global__ void __launch_bounds__(kWarps * 32) norm_bwd_map_kernel(SegNorm s) {
  extern __shared__ __align__(16) unsigned char rings[];
  const ScanNormArgs& a = s.a;
  const NormLane l = norm_lane(s);
  float dg = 0.f, db = 0.f;
  if (l.active) {
    const T* x = reinterpret_cast<const T*>(a.x) + l.b * a.xsb + l.d0;
    const T* g = reinterpret_cast<const T*>(a.dy) + l.b * a.gsb + l.d0;
    const unsigned char* m = kMask ? a.mask + (size_t)l.b * a.L : nullptr;
    const float w = __ldg(a.gamma + l.dc), eps = a.eps;
    Running st;
    st.start(run_before(s, l));
    float sv = 0.f, su = 0.f, se = 0.f;
    walk<T, 1, true, kMask>(x, a.xsl, g, a.gsl, m, l.t0, l.t1, l.left, rings + (size_t)l.warp * 2 * kRing * kTileBytes,
                            [&](int, float xv, float gv, bool pad) {
                              if (kMask && pad) return;
                              const float up = st.u;
                              float inv, r;
                              const float d = st.step(xv, eps, inv, r);
                              const float xu = d - st.u, gr = gv * r, gx = gr * xu;
                              se = fmaf(2.f * (d - up), inv, se);
                              const float wi = w * inv;
                              const float b = -0.5f * (gx * (r * r)) * wi;
                              sv += b;
                              su -= fmaf(b, se, gr * wi);
                              dg += gx;
                              db += gv;
                            });
    if (l.ok) {
      const size_t i = ((size_t)l.b * s.S + l.seg) * a.D + l.d;
      s.sv[i] = sv;
      s.su[i] = su;
      s.sw[i] = -se;
    }
  }
  __syncthreads();
  float* red = reinterpret_cast<float*>(rings);   // [2][kWarps][32]
  red[l.warp * 32 + l.lane] = dg;
  red[(kWarps + l.warp) * 32 + l.lane] = db;
  __syncthreads();
  if (l.warp < 2 && l.ok) {
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < kWarps; ++k) v += red[(l.warp * kWarps + k) * 32 + l.lane];
    atomicAdd((l.warp == 0 ? a.dgamma : a.dbeta) + l.d, v);
  }
}

template <typename T, bool kMask>
__global__ void __launch_bounds__(kWarps * 32) norm_bwd_emit_kernel(SegNorm s) {
  extern __shared__ __align__(16) unsigned char rings[];
  const ScanNormArgs& a = s.a;
  const NormLane l = norm_lane(s);
  if (!l.active) return;
  const T* x = reinterpret_cast<const T*>(a.x) + l.b * a.xsb + l.d0;
  const T* g = reinterpret_cast<const T*>(a.dy) + l.b * a.gsb + l.d0;
  T* pd = reinterpret_cast<T*>(a.y) + l.b * a.ysb + (long long)l.t0 * a.ysl + l.dc;
  const unsigned char* m = kMask ? a.mask + (size_t)l.b * a.L : nullptr;
  const float w = __ldg(a.gamma + l.dc), eps = a.eps;
  const size_t row = (size_t)l.b * a.D + l.dc;
  const float n0 = (float)a.prev_count[l.b];
  float n_end = n0;
  for (int k = 0; k < s.S; ++k) n_end += __ldg(s.rn + (size_t)l.b * s.S + k);
  const float inv_end = n_end > 0.f ? 1.f / n_end : 0.f;
  float V = a.dvar ? a.dvar[row] * inv_end : 0.f, U = a.dmean ? a.dmean[row] * inv_end : 0.f;
  const size_t at = (size_t)l.b * s.S * a.D + l.dc;
#pragma unroll 4
  for (int k = s.S - 1; k > l.seg; --k) {
    const size_t i = at + (size_t)k * a.D;
    U = fmaf(__ldg(s.sw + i), V, U + __ldg(s.su + i));
    V += __ldg(s.sv + i);
  }
  const size_t own = at + (size_t)l.seg * a.D;
  float W = fmaf(__ldg(s.sw + own), V, U + __ldg(s.su + own));   // U as it leaves the segment's first step
  V += __ldg(s.sv + own);
  if (l.seg == 0 && l.ok) {
    const bool any = n_end > n0;   // (no unmasked step: the incoming gradients pass through)
    a.dprev_mean[row] = any ? n0 * W : (a.dmean ? a.dmean[row] : 0.f);
    a.dprev_var[row] = any ? n0 * V : (a.dvar ? a.dvar[row] : 0.f);
  }
  Running st;
  st.start(run_before(s, l));
  walk<T, 1, true, kMask>(x, a.xsl, g, a.gsl, m, l.t0, l.t1, l.left, rings + (size_t)l.warp * 2 * kRing * kTileBytes,
                          [&](int, float xv, float gv, bool pad) {
                            float out = 0.f;
                            if (!(kMask && pad)) {
                              const float up = st.u;
                              float inv, r;
                              const float d = st.step(xv, eps, inv, r);
                              const float xu = d - st.u, gr = gv * r, gx = gr * xu, wi = w * inv;
                              const float b = -0.5f * (gx * (r * r)) * wi;
                              const float ev = 2.f * (d - up) * inv * V;
                              const float h = W + ev;
                              out = fmaf(gr, w, fmaf(2.f * xu, V, h));
                              W = fmaf(gr, wi, h);   // W - (a - e V) with a = -gr wi
                              V -= b;
                            }
                            if (l.ok) Elem<T>::st(pd, out);
                            pd += a.ysl;
                          });
}

// ---- SequenceNorm, per channel -----------------------------------------------------------------
// The moments of the whole sequence: those of every segment (norm_moments_kernel), combined by each block.
template <typename T, bool kMask>
__global__ void __launch_bounds__(kWarps * 32) sqn_emit_kernel(SegNorm s) {
  extern __shared__ __align__(16) unsigned char rings[];
  const ScanNormArgs& a = s.a;
  const NormLane l = norm_lane(s);
  if (!l.active) return;
  Run r{0.f, 0.f, 0.f};
  const float* pn = s.rn + (size_t)l.b * s.S;
  const float *pm = s.rm + (size_t)l.b * s.S * a.D + l.dc, *ps = s.rs + (size_t)l.b * s.S * a.D + l.dc;
#pragma unroll 4
  for (int k = 0; k < s.S; ++k) r = combine(r, Run{__ldg(pn + k), __ldg(pm + (size_t)k * a.D), __ldg(ps + (size_t)k * a.D)});
  const float rstd = rsqrtf((r.n > 0.f ? r.s / r.n : 0.f) + a.eps), mean = r.m;
  if (l.seg == 0 && l.ok) {
    a.mean_out[(size_t)l.b * a.D + l.d] = mean;
    a.var_out[(size_t)l.b * a.D + l.d] = rstd;
    if (l.d == 0) a.count_out[l.b] = (long long)(r.n + 0.5f);
  }
  const T* x = reinterpret_cast<const T*>(a.x) + l.b * a.xsb + l.d0;
  T* py = reinterpret_cast<T*>(a.y) + l.b * a.ysb + (long long)l.t0 * a.ysl + l.dc;
  const unsigned char* m = kMask ? a.mask + (size_t)l.b * a.L : nullptr;
  const float w = __ldg(a.gamma + l.dc), bb = __ldg(a.beta + l.dc);
  walk<T, 1, false, kMask>(x, a.xsl, x, 0, m, l.t0, l.t1, l.left, rings + (size_t)l.warp * kRing * kTileBytes,
                           [&](int, float xv, float, bool pad) {
                             if (l.ok) Elem<T>::st(py, kMask && pad ? 0.f : fmaf((xv - mean) * rstd, w, bb));
                             py += a.ysl;
                           });
}

// Backward: every segment's sums of dy and dy (x - mean) ...
template <typename T, bool kMask>
__global__ void __launch_bounds__(kWarps * 32) sqn_bwd_sums_kernel(SegNorm s) {
  extern __shared__ __align__(16) unsigned char rings[];
  const ScanNormArgs& a = s.a;
  const NormLane l = norm_lane(s);
  if (!l.active) return;
  const T* x = reinterpret_cast<const T*>(a.x) + l.b * a.xsb + l.d0;
  const T* g = reinterpret_cast<const T*>(a.dy) + l.b * a.gsb + l.d0;
  const unsigned char* m = kMask ? a.mask + (size_t)l.b * a.L : nullptr;
  const float u = a.prev_mean[(size_t)l.b * a.D + l.dc];
  float ds = 0.f, db = 0.f;
  walk<T, 1, true, kMask>(x, a.xsl, g, a.gsl, m, l.t0, l.t1, l.left, rings + (size_t)l.warp * 2 * kRing * kTileBytes,
                          [&](int, float xv, float gv, bool pad) {
                            const float v = kMask && pad ? 0.f : gv;
                            ds = fmaf(v, xv - u, ds);
                            db += v;
                          });
  if (l.ok) {
    const size_t i = ((size_t)l.b * s.S + l.seg) * a.D + l.d;
    s.rm[i] = ds;
    s.rs[i] = db;
  }
}

// ... and the input gradient from their totals (fairseq/csrc/ops/sequence_norm.cc:374-529).
template <typename T, bool kMask>
__global__ void __launch_bounds__(kWarps * 32) sqn_bwd_emit_kernel(SegNorm s) {
  extern __shared__ __align__(16) unsigned char rings[];
  const ScanNormArgs& a = s.a;
  const NormLane l = norm_lane(s);
  if (!l.active) return;
  const float *pm = s.rm + (size_t)l.b * s.S * a.D + l.dc, *ps = s.rs + (size_t)l.b * s.S * a.D + l.dc;
  float ds = 0.f, db = 0.f;
#pragma unroll 4
  for (int k = 0; k < s.S; ++k) {
    ds += __ldg(pm + (size_t)k * a.D);
    db += __ldg(ps + (size_t)k * a.D);
  }
  const size_t row = (size_t)l.b * a.D + l.dc;
  const float u = a.prev_mean[row], r = a.prev_var[row], w = __ldg(a.gamma + l.dc);   // (mean and rstd of the forward)
  const long long cnt = a.prev_count[l.b];
  const float coef = cnt > 0 ? 1.f / (float)cnt : 0.f;
  if (l.seg == 0 && l.ok) {
    atomicAdd(a.dgamma + l.d, r * ds);
    atomicAdd(a.dbeta + l.d, db);
  }
  const float rw = r * w, kv = -coef * (r * r * rw) * ds, ku = -coef * rw * db;
  const T* x = reinterpret_cast<const T*>(a.x) + l.b * a.xsb + l.d0;
  const T* g = reinterpret_cast<const T*>(a.dy) + l.b * a.gsb + l.d0;
  T* pd = reinterpret_cast<T*>(a.y) + l.b * a.ysb + (long long)l.t0 * a.ysl + l.dc;
  const unsigned char* m = kMask ? a.mask + (size_t)l.b * a.L : nullptr;
  walk<T, 1, true, kMask>(x, a.xsl, g, a.gsl, m, l.t0, l.t1, l.left, rings + (size_t)l.warp * 2 * kRing * kTileBytes,
                          [&](int, float xv, float gv, bool pad) {
                            if (l.ok) Elem<T>::st(pd, kMask && pad ? 0.f : fmaf(rw, gv, fmaf(kv, xv - u, ku)));
                            pd += a.ysl;
                          });
}

// Segments: enough blocks of four for the SMs (about six of them resident each) in few rounds, at least 64 steps
// each and at most 64 of them, since every segment combines those before it.
static void pick_segments(const ScanNormArgs& a, int resident, SegNorm& s) {
  const long long strips = (long long)((a.D + 31) / 32) * a.B;
  const double slots = 148.0 * resident;
  double best = 1e30;
  for (int S = 1; S <= 64; ++S) {
    int t = ((a.L + S - 1) / S + kU - 1) / kU * kU;
    if (t < 64) t = 64;
    const int n = (a.L + t - 1) / t;
    const double cost = ceil(strips * ((n + kWarps - 1) / kWarps) / slots) * (t + 32 + n);
    if (cost < best) {
      best = cost;
      s.T = t;
      s.S = n;
    }
    if (t == 64) break;
  }
}

template <typename T, bool kMask>
static void fwd_launch(const SegNorm& s, cudaStream_t st) {
  const dim3 grid((s.a.D + 31) / 32, (s.S + kWarps - 1) / kWarps, s.a.B), block(kWarps * 32);
  const size_t rings = (size_t)kWarps * kRing * kTileBytes;
  launch(norm_moments_kernel<T, kMask>, grid, block, rings, (void*)st, moments_of(s));
  launch(norm_emit_kernel<T, kMask>, grid, block, rings, (void*)st, s);
}
template <typename T, bool kMask>
static void bwd_launch(const SegNorm& s, cudaStream_t st) {
  const dim3 grid((s.a.D + 31) / 32, (s.S + kWarps - 1) / kWarps, s.a.B), block(kWarps * 32);
  const size_t rings = (size_t)kWarps * kRing * kTileBytes;
  launch(norm_moments_kernel<T, kMask>, grid, block, rings, (void*)st, moments_of(s));
  launch(norm_bwd_map_kernel<T, kMask>, grid, block, 2 * rings, (void*)st, s);
  launch(norm_bwd_emit_kernel<T, kMask>, grid, block, 2 * rings, (void*)st, s);
}

template <typename T, bool kMask>
static void sqn_launch(const SegNorm& s, bool bwd, cudaStream_t st) {
  const dim3 grid((s.a.D + 31) / 32, (s.S + kWarps - 1) / kWarps, s.a.B), block(kWarps * 32);
  const size_t rings = (size_t)kWarps * kRing * kTileBytes;
  if (bwd) {
    launch(sqn_bwd_sums_kernel<T, kMask>, grid, block, 2 * rings, (void*)st, s);
    launch(sqn_bwd_emit_kernel<T, kMask>, grid, block, 2 * rings, (void*)st, s);
  } else {
    launch(norm_moments_kernel<T, kMask>, grid, block, rings, (void*)st, moments_of(s));
    launch(sqn_emit_kernel<T, kMask>, grid, block, rings, (void*)st, s);
  }
}

static bool sqn_dispatch(int dtype, const ScanNormArgs& a, bool bwd, cudaStream_t st) {
  if (g_options[OPT_DISABLE_STREAM].load() != 0 || a.B > 65535) return false;
  SegNorm s{};
  s.a = a;
  pick_segments(a, bwd ? 3 : 6, s);
  const size_t n = (size_t)a.B * s.S * a.D;
  Scratch sc(Scratch::padded(n * 4) * 2 + Scratch::padded((size_t)a.B * s.S * 4), st);
  if (!sc) return false;
  s.rn = sc.take<float>((size_t)a.B * s.S);
  s.rm = sc.take<float>(n);
  s.rs = sc.take<float>(n);
#define MEGA_SCAN_SQN(TY)                          \
  if (a.mask) sqn_launch<TY, true>(s, bwd, st);    \
  else sqn_launch<TY, false>(s, bwd, st);          \
  return true
  switch (dtype) {
    case MEGA_F32: MEGA_SCAN_SQN(float);
    case MEGA_BF16: MEGA_SCAN_SQN(__nv_bfloat16);
    case MEGA_F16: MEGA_SCAN_SQN(__half);
    default: return false;
  }
#undef MEGA_SCAN_SQN
}

template <bool kBwd>
static bool dispatch(int dtype, const ScanNormArgs& a, cudaStream_t st) {
  if (g_options[OPT_DISABLE_STREAM].load() != 0 || a.B > 65535) return false;
  SegNorm s{};
  s.a = a;
  pick_segments(a, kBwd ? 3 : 6, s);
  const size_t n = (size_t)a.B * s.S * a.D;
  Scratch sc(Scratch::padded(n * 4) * (kBwd ? 5 : 2) + Scratch::padded((size_t)a.B * s.S * 4), st);
  if (!sc) return false;
  s.rn = sc.take<float>((size_t)a.B * s.S);
  s.rm = sc.take<float>(n);
  s.rs = sc.take<float>(n);
  if (kBwd) {
    s.sv = sc.take<float>(n);
    s.su = sc.take<float>(n);
    s.sw = sc.take<float>(n);
  }
#define MEGA_SCAN_NORM(TY)                                                        \
  if (kBwd) {                                                                     \
    if (a.mask) bwd_launch<TY, true>(s, st);                                      \
    else bwd_launch<TY, false>(s, st);                                            \
  } else {                                                                        \
    if (a.mask) fwd_launch<TY, true>(s, st);                                      \
    else fwd_launch<TY, false>(s, st);                                            \
  }                                                                               \
  return true
  switch (dtype) {
    case MEGA_F32: MEGA_SCAN_NORM(float);
    case MEGA_BF16: MEGA_SCAN_NORM(__nv_bfloat16);
    case MEGA_F16: MEGA_SCAN_NORM(__half);
    default: return false;
  }
#undef MEGA_SCAN_NORM
}

}  // namespace

bool scan_norm_fwd_try(int dtype, const ScanNormArgs& a, long long xsd, long long ysd, cudaStream_t s) {
  if (!rows_ok(dtype, a.x, a.xsb, a.xsl, xsd, a.D) || ysd != 1 || a.x == a.y) return false;
  return dispatch<false>(dtype, a, s);
}

bool scan_norm_bwd_try(int dtype, const ScanNormArgs& a, long long xsd, long long ysd, long long gsd, cudaStream_t s) {
  if (!rows_ok(dtype, a.x, a.xsb, a.xsl, xsd, a.D) || !rows_ok(dtype, a.dy, a.gsb, a.gsl, gsd, a.D) || ysd != 1 ||
      a.y == a.x || a.y == a.dy)
    return false;
  return dispatch<true>(dtype, a, s);
}

bool scan_sqn_fwd_try(int dtype, const ScanNormArgs& a, long long xsd, long long ysd, cudaStream_t s) {
  if (!rows_ok(dtype, a.x, a.xsb, a.xsl, xsd, a.D) || ysd != 1) return false;
  return sqn_dispatch(dtype, a, false, s);
}

bool scan_sqn_bwd_try(int dtype, const ScanNormArgs& a, long long xsd, long long ysd, long long gsd, cudaStream_t s) {
  if (!rows_ok(dtype, a.x, a.xsb, a.xsl, xsd, a.D) || !rows_ok(dtype, a.dy, a.gsb, a.gsl, gsd, a.D) || ysd != 1 ||
      a.y == a.x || a.y == a.dy)
    return false;
  return sqn_dispatch(dtype, a, true, s);
}

}  // namespace mega
