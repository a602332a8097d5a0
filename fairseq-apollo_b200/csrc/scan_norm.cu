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
// Bound: the issue slots and memory alike; a lane takes two channels in packed arithmetic (one channel per lane: 74 us
// forward behind the moments, 109 and 129 us backward, at B = 16, L = 4096, D = 1024 bf16; in pairs 64, 104 and 106).
// HBM moves x twice and y once forward, x three times, dy twice and dx once backward.  B = 16, L = 4096, D = 1024, bf16: the
// walk of whole sequences (16384 chains of 4096 steps, statistics of every step saved in fp32) took 370 us
// forward and 365 us backward.  SequenceNorm needs the moments of the whole sequence only (B = 16, L = 1024, D = 256
// bf16: 403 us as one thread per column, its backward 99 us as one strided block per column).
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "norm_run.cuh"
#include "scan_norm.cuh"
#include "scratch.cuh"
#include "walk.cuh"

namespace mega {

namespace {

// Tiles in flight of the walks that read x and dy: with three of a 16-bit type a fourth block fits an SM (16 x 4096 x 1024 bf16 with
// the moments 230 us -> 226, 32 x 2048 x 512 136 -> 128); in fp32, at the rate of memory, four (285 us, three 304).
template <typename T>
constexpr int kRingTwo = sizeof(T) == 4 ? kRing : 3;

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

// ---- two channels per lane ----------------------------------------------------------------------
struct PairLane {
  int lane, warp, d, dc, d0, left, b, seg, t0, t1;   // d: first of the lane's two channels
  bool ok, active;
};
__device__ __forceinline__ PairLane pair_lane(const SegNorm& s) {
  PairLane l;
  l.lane = threadIdx.x & 31;
  l.warp = threadIdx.x >> 5;
  l.d0 = blockIdx.x * 64;
  l.left = s.a.D - l.d0;
  l.d = l.d0 + 2 * l.lane;
  l.ok = l.d < s.a.D;   // (rows are whole 16-byte pieces: channels come in pairs)
  l.dc = l.ok ? l.d : s.a.D - 2;
  l.seg = blockIdx.y * kWarps + l.warp;
  l.b = blockIdx.z;
  l.active = l.seg < s.S;
  l.t0 = min(s.a.L, l.seg * s.T);
  l.t1 = min(s.a.L, l.t0 + s.T);
  return l;
}
__device__ __forceinline__ f32x2 ldg2(const float* p) { return pack2(__ldg(p), __ldg(p + 1)); }
__device__ __forceinline__ f32x2 both(float v) { return pack2(v, v); }

// What a segment starts from: the prior and the segments before it (for two channels).
__device__ __forceinline__ void pair_before(const SegNorm& s, const PairLane& l, Run (&r)[2]) {
  const float n0 = (float)s.a.prev_count[l.b];
  float seen = 0.f;   // (unmasked steps of the call: a float count that starts beyond 2^24 would round them)
  const size_t i = (size_t)l.b * s.a.D + l.dc;
  const float* pn = s.rn + (size_t)l.b * s.S;
  const size_t at = (size_t)l.b * s.S * s.a.D + l.dc;
#pragma unroll
  for (int c = 0; c < 2; ++c) r[c] = Run{n0, s.a.prev_mean[i + c], s.a.prev_var[i + c] * n0};
  auto add = [&](float n, float2 m, float2 q) {
    r[0] = combine(r[0], Run{n, m.x, q.x});
    r[1] = combine(r[1], Run{n, m.y, q.y});
    seen += n;
  };
  auto mean = [&](int k) { return __ldg(reinterpret_cast<const float2*>(s.rm + at + (size_t)k * s.a.D)); };
  auto dev2 = [&](int k) { return __ldg(reinterpret_cast<const float2*>(s.rs + at + (size_t)k * s.a.D)); };
  // (eight at a time: between the branches of the combinations each load waits for its own, 2 x 5565 x 32 backward 57 us, so 46)
  int k = 0;
  auto batches = [&](auto size) {
    constexpr int kB = decltype(size)::value;
    for (; k + kB <= l.seg; k += kB) {
      float n[kB];
      float2 m[kB], q[kB];
#pragma unroll
      for (int u = 0; u < kB; ++u) {
        n[u] = __ldg(pn + k + u);
        m[u] = mean(k + u);
        q[u] = dev2(k + u);
      }
#pragma unroll
      for (int u = 0; u < kB; ++u) add(n[u], m[u], q[u]);
    }
  };
  batches(std::integral_constant<int, 8>{});
  batches(std::integral_constant<int, 3>{});
  batches(std::integral_constant<int, 1>{});
  r[0].n = r[1].n = n0 + seen;
}

// Running (norm_run.cuh) for two channels.  Its walks are bound by the FMA pipe, in which a packed instruction takes two cycles: so
// no sign is turned in packed arithmetic, and what all steps of a walk share is a factor of its sums.  (16 x 4096 x 1024 bf16,
// with 26, 23 and 11 packed instructions a step the map 103 us, the gradients 113, the outputs 67; with 18, 19 and 9
// 88, 98 and 63.)
struct PairRunning {
  f32x2 c, s1, s2, in_s, u, eps2;
  float n0, seen, n, eps;
  // x: the segment's first step of the lane's channels (one that counts is the centre where nothing came in)
  template <typename T>
  __device__ __forceinline__ void start(const Run (&r)[2], float e, const T* x, long long xsl, const unsigned char* m, int t0, int t1) {
    c = pack2(r[0].m, r[1].m);
    s1 = s2 = u = both(0.f);
    n0 = n = r[0].n;
    seen = 0.f;
    in_s = pack2(r[0].s, r[1].s);
    eps = e;
    eps2 = both(e);
    if (n0 == 0.f) {
      int t = t0;
      while (m && t < t1 && m[t]) ++t;
      if (t < t1) c = pack2(Elem<T>::ld(x + t * xsl), Elem<T>::ld(x + t * xsl + 1));
    }
  }
  // returns x - c; inv = 1 / n, r = 1 / sqrt(var + eps)
  __device__ __forceinline__ f32x2 step(f32x2 x, f32x2& inv, f32x2& r) {
    const f32x2 d = sub2(x, c);
    s1 = add2(s1, d);
    s2 = fma2(d, d, s2);
    seen += 1.f;
    n = n0 + seen;
    inv = both(rcp_approx(n));
    u = mul2(s1, inv);
    const f32x2 q = fma2(add2(in_s, s2), inv, eps2);
    float a, b, ua, ub;
    unpack2(q, a, b);
    unpack2(u, ua, ub);
    r = pack2(rsqrt_approx(fmaxf(fmaf(-ua, ua, a), eps)), rsqrt_approx(fmaxf(fmaf(-ub, ub, b), eps)));
    return d;
  }
};

// kWide: the output in fp32 for what follows on it, beside that of type T or in its place.
template <typename T, bool kMask, bool kWide>
__global__ void __launch_bounds__(kWarps * 32) norm_emit_kernel(SegNorm s) {
  extern __shared__ __align__(16) unsigned char rings[];
  const ScanNormArgs& a = s.a;
  const PairLane l = pair_lane(s);
  if (!l.active) return;
  const T* x = reinterpret_cast<const T*>(a.x) + l.b * a.xsb + l.d0;
  const bool own = !kWide || a.y != nullptr;
  T* py = own ? reinterpret_cast<T*>(a.y) + l.b * a.ysb + (long long)l.t0 * a.ysl + l.dc : nullptr;
  float* pw = kWide ? a.wide + ((size_t)l.b * a.L + l.t0) * a.D + l.dc : nullptr;
  const unsigned char* m = kMask ? a.mask + (size_t)l.b * a.L : nullptr;
  const f32x2 w = ldg2(a.gamma + l.dc), bb = ldg2(a.beta + l.dc);
  Run in[2];
  pair_before(s, l, in);
  PairRunning st;
  st.start(in, a.eps, x + (l.dc - l.d0), a.xsl, m, l.t0, l.t1);
  walk_pairs<T, false, kMask>(x, a.xsl, x, 0, m, l.t0, l.t1, l.left, rings + (size_t)l.warp * kRing * kTileBytes,
                              [&](f32x2 xv, f32x2, bool pad) {
                                f32x2 out = both(0.f);
                                if (!(kMask && pad)) {
                                  f32x2 inv, r;
                                  const f32x2 d = st.step(xv, inv, r);
                                  out = fma2(mul2(sub2(d, st.u), r), w, bb);
                                }
                                if (kWide) {
                                  if (l.ok) *reinterpret_cast<f32x2*>(pw) = out;
                                  pw += a.D;
                                }
                                if (own) {
                                  if (l.ok) pair_st(py, out);
                                  py += a.ysl;
                                }
                              });
  if (l.seg == s.S - 1 && l.ok) {
    const bool any = st.n > 0.f;
    const float inv = any ? 1.f / st.n : 0.f;
    float c[2], s1[2], s2[2], q[2];
    unpack2(st.c, c[0], c[1]);
    unpack2(st.s1, s1[0], s1[1]);
    unpack2(st.s2, s2[0], s2[1]);
    unpack2(st.in_s, q[0], q[1]);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const size_t i = (size_t)l.b * a.D + l.d + k;
      const float u = s1[k] * inv;
      a.mean_out[i] = any ? c[k] + u : a.prev_mean[i];
      a.var_out[i] = any ? not_negative(fmaf(-u, u, (q[k] + s2[k]) * inv)) : a.prev_var[i];
    }
    if (l.d == 0) {
      long long total = a.prev_count[l.b];
      for (int k = 0; k < s.S; ++k) total += (long long)__ldg(s.rn + (size_t)l.b * s.S + k);
      a.count_out[l.b] = total;
    }
  }
}

// The affine map of every segment, and the sums for dgamma and dbeta.
template <typename T, bool kMask>
__global__ void __launch_bounds__(kWarps * 32) norm_bwd_map_kernel(SegNorm s) {
  extern __shared__ __align__(16) unsigned char rings[];
  const ScanNormArgs& a = s.a;
  const PairLane l = pair_lane(s);
  f32x2 dg = both(0.f), db = both(0.f);
  if (l.active) {
    const T* x = reinterpret_cast<const T*>(a.x) + l.b * a.xsb + l.d0;
    const T* g = reinterpret_cast<const T*>(a.dy) + l.b * a.gsb + l.d0;
    const unsigned char* m = kMask ? a.mask + (size_t)l.b * a.L : nullptr;
    const f32x2 w = ldg2(a.gamma + l.dc);
    Run in[2];
    pair_before(s, l, in);
    PairRunning st;
    st.start(in, a.eps, x + (l.dc - l.d0), a.xsl, m, l.t0, l.t1);
    // sums whose factors -w / 2 (sv), w (su) and 2 (se) follow; se with its sign turned
    f32x2 sv = both(0.f), su = sv, se = sv;
    walk_pairs<T, true, kMask, kRingTwo<T>>(x, a.xsl, g, a.gsl, m, l.t0, l.t1, l.left, rings + (size_t)l.warp * 2 * kRingTwo<T> * kTileBytes,
                               [&](f32x2 xv, f32x2 gv, bool pad) {
                                 if (kMask && pad) return;
                                 const f32x2 up = st.u;
                                 f32x2 inv, r;
                                 const f32x2 d = st.step(xv, inv, r);
                                 const f32x2 gr = mul2(gv, r), gx = mul2(gr, sub2(d, st.u)), b = mul2(gx, mul2(r, r));
                                 se = fma2(sub2(up, d), inv, se);
                                 sv = fma2(b, inv, sv);
                                 su = fma2(fma2(b, se, gr), inv, su);
                                 dg = add2(dg, gx);
                                 db = add2(db, gv);
                               });
    if (l.ok) {
      const size_t i = ((size_t)l.b * s.S + l.seg) * a.D + l.d;
      *reinterpret_cast<f32x2*>(s.sv + i) = mul2(sv, mul2(w, both(-0.5f)));
      *reinterpret_cast<f32x2*>(s.su + i) = mul2(su, mul2(w, both(-1.f)));
      *reinterpret_cast<f32x2*>(s.sw + i) = add2(se, se);
    }
  }
  __syncthreads();
  float* red = reinterpret_cast<float*>(rings);   // [2][kWarps][64]
  *reinterpret_cast<f32x2*>(red + l.warp * 64 + 2 * l.lane) = dg;
  *reinterpret_cast<f32x2*>(red + (kWarps + l.warp) * 64 + 2 * l.lane) = db;
  __syncthreads();
  const int c = threadIdx.x & 63, which = threadIdx.x >> 6;   // (128 threads: the 64 channels of either sum)
  if (l.d0 + c < a.D) {
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < kWarps; ++k) v += red[(which * kWarps + k) * 64 + c];
    atomicAdd((which == 0 ? a.dgamma : a.dbeta) + l.d0 + c, v);
  }
}

template <typename T, bool kMask>
__global__ void __launch_bounds__(kWarps * 32) norm_bwd_emit_kernel(SegNorm s) {
  extern __shared__ __align__(16) unsigned char rings[];
  const ScanNormArgs& a = s.a;
  const PairLane l = pair_lane(s);
  if (!l.active) return;
  const T* x = reinterpret_cast<const T*>(a.x) + l.b * a.xsb + l.d0;
  const T* g = reinterpret_cast<const T*>(a.dy) + l.b * a.gsb + l.d0;
  T* pd = reinterpret_cast<T*>(a.y) + l.b * a.ysb + (long long)l.t0 * a.ysl + l.dc;
  const unsigned char* m = kMask ? a.mask + (size_t)l.b * a.L : nullptr;
  const f32x2 w = ldg2(a.gamma + l.dc);
  const size_t row = (size_t)l.b * a.D + l.dc;
  const float n0 = (float)a.prev_count[l.b];
  float total = 0.f;   // unmasked steps of the call
  for (int k = 0; k < s.S; ++k) total += __ldg(s.rn + (size_t)l.b * s.S + k);
  const float n_end = n0 + total;
  const f32x2 inv_end = both(n_end > 0.f ? 1.f / n_end : 0.f);
  f32x2 V = a.dvar ? mul2(pack2(a.dvar[row], a.dvar[row + 1]), inv_end) : both(0.f);
  f32x2 U = a.dmean ? mul2(pack2(a.dmean[row], a.dmean[row + 1]), inv_end) : both(0.f);
  const size_t at = (size_t)l.b * s.S * a.D + l.dc;
  auto map = [&](const float* p, int k) { return __ldg(reinterpret_cast<const unsigned long long*>(p + at + (size_t)k * a.D)); };
#pragma unroll 4
  for (int k = s.S - 1; k > l.seg; --k) {
    U = fma2(map(s.sw, k), V, add2(U, map(s.su, k)));
    V = add2(V, map(s.sv, k));
  }
  f32x2 W = fma2(map(s.sw, l.seg), V, add2(U, map(s.su, l.seg)));   // U as it leaves the segment's first step
  V = add2(V, map(s.sv, l.seg));
  if (l.seg == 0 && l.ok) {
    const bool any = total > 0.f;   // (no unmasked step: the incoming gradients pass through)
    float wv[2], vv[2];
    unpack2(W, wv[0], wv[1]);
    unpack2(V, vv[0], vv[1]);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      a.dprev_mean[row + k] = any ? n0 * wv[k] : (a.dmean ? a.dmean[row + k] : 0.f);
      a.dprev_var[row + k] = any ? n0 * vv[k] : (a.dvar ? a.dvar[row + k] : 0.f);
    }
  }
  f32x2 V2 = add2(V, V);
  Run in[2];
  pair_before(s, l, in);
  PairRunning st;
  st.start(in, a.eps, x + (l.dc - l.d0), a.xsl, m, l.t0, l.t1);
  walk_pairs<T, true, kMask, kRingTwo<T>>(x, a.xsl, g, a.gsl, m, l.t0, l.t1, l.left, rings + (size_t)l.warp * 2 * kRingTwo<T> * kTileBytes,
                             [&](f32x2 xv, f32x2 gv, bool pad) {
                               f32x2 out = both(0.f);
                               if (!(kMask && pad)) {
                                 const f32x2 up = st.u;
                                 f32x2 inv, r;
                                 const f32x2 d = st.step(xv, inv, r);
                                 const f32x2 xu = sub2(d, st.u), gr = mul2(gv, r), wi = mul2(w, inv);
                                 const f32x2 h = fma2(mul2(sub2(d, up), inv), V2, W);   // W + e V
                                 out = fma2(gr, w, fma2(xu, V2, h));
                                 W = fma2(gr, wi, h);                                   // W - (a - e V) with a = -gr w / n
                                 V2 = fma2(mul2(mul2(gr, xu), mul2(r, r)), wi, V2);     // V - b
                               }
                               if (l.ok) pair_st(pd, out);
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
                            if (kMask && pad) return;   // (whatever stands there, NaN included)
                            ds = fmaf(gv, xv - u, ds);
                            db += gv;
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
static double pick_segments(const ScanNormArgs& a, int resident, int width, SegNorm& s) {
  const long long strips = (long long)((a.D + width - 1) / width) * a.B;
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
  return best;
}

template <typename T, bool kMask>
static void fwd_launch(const SegNorm& s, cudaStream_t st) {
  const dim3 grid((s.a.D + 31) / 32, (s.S + kWarps - 1) / kWarps, s.a.B), block(kWarps * 32);
  const dim3 pairs((s.a.D + 63) / 64, grid.y, grid.z);
  const size_t rings = (size_t)kWarps * kRing * kTileBytes;
  launch(norm_moments_kernel<T, kMask>, grid, block, rings, (void*)st, moments_of(s));
  if (s.a.wide) launch(norm_emit_kernel<T, kMask, true>, pairs, block, rings, (void*)st, s);
  else launch(norm_emit_kernel<T, kMask, false>, pairs, block, rings, (void*)st, s);
}
template <typename T, bool kMask>
static void bwd_launch(const SegNorm& s, cudaStream_t st) {
  const dim3 grid((s.a.D + 31) / 32, (s.S + kWarps - 1) / kWarps, s.a.B), block(kWarps * 32);
  const dim3 pairs((s.a.D + 63) / 64, grid.y, grid.z);
  const size_t rings = (size_t)kWarps * kRing * kTileBytes, two = (size_t)kWarps * 2 * kRingTwo<T> * kTileBytes;
  launch(norm_moments_kernel<T, kMask>, grid, block, rings, (void*)st, moments_of(s));
  launch(norm_bwd_map_kernel<T, kMask>, pairs, block, two, (void*)st, s);
  launch(norm_bwd_emit_kernel<T, kMask>, pairs, block, two, (void*)st, s);
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
  pick_segments(a, bwd ? 3 : 6, 32, s);
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
  // Resident blocks.  Backward: a fourth shares the FMA pipe with the others, so in one round it has to make the walks a good deal shorter
  // (32 x 2048 x 512 136 us with three, 128 with four; 50 x 273 x 288 36 and 42; in two rounds 38 x 1706 x 480 142 and 125).
  const double cost = pick_segments(a, kBwd ? 3 : 6, 64, s);
  if (kBwd && dtype != MEGA_F32) {
    SegNorm four = s;
    const double least = pick_segments(a, 4, 64, four);
    const bool rounds = (long long)((a.D + 63) / 64) * a.B * ((four.S + kWarps - 1) / kWarps) > 4 * 148;
    if (least < (rounds ? 1. : 0.85) * cost) s = four;
  }
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

// outputs are stored two channels at a time
static bool pairs_ok(int dtype, const ScanNormArgs& a, long long ysd) {
  return ysd == 1 && aligned_to(a.y, 2 * elem_size(dtype)) && a.ysb % 2 == 0 && a.ysl % 2 == 0;
}

// (us, from 15 shapes of 2 to 67 M elements to 4 %; 537 M are 614)
double scan_norm_us(const ScanNormArgs& a) { return (14.0 + (double)a.B * a.D * a.L / 740e3) * (a.mask ? 1.32 : 1.0); }

bool stats_in_place(const ScanNormArgs& a) {
  const size_t n = (size_t)a.B * a.D;
  for (const float* out : {a.mean_out, a.var_out})
    if (overlap(out, a.prev_mean, n) || overlap(out, a.prev_var, n)) return true;
  return false;
}

bool scan_norm_fwd_try(int dtype, const ScanNormArgs& a, long long xsd, long long ysd, cudaStream_t s) {
  if (!pieces_ok(dtype, a.D) || !rows_ok(dtype, a.x, a.xsb, a.xsl, xsd) || !((a.wide && !a.y) || pairs_ok(dtype, a, ysd)) ||
      a.x == a.y)
    return false;
  if (stats_in_place(a)) return false;   // (every segment's block reads the incoming statistics, the last one's writes the new ones)
  return dispatch<false>(dtype, a, s);
}

bool scan_norm_bwd_try(int dtype, const ScanNormArgs& a, long long xsd, long long ysd, long long gsd, cudaStream_t s) {
  if (!pieces_ok(dtype, a.D) || !rows_ok(dtype, a.x, a.xsb, a.xsl, xsd) || !rows_ok(dtype, a.dy, a.gsb, a.gsl, gsd) ||
      !pairs_ok(dtype, a, ysd) || a.y == a.x || a.y == a.dy)
    return false;
  return dispatch<true>(dtype, a, s);
}

bool scan_sqn_fwd_try(int dtype, const ScanNormArgs& a, long long xsd, long long ysd, cudaStream_t s) {
  if (!pieces_ok(dtype, a.D) || !rows_ok(dtype, a.x, a.xsb, a.xsl, xsd) || ysd != 1) return false;
  return sqn_dispatch(dtype, a, false, s);
}

bool scan_sqn_bwd_try(int dtype, const ScanNormArgs& a, long long xsd, long long ysd, long long gsd, cudaStream_t s) {
  if (!pieces_ok(dtype, a.D) || !rows_ok(dtype, a.x, a.xsb, a.xsl, xsd) || !rows_ok(dtype, a.dy, a.gsb, a.gsl, gsd) || ysd != 1 ||
      a.y == a.x || a.y == a.dy)
    return false;
  return sqn_dispatch(dtype, a, true, s);
}

}  // namespace mega
