// The EMA layer and its backward, parallel over time: real or complex poles, causal or bidirectional, any
// activation type, any strides along batch and time, channels contiguous.
//
// A pole state is a linear recurrence, so the sequence is cut into segments that run at the same time.
// (1) every segment folds its inputs into a state of its own, from zero; (2) a small launch carries the
// states over the segments (H <- q^T H + h); (3) every segment runs again from the state it really starts
// with and emits its outputs.  A warp owns 32 adjacent channels of one segment, a lane one channel with
// its 16 poles in registers (ndim < 16: the rest are inert), so memory is read in whole rows and nothing is
// exchanged between lanes.  Work per element and direction: 16 + 32 FMA real, twice to three times that
// complex (the walk of one segment per sequence needs no first pass: 32).
// Bound: the FMA pipe, when segments x channels fill the SMs; a sequence walked as one chain is bound by its
// own latency instead (B = 8, L = 1024, D = 512 fp32: 103 us as 128 chains of 1024 steps).
//
// TimestepNorm in front (norm_run.cuh): two small launches give every segment the statistics it starts from, and the
// walks normalise their inputs as they read them, in fp32, so nothing but x is read and nothing but y written.
//
// Backward.  With h the states for unit input gain, s = dh/dq and lambda the adjoint scaled by 1 / (p g):
//   h_t = q h_{t-1} + x~_t,  s_t = q s_{t-1} + h_{t-1},  lambda_t = q lambda_{t+1} + dy_t,
//   dx~_t = sum_n p g lambda_t,  dg = p sum dy h,  dp = g sum dy h,  dq = p g sum dy s,
// with real parts taken for complex poles; the anti-causal half runs the same in reversed time.  The same
// three steps: local (h, s, lambda) per segment, carried over the segments, then the sums and dx.
#include <cmath>

#include "common.cuh"
#include "norm_run.cuh"
#include "poles.cuh"
#include "scan_cluster.cuh"
#include "scan_ema.cuh"
#include "scratch.cuh"
#include "tma.cuh"
#include "walk.cuh"

namespace mega {

namespace {


struct SegArgs {
  ScanArgs a;
  int T, S;          // steps per segment, segments
  int wide;          // one segment: the warps of a block own adjacent channel groups instead of segments
  float *rn, *rm, *rs;   // TimestepNorm in front: what every segment starts from (count; mean, squared deviations)
  int parts;         // values per (batch, direction, segment, pole, channel) in the carry array
  float* carry;      // [B][dirs][S][parts][16][D]
};

// Entry of a state in the carry array: lanes are adjacent channels.
template <bool kC>
__device__ __forceinline__ void store_state(const State<kC>& h, float* dst, int D, bool ok) {
  if (!ok) return;
#pragma unroll
  for (int j = 0; j < kP2; ++j) {
    float lo, hi;
    unpack2(h.r[j], lo, hi);
    dst[(size_t)(2 * j) * D] = lo;
    dst[(size_t)(2 * j + 1) * D] = hi;
    if (kC) {
      unpack2(h.i[j], lo, hi);
      dst[(size_t)(16 + 2 * j) * D] = lo;
      dst[(size_t)(16 + 2 * j + 1) * D] = hi;
    }
  }
}
template <bool kC>
__device__ __forceinline__ void load_state(State<kC>& h, const float* src, int D) {
#pragma unroll
  for (int j = 0; j < kP2; ++j) {
    h.r[j] = pack2(__ldg(src + (size_t)(2 * j) * D), __ldg(src + (size_t)(2 * j + 1) * D));
    if (kC) h.i[j] = pack2(__ldg(src + (size_t)(16 + 2 * j) * D), __ldg(src + (size_t)(16 + 2 * j + 1) * D));
  }
}

// (batch, direction, segment) entry of the carry array
__device__ __forceinline__ float* carry_at(const SegArgs& s, int b, int dir, int seg, int part, int d) {
  const int dirs = s.a.bidir ? 2 : 1;
  return s.carry + ((((size_t)b * dirs + dir) * s.S + seg) * s.parts + part) * 16 * s.a.D + d;
}

struct Lane {
  int lane, warp, d, dc, b, seg, t0, t1, d0, left;   // d0: first channel of the warp, left: channels from there
  bool ok;
};
__device__ __forceinline__ Lane lane_of(const SegArgs& s) {
  Lane l;
  l.lane = threadIdx.x & 31;
  l.warp = threadIdx.x >> 5;
  l.d = (s.wide ? blockIdx.x * kWarps + l.warp : blockIdx.x) * 32 + l.lane;
  l.d0 = l.d - l.lane < s.a.D ? l.d - l.lane : 0;
  l.left = s.a.D - (l.d - l.lane);
  l.ok = l.d < s.a.D;
  l.dc = l.ok ? l.d : s.a.D - 1;
  l.seg = s.wide ? 0 : blockIdx.y * kWarps + l.warp;
  l.b = blockIdx.z;
  l.t0 = min(s.a.L, l.seg * s.T);
  l.t1 = min(s.a.L, l.t0 + s.T);
  return l;
}

// ---- TimestepNorm in front --------------------------------------------------------------------------
// Moments of the segments -> what each segment starts from, and the statistics after the last (mean_out and var_out may
// be prev_mean and prev_var: the thread that writes a channel's is the only one to read them).
__global__ void __launch_bounds__(128) scan_stats_kernel(SegArgs s) {
  const ScanArgs& a = s.a;
  const int d = blockIdx.x * 128 + threadIdx.x, b = blockIdx.y;
  if (d >= a.D) return;
  const long long cnt0 = a.prev_count[b];
  const float n0 = (float)cnt0;
  const size_t i = (size_t)b * a.D + d;
  Run r{n0, a.prev_mean[i], a.prev_var[i] * n0};
  long long seen = 0;   // unmasked steps of the call (a float count that starts beyond 2^24 would round them)
  const float* pn = s.rn + (size_t)b * s.S;
  float *pm = s.rm + (size_t)b * s.S * a.D + d, *ps = s.rs + (size_t)b * s.S * a.D + d;
  constexpr int kB = 8;
  for (int k0 = 0; k0 < s.S; k0 += kB) {
    Run seg[kB];
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const int k = min(k0 + u, s.S - 1);
      seg[u] = Run{__ldg(pn + k), __ldcg(pm + (size_t)k * a.D), __ldcg(ps + (size_t)k * a.D)};
    }
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      if (k0 + u < s.S) {
        pm[(size_t)(k0 + u) * a.D] = r.m;
        ps[(size_t)(k0 + u) * a.D] = r.s;
        r = combine(r, seg[u]);
        seen += (long long)seg[u].n;
      }
    }
  }
  a.mean_out[i] = r.n > 0.f ? r.m : a.prev_mean[i];
  a.var_out[i] = r.n > 0.f ? r.s / r.n : a.prev_var[i];
  if (d == 0) a.count_out[b] = cnt0 + seen;
}

// The statistics a segment starts from.
__device__ __forceinline__ Run stats_of(const SegArgs& s, int b, int seg, int d) {
  float seen = 0.f;
  for (int k = 0; k < seg; ++k) seen += __ldg(s.rn + (size_t)b * s.S + k);
  const float n = (float)s.a.prev_count[b] + seen;
  const size_t i = ((size_t)b * s.S + seg) * s.a.D + d;
  return Run{n, __ldg(s.rm + i), __ldg(s.rs + i)};
}
// ---- (1) local states ---------------------------------------------------------------------------
// forward: h of each direction.  backward: (h, s) of each direction and the adjoint, which runs the other way.
template <typename T, bool kC, bool kMask, bool kBwd, bool kNorm = false>
__global__ void __launch_bounds__(kWarps * 32) scan_local_kernel(SegArgs s) {
  static_assert(!kNorm || !kBwd, "the norm in front is a forward form");
  const ScanArgs& a = s.a;
  const int dirs = a.bidir ? 2 : 1;
  SegArgs ss = s;
  Lane l = lane_of(ss);
  const int dir = l.b % dirs;
  l.b /= dirs;
  if (l.seg >= s.S) return;
  const T* x = reinterpret_cast<const T*>(a.x) + l.b * a.xsb + l.d0;
  const unsigned char* m = kMask ? a.mask + (size_t)l.b * a.L : nullptr;
  Poles<kC> P;
  load_poles<kC>(P, a, l.dc + dir * a.D);
  extern __shared__ __align__(16) unsigned char rings[];
  unsigned char* ring = rings + (size_t)l.warp * kRing * kTileBytes;
  State<kC> h;
  h.zero();
  constexpr int kOne = kC ? 2 : 1;   // parts of a state
  if (kBwd) {
    State<kC> sn;
    sn.zero();
    auto step = [&](int, float xv, float, bool pad) {
      advance_sens<kC>(sn, h, P);
      advance<kC>(h, P, splat(kMask && pad ? 0.f : xv));
    };
    if (dir == 0) walk<T, 1, false, kMask>(x, a.xsl, x, 0, m, l.t0, l.t1, l.left, ring, step);
    else walk<T, -1, false, kMask>(x, a.xsl, x, 0, m, l.t0, l.t1, l.left, ring, step);
    store_state<kC>(h, carry_at(s, l.b, dir, l.seg, 0, l.dc), a.D, l.ok);
    store_state<kC>(sn, carry_at(s, l.b, dir, l.seg, kOne, l.dc), a.D, l.ok);
    h.zero();
    const T* g = reinterpret_cast<const T*>(a.dy) + l.b * a.gsb + l.d0;
    auto adj = [&](int, float gv, float, bool) { advance<kC>(h, P, splat(gv)); };
    if (dir == 0) walk<T, -1, false, false>(g, a.gsl, g, 0, m, l.t0, l.t1, l.left, ring, adj);
    else walk<T, 1, false, false>(g, a.gsl, g, 0, m, l.t0, l.t1, l.left, ring, adj);
    store_state<kC>(h, carry_at(s, l.b, dir, l.seg, 2 * kOne, l.dc), a.D, l.ok);
  } else if constexpr (kNorm) {
    Running st;
    st.start(stats_of(s, l.b, l.seg, l.dc));
    const float w = __ldg(a.gamma + l.dc), bb = __ldg(a.beta + l.dc), eps = a.eps;
    walk<T, 1, false, kMask>(x, a.xsl, x, 0, m, l.t0, l.t1, l.left, ring, [&](int, float xv, float, bool pad) {
      advance<kC>(h, P, splat(normed(st, xv, kMask && pad, w, bb, eps)));
    });
    store_state<kC>(h, carry_at(s, l.b, dir, l.seg, 0, l.dc), a.D, l.ok);
  } else {
    auto step = [&](int, float xv, float, bool pad) { advance<kC>(h, P, splat(kMask && pad ? 0.f : xv)); };
    if (dir == 0) walk<T, 1, false, kMask>(x, a.xsl, x, 0, m, l.t0, l.t1, l.left, ring, step);
    else walk<T, -1, false, kMask>(x, a.xsl, x, 0, m, l.t0, l.t1, l.left, ring, step);
    store_state<kC>(h, carry_at(s, l.b, dir, l.seg, 0, l.dc), a.D, l.ok);
  }
}

// ---- (2) carry over the segments -----------------------------------------------------------------
// One thread per (channel, pole, direction, batch): replaces each segment's local values by the values the
// segment starts from.  kGain: true states (input gain applied), from h_in, the last one to h_out.
template <bool kC, bool kBwd>
__global__ void __launch_bounds__(128) scan_carry_kernel(SegArgs s, int gain) {
  const ScanArgs& a = s.a;
  const int dirs = a.bidir ? 2 : 1;
  const int d = blockIdx.x * 128 + threadIdx.x;
  const int n = blockIdx.y;
  const int dir = blockIdx.z % dirs, b = blockIdx.z / dirs;
  if (d >= a.D) return;
  const bool live = n < a.N;
  const size_t c = (size_t)(d + dir * a.D) * a.N + n;
  float2 q = make_float2(0.f, 0.f);
  if (live) q = kC ? make_float2(__ldg(a.q + 2 * c), __ldg(a.q + 2 * c + 1)) : make_float2(__ldg(a.q + c), 0.f);
  const int last = a.L - (s.S - 1) * s.T;   // steps of the last segment
  float2 qT, qLast, qT1 = make_float2(0.f, 0.f), qLast1 = make_float2(0.f, 0.f);
  if (kC) {
    qT = ipow(q, s.T);
    qLast = ipow(q, last);
    if (kBwd) {
      qT1 = ipow(q, s.T - 1);
      qLast1 = ipow(q, last - 1);
    }
  } else {
    qT = make_float2(powf(q.x, (float)s.T), 0.f);
    qLast = make_float2(powf(q.x, (float)last), 0.f);
    if (kBwd) {
      qT1 = make_float2(powf(q.x, (float)(s.T - 1)), 0.f);
      qLast1 = make_float2(powf(q.x, (float)(last - 1)), 0.f);
    }
  }
  constexpr int kOne = kC ? 2 : 1;
  const size_t step = (size_t)s.parts * 16 * a.D;
  float* base = carry_at(s, b, dir, 0, 0, d) + (size_t)n * a.D;
  const size_t im = (size_t)16 * a.D;   // imaginary part of the same value
  const size_t part = (size_t)kOne * 16 * a.D;
  float2 H = make_float2(0.f, 0.f), Sn = make_float2(0.f, 0.f);
  const float pg = (gain && live) ? __ldg(a.p + c) : 1.f;
  const size_t sidx = ((size_t)b * a.D + d) * a.N + n;
  if (gain && a.h_in && live) H = kC ? make_float2(a.h_in[2 * sidx], a.h_in[2 * sidx + 1]) : make_float2(a.h_in[sidx], 0.f);
  // (the loads of kB segments go out together: a load that follows the store of the segment before would wait
  // for the whole round trip of every segment)
  constexpr int kB = 8;
  for (int k0 = 0; k0 < s.S; k0 += kB) {
    float2 loc[kB], ls[kBwd ? kB : 1];
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const int k = min(k0 + u, s.S - 1);
      const float* v = base + (size_t)(dir == 0 ? k : s.S - 1 - k) * step;
      loc[u] = make_float2(__ldcg(v), kC ? __ldcg(v + im) : 0.f);
      if (kBwd) ls[kBwd ? u : 0] = make_float2(__ldcg(v + part), kC ? __ldcg(v + part + im) : 0.f);
    }
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      if (k0 + u < s.S) {
        const int seg = dir == 0 ? k0 + u : s.S - 1 - (k0 + u);
        float* v = base + (size_t)seg * step;
        const bool lst = seg == s.S - 1;
        const float2 w = lst ? qLast : qT;
        v[0] = H.x;
        if (kC) v[im] = H.y;
        if (kBwd) {
          float* uu = v + part;
          const float2 w1 = lst ? qLast1 : qT1;
          const float len = lst ? (float)last : (float)s.T;
          const float2 l2 = ls[kBwd ? u : 0];
          uu[0] = Sn.x;
          if (kC) {
            uu[im] = Sn.y;
            const float2 a1 = cmul(w, Sn), a2 = cmul(w1, H);
            Sn = make_float2(a1.x + fmaf(len, a2.x, l2.x), a1.y + fmaf(len, a2.y, l2.y));
          } else {
            Sn.x = fmaf(w.x, Sn.x, fmaf(len * w1.x, H.x, l2.x));
          }
        }
        if (kC) {
          const float2 a1 = cmul(w, H);
          H = make_float2(fmaf(pg, loc[u].x, a1.x), fmaf(pg, loc[u].y, a1.y));
        } else {
          H.x = fmaf(w.x, H.x, pg * loc[u].x);
        }
      }
    }
  }
  if (gain && a.h_out && live) {
    if (kC) {
      a.h_out[2 * sidx] = H.x;
      a.h_out[2 * sidx + 1] = H.y;
    } else {
      a.h_out[sidx] = H.x;
    }
  }
  if (kBwd) {   // the adjoint, against the direction
    float2 A = make_float2(0.f, 0.f);
    for (int k0 = s.S - 1; k0 >= 0; k0 -= kB) {
      float2 loc[kB];
#pragma unroll
      for (int u = 0; u < kB; ++u) {
        const int k = max(k0 - u, 0);
        const float* v = base + (size_t)(dir == 0 ? k : s.S - 1 - k) * step + 2 * part;
        loc[u] = make_float2(__ldcg(v), kC ? __ldcg(v + im) : 0.f);
      }
#pragma unroll
      for (int u = 0; u < kB; ++u) {
        if (k0 - u >= 0) {
          const int seg = dir == 0 ? k0 - u : s.S - 1 - (k0 - u);
          float* v = base + (size_t)seg * step + 2 * part;
          const float2 w = seg == s.S - 1 ? qLast : qT;
          v[0] = A.x;
          if (kC) {
            v[im] = A.y;
            const float2 a1 = cmul(w, A);
            A = make_float2(a1.x + loc[u].x, a1.y + loc[u].y);
          } else {
            A.x = fmaf(w.x, A.x, loc[u].x);
          }
        }
      }
    }
  }
}

// ---- (3) outputs -----------------------------------------------------------------------------------
template <typename T, bool kC, bool kMask, bool kState, bool kNorm = false>
__global__ void __launch_bounds__(kWarps * 32, kC || kNorm ? 3 : 4) scan_emit_kernel(SegArgs s) {
  const ScanArgs& a = s.a;
  const Lane l = lane_of(s);
  if (l.seg >= s.S) return;
  const T* x = reinterpret_cast<const T*>(a.x) + l.b * a.xsb + l.d0;
  T* y = reinterpret_cast<T*>(a.y) + l.b * a.ysb + l.dc;
  const unsigned char* m = kMask ? a.mask + (size_t)l.b * a.L : nullptr;
  const float om = __ldg(a.omega + l.dc);
  extern __shared__ __align__(16) unsigned char rings[];
  unsigned char* ring = rings + (size_t)l.warp * kRing * kTileBytes;
  Poles<kC> P;
  State<kC> c, h;
  f32x2 p[kState ? kP2 : 1];
  load_poles<kC>(P, a, l.dc);
  load_weights<kC>(c, a, l.dc, !kState);
  if (kState) {
#pragma unroll
    for (int j = 0; j < kP2; ++j) {
      const size_t n = (size_t)l.dc * a.N + 2 * j;
      p[kState ? j : 0] = pack2(2 * j < a.N ? __ldg(a.p + n) : 0.f, 2 * j + 1 < a.N ? __ldg(a.p + n + 1) : 0.f);
    }
  }
  h.zero();
  if (s.carry) {
    load_state<kC>(h, carry_at(s, l.b, 0, l.seg, 0, l.dc), a.D);
  } else if (kState && a.h_in) {
#pragma unroll
    for (int j = 0; j < kP2; ++j) {
      const size_t n = ((size_t)l.b * a.D + l.dc) * a.N + 2 * j;
      float r[2] = {0.f, 0.f}, i[2] = {0.f, 0.f};
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (2 * j + k < a.N) {
          r[k] = kC ? __ldg(a.h_in + 2 * (n + k)) : __ldg(a.h_in + n + k);
          if (kC) i[k] = __ldg(a.h_in + 2 * (n + k) + 1);
        }
      h.r[j] = pack2(r[0], r[1]);
      if (kC) h.i[j] = pack2(i[0], i[1]);
    }
  }
  if (a.bidir) {   // the causal half leaves its share of the outputs in shared memory
    float* part = reinterpret_cast<float*>(rings + kWarps * kRing * kTileBytes);
    float* mine = part + (size_t)l.warp * s.T * 32 + l.lane;
    walk<T, 1, false, kMask>(x, a.xsl, x, 0, m, l.t0, l.t1, l.left, ring, [&](int k, float xv, float, bool pad) {
      advance<kC>(h, P, splat(kMask && pad ? 0.f : xv));
      mine[k * 32] = fmaf(om, xv, dot<kC>(c, h));
    });
    load_poles<kC>(P, a, l.dc + a.D);
    load_weights<kC>(c, a, l.dc + a.D, true);
    load_state<kC>(h, carry_at(s, l.b, 1, l.seg, 0, l.dc), a.D);
    const bool shift = a.shift != 0;
    const float* last = mine + (l.t1 - l.t0 - 1) * 32;
    T* py = y + (long long)(l.t1 - 1) * a.ysl;
    walk<T, -1, false, kMask>(x, a.xsl, x, 0, m, l.t0, l.t1, l.left, ring, [&](int k, float xv, float, bool pad) {
      float v = last[-k * 32];
      if (shift) v += dot<kC>(c, h);
      advance<kC>(h, P, splat(kMask && pad ? 0.f : xv));
      if (!shift) v += dot<kC>(c, h);
      if (a.silu) v = siluf_(v);
      if (l.ok) Elem<T>::st(py, v);
      py -= a.ysl;
    });
    return;
  }
  T* py = y + (long long)l.t0 * a.ysl;
  if constexpr (kNorm) {
    Running st;
    st.start(stats_of(s, l.b, l.seg, l.dc));
    const float w = __ldg(a.gamma + l.dc), bb = __ldg(a.beta + l.dc), eps = a.eps;
    T* pn = a.xn ? reinterpret_cast<T*>(a.xn) + (py - reinterpret_cast<T*>(a.y)) : nullptr;   // (strided like y)
    walk<T, 1, false, kMask>(x, a.xsl, x, 0, m, l.t0, l.t1, l.left, ring, [&](int, float xv, float, bool pad) {
      const float xn = normed(st, xv, kMask && pad, w, bb, eps);
      const f32x2 x2 = splat(xn);
      if constexpr (kState) advance_gain<kC>(h, P, p, x2);
      else advance<kC>(h, P, x2);
      float v = fmaf(om, xn, dot<kC>(c, h));
      if (a.silu) v = siluf_(v);
      if (l.ok) Elem<T>::st(py, v);
      py += a.ysl;
      if (pn) {
        if (l.ok) Elem<T>::st(pn, xn);
        pn += a.ysl;
      }
    });
  } else walk<T, 1, false, kMask>(x, a.xsl, x, 0, m, l.t0, l.t1, l.left, ring, [&](int k, float xv, float, bool pad) {
    const f32x2 x2 = splat(kMask && pad ? 0.f : xv);
    if constexpr (kState) advance_gain<kC>(h, P, p, x2);
    else advance<kC>(h, P, x2);
    float v = fmaf(om, xv, dot<kC>(c, h));
    if (a.silu) v = siluf_(v);
    if (l.ok) Elem<T>::st(py, v);
    py += a.ysl;
  });
  if (kState && !s.carry && a.h_out && l.ok) {
#pragma unroll
    for (int j = 0; j < kP2; ++j) {
      const size_t n = ((size_t)l.b * a.D + l.d) * a.N + 2 * j;
      float r[2], i[2] = {0.f, 0.f};
      unpack2(h.r[j], r[0], r[1]);
      if (kC) unpack2(h.i[j], i[0], i[1]);
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (2 * j + k < a.N) {
          if (kC) {
            a.h_out[2 * (n + k)] = r[k];
            a.h_out[2 * (n + k) + 1] = i[k];
          } else {
            a.h_out[n + k] = r[k];
          }
        }
    }
  }
}

// Sums of a block's segments, then one atomic add per parameter.  red: [kWarps][32][32] floats.
template <bool kC>
__device__ __forceinline__ void reduce_grads(const State<kC>& ah, const State<kC>& as, const ScanArgs& a, int row, bool ok,
                                             bool active, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kV = kC ? 64 : 32;   // sums per channel: dy h, dy s
  for (int r0 = 0; r0 < kV; r0 += 32) {
    // kV values of every lane go through shared memory, 32 at a time
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kP2; ++j) {
      float v0, v1;
      if (r0 == 0) {
        unpack2(ah.r[j], v0, v1);
        red[(warp * 32 + 2 * j) * 32 + lane] = active ? v0 : 0.f;
        red[(warp * 32 + 2 * j + 1) * 32 + lane] = active ? v1 : 0.f;
        unpack2(as.r[j], v0, v1);
        red[(warp * 32 + 16 + 2 * j) * 32 + lane] = active ? v0 : 0.f;
        red[(warp * 32 + 16 + 2 * j + 1) * 32 + lane] = active ? v1 : 0.f;
      } else if (kC) {
        unpack2(ah.i[kC ? j : 0], v0, v1);
        red[(warp * 32 + 2 * j) * 32 + lane] = active ? v0 : 0.f;
        red[(warp * 32 + 2 * j + 1) * 32 + lane] = active ? v1 : 0.f;
        unpack2(as.i[kC ? j : 0], v0, v1);
        red[(warp * 32 + 16 + 2 * j) * 32 + lane] = active ? v0 : 0.f;
        red[(warp * 32 + 16 + 2 * j + 1) * 32 + lane] = active ? v1 : 0.f;
      }
    }
    __syncthreads();
    // warp w finishes poles 4w .. 4w + 3
    for (int n = warp * 4; ok && n < warp * 4 + 4 && n < a.N; ++n) {
      float vh = 0.f, vs = 0.f;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        vh += red[(w * 32 + n) * 32 + lane];
        vs += red[(w * 32 + 16 + n) * 32 + lane];
      }
      const size_t c = (size_t)row * a.N + n;
      const float p = __ldg(a.p + c);
      if (kC) {
        const float gr = __ldg(a.g + 2 * c), gi = __ldg(a.g + 2 * c + 1);
        if (r0 == 0) {   // real parts
          atomicAdd(a.dp + c, gr * vh);
          atomicAdd(a.dg + 2 * c, p * vh);
          atomicAdd(a.dq + 2 * c, p * gr * vs);
          atomicAdd(a.dq + 2 * c + 1, -p * gi * vs);
        } else {
          atomicAdd(a.dp + c, -gi * vh);
          atomicAdd(a.dg + 2 * c + 1, -p * vh);
          atomicAdd(a.dq + 2 * c, -p * gi * vs);
          atomicAdd(a.dq + 2 * c + 1, -p * gr * vs);
        }
      } else {
        const float g = __ldg(a.g + c);
        atomicAdd(a.dp + c, g * vh);
        atomicAdd(a.dg + c, p * vh);
        atomicAdd(a.dq + c, p * g * vs);
      }
    }
  }
}

template <typename T, bool kC, bool kMask>
__global__ void __launch_bounds__(kWarps * 32, kC ? 2 : 3) scan_bwd_kernel(SegArgs s) {
  // rings; bidirectional: [kWarps][T][32] share of dx.  The sums of the block go through the rings' memory.
  extern __shared__ __align__(16) unsigned char rings[];
  const ScanArgs& a = s.a;
  const Lane l = lane_of(s);
  unsigned char* ring = rings + (size_t)l.warp * 2 * kRing * kTileBytes;
  float* part = reinterpret_cast<float*>(rings + kWarps * 2 * kRing * kTileBytes);
  float* red = reinterpret_cast<float*>(rings);
  const bool active = l.seg < s.S;
  const T* x = reinterpret_cast<const T*>(a.x) + l.b * a.xsb + l.d0;
  const T* g = reinterpret_cast<const T*>(a.dy) + l.b * a.gsb + l.d0;
  T* dx = reinterpret_cast<T*>(a.y) + l.b * a.ysb + l.dc;
  const unsigned char* m = kMask ? a.mask + (size_t)l.b * a.L : nullptr;
  const float om = __ldg(a.omega + l.dc);
  constexpr int kOne = kC ? 2 : 1;
  float dom = 0.f;
  for (int dir = 0; dir < (a.bidir ? 2 : 1); ++dir) {
    State<kC> ah, as;
    ah.zero();
    as.zero();
    if (active) {
      Poles<kC> P;
      load_poles<kC>(P, a, l.dc + dir * a.D);
      State<kC> h, sn;
      h.zero();
      sn.zero();
      if (s.carry) {
        load_state<kC>(h, carry_at(s, l.b, dir, l.seg, 0, l.dc), a.D);
        load_state<kC>(sn, carry_at(s, l.b, dir, l.seg, kOne, l.dc), a.D);
      }
      if (dir == 0) {
        walk<T, 1, true, kMask>(x, a.xsl, g, a.gsl, m, l.t0, l.t1, l.left, ring, [&](int, float xv, float gv, bool pad) {
          dom = fmaf(gv, xv, dom);
          advance_sens<kC>(sn, h, P);
          advance<kC>(h, P, splat(kMask && pad ? 0.f : xv));
          accumulate<kC>(ah, h, splat(gv));
          accumulate<kC>(as, sn, splat(gv));
        });
      } else {
        const bool shift = a.shift != 0;
        walk<T, -1, true, kMask>(x, a.xsl, g, a.gsl, m, l.t0, l.t1, l.left, ring, [&](int, float xv, float gv, bool pad) {
          if (shift) {
            accumulate<kC>(ah, h, splat(gv));
            accumulate<kC>(as, sn, splat(gv));
          }
          advance_sens<kC>(sn, h, P);
          advance<kC>(h, P, splat(kMask && pad ? 0.f : xv));
          if (!shift) {
            accumulate<kC>(ah, h, splat(gv));
            accumulate<kC>(as, sn, splat(gv));
          }
        });
      }
      // the adjoint
      State<kC> c;
      load_weights<kC>(c, a, l.dc + dir * a.D, true);
      h.zero();
      if (s.carry) load_state<kC>(h, carry_at(s, l.b, dir, l.seg, 2 * kOne, l.dc), a.D);
      float* mine = part + (size_t)l.warp * s.T * 32 + l.lane;
      if (dir == 0) {
        const bool bidir = a.bidir != 0;
        float* last = mine + (l.t1 - l.t0 - 1) * 32;
        T* pd = dx + (long long)(l.t1 - 1) * a.ysl;
        walk<T, -1, false, kMask>(g, a.gsl, g, 0, m, l.t0, l.t1, l.left, ring, [&](int k, float gv, float, bool pad) {
          advance<kC>(h, P, splat(gv));
          const float v = fmaf(om, gv, kMask && pad ? 0.f : dot<kC>(c, h));
          if (bidir) last[-k * 32] = v;
          else if (l.ok) Elem<T>::st(pd, v);
          pd -= a.ysl;
        });
      } else {
        const bool shift = a.shift != 0;
        T* pd = dx + (long long)l.t0 * a.ysl;
        walk<T, 1, false, kMask>(g, a.gsl, g, 0, m, l.t0, l.t1, l.left, ring, [&](int k, float gv, float, bool pad) {
          float v = 0.f;
          if (shift) v = dot<kC>(c, h);
          advance<kC>(h, P, splat(gv));
          if (!shift) v = dot<kC>(c, h);
          v = mine[k * 32] + (kMask && pad ? 0.f : v);
          if (l.ok) Elem<T>::st(pd, v);
          pd += a.ysl;
        });
      }
    }
    reduce_grads<kC>(ah, as, a, l.dc + dir * a.D, l.ok, active, red);
    __syncthreads();   // (the rings are free again)
  }
  // domega: the block's four segments
  __syncthreads();
  red[l.warp * 32 + l.lane] = dom;
  __syncthreads();
  if (l.warp == 0 && l.ok) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) v += red[w * 32 + l.lane];
    atomicAdd(a.domega + l.d, v);
  }
}

// Segments of a call.  A block takes four segments of 32 channels; `resident` blocks of the last kernel fit an SM.
// The choice minimises (rounds of blocks over the 148 SMs) x (steps of a segment + what its states cost beside
// them: written, carried and read, 64 steps' worth backward and 40 forward), so that neither a nearly empty last round nor short segments dominate; it is returned.  Segments
// are at least 32 steps; a bidirectional one keeps its share of the outputs in shared memory, so at most 64: beyond 4096
// of those the counts start from what the length asks for.
// One segment per sequence when the channels alone fill the device: no first pass then.
static double pick_segments(const ScanArgs& a, int resident, bool bwd, SegArgs& s) {
  const long long strips = (long long)((a.D + 31) / 32) * a.B;
  const double slots = 148.0 * resident;
  double best = 1e30;
  s.wide = 0;
  if (!a.bidir && !bwd && !a.prev_count) {
    s.T = a.L;
    s.S = 1;
    s.wide = 1;
    const long long blocks = (long long)((a.D + 32 * kWarps - 1) / (32 * kWarps)) * a.B;
    // (2/3: without the first pass; few warps on an SM still leave its pipes idle: at least half of the slots)
    best = ceil(blocks / slots) * a.L * (2.0 / 3.0) * (blocks * 2 < slots ? 2.0 : 1.0);
  }
  const int least = a.bidir ? (a.L + 63) / 64 : 1, from = (least + kWarps - 1) / kWarps * kWarps;
  for (int S = from; S < from + 4096; S += kWarps) {
    int t = ((a.L + S - 1) / S + kU - 1) / kU * kU;
    if (t < 32) t = 32;
    if (a.bidir && t > 64) continue;
    const int n = (a.L + t - 1) / t;
    const long long blocks = strips * ((n + kWarps - 1) / kWarps);
    const double cost = ceil(blocks / slots) * (t + (bwd ? 64 : 40));
    if (cost < best) {
      best = cost;
      s.T = t;
      s.S = n;
      s.wide = 0;
    }
    if (t == 32) break;
  }
  return best;
}

template <typename T, bool kC, bool kMask, bool kNorm>
static bool fwd_launch(const SegArgs& s, cudaStream_t st) {
  const ScanArgs& a = s.a;
  const int dirs = a.bidir ? 2 : 1;
  const dim3 block(kWarps * 32);
  const dim3 grid(s.wide ? (a.D + 32 * kWarps - 1) / (32 * kWarps) : (a.D + 31) / 32, (s.S + kWarps - 1) / kWarps, a.B);
  const bool state = a.h_in || a.h_out;
  const size_t rings = (size_t)kWarps * kRing * kTileBytes;
  if (kNorm) {
    const MomentArgs m{a.x, a.xsb, a.xsl, a.mask, a.L, a.D, s.T, s.S, s.rn, s.rm, s.rs};
    launch(norm_moments_kernel<T, kMask>, grid, block, rings, (void*)st, m);
    launch(scan_stats_kernel, dim3((a.D + 127) / 128, a.B), 128, 0, (void*)st, s);
  }
  if (s.carry) {
    launch(scan_local_kernel<T, kC, kMask, false, kNorm>, dim3(grid.x, grid.y, a.B * dirs), block, rings, (void*)st, s);
    launch(scan_carry_kernel<kC, false>, dim3((a.D + 127) / 128, 16, a.B * dirs), 128, 0, (void*)st, s, state ? 1 : 0);
  }
  const size_t smem = rings + (a.bidir ? (size_t)kWarps * s.T * 32 * 4 : 0);
  if (state) launch(scan_emit_kernel<T, kC, kMask, true, kNorm>, grid, block, smem, (void*)st, s);
  else launch(scan_emit_kernel<T, kC, kMask, false, kNorm>, grid, block, smem, (void*)st, s);
  return true;
}

template <typename T, bool kC, bool kMask>
static bool bwd_launch(const SegArgs& s, cudaStream_t st) {
  const ScanArgs& a = s.a;
  const int dirs = a.bidir ? 2 : 1;
  const dim3 block(kWarps * 32);
  const dim3 grid((a.D + 31) / 32, (s.S + kWarps - 1) / kWarps, a.B);
  const size_t rings = (size_t)kWarps * kRing * kTileBytes;
  if (s.carry) {
    launch(scan_local_kernel<T, kC, kMask, true>, dim3(grid.x, grid.y, a.B * dirs), block, rings, (void*)st, s);
    launch(scan_carry_kernel<kC, true>, dim3((a.D + 127) / 128, 16, a.B * dirs), 128, 0, (void*)st, s, 0);
  }
  const size_t smem = 2 * rings + (a.bidir ? (size_t)kWarps * s.T * 32 * 4 : 0);
  launch(scan_bwd_kernel<T, kC, kMask>, grid, block, smem, (void*)st, s);
  return true;
}

template <bool kBwd>
static bool dispatch(int dtype, const ScanArgs& a, cudaStream_t st) {
  if (g_options[OPT_DISABLE_STREAM].load() != 0) return false;
  const int dirs = a.bidir ? 2 : 1;
  if (a.N > 16 || (long long)a.B * dirs > 65535 || a.L < 1) return false;
  SegArgs s{};
  s.a = a;
  // blocks per SM by registers
  pick_segments(a, kBwd ? (a.cplx ? 2 : 3) : (a.cplx || a.prev_count ? 3 : 4), kBwd, s);
  if (s.S < 1 || (s.S + kWarps - 1) / kWarps > 65535) return false;
  s.parts = (kBwd ? 3 : 1) * (a.cplx ? 2 : 1);
  const size_t floats = (!s.wide) ? (size_t)a.B * dirs * s.S * s.parts * 16 * a.D : 0;
  const bool norm = !kBwd && a.prev_count != nullptr;
  const size_t stats = norm ? (size_t)a.B * s.S * a.D : 0;
  Scratch sc(Scratch::padded(floats * 4) + 2 * Scratch::padded(stats * 4) + Scratch::padded((size_t)a.B * s.S * 4), st);
  if (!sc) return false;
  if (norm) {
    s.rn = sc.take<float>((size_t)a.B * s.S);
    s.rm = sc.take<float>(stats);
    s.rs = sc.take<float>(stats);
  }
  s.carry = floats ? sc.take<float>(floats) : nullptr;
#define MEGA_SCAN_FORM(TY, CPLX, MASK)                                             \
  (kBwd ? bwd_launch<TY, CPLX, MASK>(s, st)                                        \
        : norm ? fwd_launch<TY, CPLX, MASK, true>(s, st) : fwd_launch<TY, CPLX, MASK, false>(s, st))
#define MEGA_SCAN(TY)                                                              \
  (a.cplx ? (a.mask ? MEGA_SCAN_FORM(TY, true, true) : MEGA_SCAN_FORM(TY, true, false)) \
          : (a.mask ? MEGA_SCAN_FORM(TY, false, true) : MEGA_SCAN_FORM(TY, false, false)))
  switch (dtype) {
    case MEGA_F32: return MEGA_SCAN(float);
    case MEGA_BF16: return MEGA_SCAN(__nv_bfloat16);
    case MEGA_F16: return MEGA_SCAN(__half);
    default: return false;
  }
#undef MEGA_SCAN
#undef MEGA_SCAN_FORM
}

}  // namespace

bool scan_ema_fwd_ok(int dtype, const ScanArgs& a, long long xsd, long long ysd) {
  return g_options[OPT_DISABLE_STREAM].load() == 0 && rows_ok(dtype, a.x, a.xsb, a.xsl, xsd) && (!a.prev_count || pieces_ok(dtype, a.D)) &&
         ysd == 1 && a.N <= 16 &&
         (long long)a.B * (a.bidir ? 2 : 1) <= 65535 && (a.x != a.y || (a.xsb == a.ysb && a.xsl == a.ysl));
}

// (16 x 4096 x 1024: 254 us real, 565 complex; 64 x 256 x 1024: 52 and 110)
double scan_ema_fwd_us(const ScanArgs& a) {
  SegArgs s{};
  return 10. + pick_segments(a, a.cplx || a.prev_count ? 3 : 4, false, s) * (a.cplx ? 0.33 : 0.23);
}

bool scan_ema_fwd_try(int dtype, const ScanArgs& a, long long xsd, long long ysd, cudaStream_t s) {
  if (!scan_ema_fwd_ok(dtype, a, xsd, ysd)) return false;
  if (scan_cluster_try(dtype, a, s)) return true;
  return dispatch<false>(dtype, a, s);
}

bool scan_ema_bwd_try(int dtype, const ScanArgs& a, long long xsd, long long ysd, long long gsd, cudaStream_t s) {
  if (!rows_ok(dtype, a.x, a.xsb, a.xsl, xsd) || !rows_ok(dtype, a.dy, a.gsb, a.gsl, gsd) || ysd != 1 || a.h_in ||
      a.h_out)
    return false;
  return dispatch<true>(dtype, a, s);
}

}  // namespace mega
