// The poles of a channel in the registers of a lane (scan_ema.cu, scan_cluster.cu).
#pragma once
#include "common.cuh"
#include "norm_run.cuh"
#include "scan_ema.cuh"
#include "tma.cuh"

namespace mega {

namespace {

constexpr int kP2 = 8;      // pole pairs of a lane (16 poles)

// One pole-state vector: real parts, and imaginary parts for complex poles.
template <bool kC>
struct State {
  f32x2 r[kP2];
  f32x2 i[kC ? kP2 : 1];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int j = 0; j < kP2; ++j) {
      r[j] = pack2(0.f, 0.f);
      if (kC) i[j] = pack2(0.f, 0.f);
    }
  }
};

// Poles of a lane's channel.  q; ni = -Im q; c (and nc = -Im c): output weight.
template <bool kC>
struct Poles {
  f32x2 q[kP2];
  f32x2 qi[kC ? kP2 : 1], ni[kC ? kP2 : 1];
};

template <bool kC>
__device__ __forceinline__ void load_poles(Poles<kC>& P, const ScanArgs& a, int row) {
#pragma unroll
  for (int j = 0; j < kP2; ++j) {
    float qr[2], qi[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int n = 2 * j + k;
      const size_t c = (size_t)row * a.N + n;
      qr[k] = qi[k] = 0.f;
      if (n < a.N) {
        qr[k] = kC ? __ldg(a.q + 2 * c) : __ldg(a.q + c);
        if (kC) qi[k] = __ldg(a.q + 2 * c + 1);
      }
    }
    P.q[j] = pack2(qr[0], qr[1]);
    if (kC) {
      P.qi[j] = pack2(qi[0], qi[1]);
      P.ni[j] = pack2(-qi[0], -qi[1]);
    }
  }
}

// Output weights p gamma (kGain) or gamma alone; the imaginary part negated (y = Re(c h) = cr hr - ci hi).
template <bool kC>
__device__ __forceinline__ void load_weights(State<kC>& C, const ScanArgs& a, int row, bool gain) {
#pragma unroll
  for (int j = 0; j < kP2; ++j) {
    float cr[2], ci[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int n = 2 * j + k;
      const size_t c = (size_t)row * a.N + n;
      cr[k] = ci[k] = 0.f;
      if (n < a.N) {
        const float p = gain ? __ldg(a.p + c) : 1.f;
        cr[k] = p * (kC ? __ldg(a.g + 2 * c) : __ldg(a.g + c));
        if (kC) ci[k] = -p * __ldg(a.g + 2 * c + 1);
      }
    }
    C.r[j] = pack2(cr[0], cr[1]);
    if (kC) C.i[j] = pack2(ci[0], ci[1]);
  }
}

// h <- q h + x
template <bool kC>
__device__ __forceinline__ void advance(State<kC>& h, const Poles<kC>& P, f32x2 x2) {
#pragma unroll
  for (int j = 0; j < kP2; ++j) {
    if (kC) {
      const f32x2 nr = fma2(P.q[j], h.r[j], fma2(P.ni[j], h.i[j], x2));
      h.i[j] = fma2(P.qi[j], h.r[j], mul2(P.q[j], h.i[j]));
      h.r[j] = nr;
    } else {
      h.r[j] = fma2(P.q[j], h.r[j], x2);
    }
  }
}
// h <- q h + p x
template <bool kC>
__device__ __forceinline__ void advance_gain(State<kC>& h, const Poles<kC>& P, const f32x2 (&p)[kP2], f32x2 x2) {
#pragma unroll
  for (int j = 0; j < kP2; ++j) {
    const f32x2 in = mul2(p[j], x2);
    if (kC) {
      const f32x2 nr = fma2(P.q[j], h.r[j], fma2(P.ni[j], h.i[j], in));
      h.i[j] = fma2(P.qi[j], h.r[j], mul2(P.q[j], h.i[j]));
      h.r[j] = nr;
    } else {
      h.r[j] = fma2(P.q[j], h.r[j], in);
    }
  }
}
// s <- q s + h (h before its own step)
template <bool kC>
__device__ __forceinline__ void advance_sens(State<kC>& s, const State<kC>& h, const Poles<kC>& P) {
#pragma unroll
  for (int j = 0; j < kP2; ++j) {
    if (kC) {
      const f32x2 nr = fma2(P.q[j], s.r[j], fma2(P.ni[j], s.i[j], h.r[j]));
      s.i[j] = fma2(P.qi[j], s.r[j], fma2(P.q[j], s.i[j], h.i[j]));
      s.r[j] = nr;
    } else {
      s.r[j] = fma2(P.q[j], s.r[j], h.r[j]);
    }
  }
}
// Re(sum c h)
template <bool kC>
__device__ __forceinline__ float dot(const State<kC>& c, const State<kC>& h) {
  f32x2 a0 = pack2(0.f, 0.f), a1 = pack2(0.f, 0.f);
#pragma unroll
  for (int j = 0; j < kP2; j += 2) {
    a0 = fma2(c.r[j], h.r[j], a0);
    a1 = fma2(c.r[j + 1], h.r[j + 1], a1);
    if (kC) {
      a0 = fma2(c.i[j], h.i[j], a0);
      a1 = fma2(c.i[j + 1], h.i[j + 1], a1);
    }
  }
  float lo, hi;
  unpack2(add2(a0, a1), lo, hi);
  return lo + hi;
}
// acc += dy h
template <bool kC>
__device__ __forceinline__ void accumulate(State<kC>& acc, const State<kC>& h, f32x2 g2) {
#pragma unroll
  for (int j = 0; j < kP2; ++j) {
    acc.r[j] = fma2(g2, h.r[j], acc.r[j]);
    if (kC) acc.i[j] = fma2(g2, h.i[j], acc.i[j]);
  }
}

__device__ __forceinline__ f32x2 splat(float v) { return pack2(v, v); }

// the normalised input (0 at a padded position)
__device__ __forceinline__ float normed(Running& st, float x, bool pad, float w, float bb, float eps) {
  if (pad) return 0.f;
  float inv, r;
  const float d = st.step(x, eps, inv, r);
  return fmaf((d - st.u) * r, w, bb);
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ float2 ipow(float2 q, int n) {
  float2 r = make_float2(1.f, 0.f);
  for (; n > 0; n >>= 1) {
    if (n & 1) r = cmul(r, q);
    q = cmul(q, q);
  }
  return r;
}

}  // namespace

}  // namespace mega
