// Running statistics of TimestepNorm as the kernels that are parallel over time take them (scan_norm.cu, scan_ema.cu):
// the moments of segments, their combination, and a walk's update.
#pragma once
#include "common.cuh"
#include "walk.cuh"

namespace mega {

namespace {

// count, mean, squared deviations (Chan et al.'s pairwise combination)
struct Run {
  float n, m, s;
};
__device__ __forceinline__ Run combine(Run a, Run b) {
  const float n = a.n + b.n;
  if (b.n == 0.f) return a;
  if (a.n == 0.f) return b;
  const float w = b.n * rcp_approx(n), d = b.m - a.m;
  return {n, fmaf(d, w, a.m), a.s + b.s + d * d * a.n * w};
}

// The statistics of a walk, advanced by one unmasked input.  The walk's own steps are counted from zero: added one by one
// to a count beyond 2^24 they would be lost.
struct Running {
  float c, s1, s2, n0, in_s;   // centre, sums about it, count and squared deviations that came in
  float seen, n;               // steps of the walk, count
  float u;                     // mean - c
  __device__ __forceinline__ void start(const Run& r) {
    c = r.m;
    s1 = s2 = u = seen = 0.f;
    n0 = n = r.n;
    in_s = r.s;
  }
  // returns x - c; inv = 1 / n, r = 1 / sqrt(var + eps)
  __device__ __forceinline__ float step(float x, float eps, float& inv, float& r) {
    if (n == 0.f) c = x;
    const float d = x - c;
    s1 += d;
    s2 = fmaf(d, d, s2);
    seen += 1.f;
    n = n0 + seen;
    inv = rcp_approx(n);
    u = s1 * inv;
    r = rsqrt_approx(fmaxf(fmaf(-u, u, (in_s + s2) * inv), 0.f) + eps);
    return d;
  }
};

// The moments of every segment of T steps: unmasked steps rn (B, S), mean rm and squared deviations rs (B, S, D).
// Sums about the mean of the first 32 steps, 32 steps at a time: about the segment's first value, and one step after the
// other, the variance of 5000 steps was 1.9e-6 off its own size, further than a step-by-step Welford update (1.2e-6).
struct MomentArgs {
  const void* x;
  long long xsb, xsl;
  const unsigned char* mask;
  int L, D, T, S;
  float *rn, *rm, *rs;
};

template <typename T, bool kMask>
__global__ void __launch_bounds__(kWarps * 32) norm_moments_kernel(MomentArgs s) {
  extern __shared__ __align__(16) unsigned char rings[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int d0 = blockIdx.x * 32, seg = blockIdx.y * kWarps + warp, b = blockIdx.z;
  if (seg >= s.S) return;
  const int t0 = min(s.L, seg * s.T), t1 = min(s.L, t0 + s.T);
  const T* x = reinterpret_cast<const T*>(s.x) + b * s.xsb + d0;
  const unsigned char* m = kMask ? s.mask + (size_t)b * s.L : nullptr;
  float c = 0.f, s1 = 0.f, s2 = 0.f, n = 0.f, p1 = 0.f, p2 = 0.f;   // p1, p2: of the present 32 steps
  walk<T, 1, false, kMask>(x, s.xsl, x, 0, m, t0, t1, s.D - d0, rings + (size_t)warp * kRing * kTileBytes,
                           [&](int k, float xv, float, bool pad) {
                             if (!(kMask && pad)) {
                               if (kMask ? n == 0.f : k == 0) c = xv;
                               const float d = xv - c;
                               p1 += d;
                               p2 = fmaf(d, d, p2);
                               if (kMask) n += 1.f;
                             }
                             if ((k & 31) == 31) {
                               if (k == 31) {   // (from here on about their mean)
                                 const float n32 = kMask ? n : 32.f, to = n32 > 0.f ? c + p1 / n32 : c, e = to - c;
                                 p2 = fmaf(e, fmaf(n32, e, -2.f * p1), p2);
                                 p1 = fmaf(-n32, e, p1);
                                 c = to;
                               }
                               s1 += p1;
                               s2 += p2;
                               p1 = p2 = 0.f;
                             }
                           });
  s1 += p1;
  s2 += p2;
  if (!kMask) n = (float)(t1 - t0);
  const float inv = n > 0.f ? 1.f / n : 0.f;
  const int d = d0 + lane;
  const size_t i = ((size_t)b * s.S + seg) * s.D + d;
  if (d < s.D) {
    s.rm[i] = fmaf(s1, inv, c);
    s.rs[i] = not_negative(fmaf(-s1 * inv, s1, s2));
  }
  if (blockIdx.x == 0 && lane == 0) s.rn[(size_t)b * s.S + seg] = n;
}

}  // namespace

}  // namespace mega
