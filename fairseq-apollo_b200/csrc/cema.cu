// Complex EMA layer (MultiHeadComplexEMA): poles q_n = r_n e^{i theta_n}, real input gain p_n,
// complex output weights gamma_n.  h_t = q h_{t-1} + p x_t (complex state), y_t = Re(sum_n gamma_n
// h_{n,t}) + omega x_t.  Evaluated as the recurrence itself: O(L) per row, one pass over x, no
// length cap.  Four lanes share a (batch, channel) row and split its poles; the per-step output is
// a two-shuffle reduction.
#include "chunk_ema.cuh"
#include "common.cuh"
#include "stream_bwd.cuh"
#include "stream_cl.cuh"
#include "block_step.cuh"
#include "norm_ema_split.cuh"
#include "scan_cluster.cuh"
#include "scan_ema.cuh"

namespace mega {

// theta_n = (n + 1) sigmoid(theta) 2 pi / N ; r = 1 - sigmoid(alpha) sigmoid(delta) ;
// p = sigmoid(alpha) ; gamma_hat = gamma / sqrt(N)
template <typename T>
__global__ void cema_coeffs_kernel(const T* __restrict__ alpha, const T* __restrict__ delta,
                                   const T* __restrict__ theta, const T* __restrict__ gamma, int K, int N,
                                   float scale, float* __restrict__ p, float* __restrict__ q,
                                   float* __restrict__ g) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= K * N) return;
  const int k = i / N, n = i % N;
  const float a = 1.0f / (1.0f + expf(-Elem<T>::ld(alpha + i)));
  const float d = 1.0f / (1.0f + expf(-Elem<T>::ld(delta + i)));
  const float th = 1.0f / (1.0f + expf(-Elem<T>::ld(theta + k))) * (6.283185307179586f / (float)N) * (float)(n + 1);
  const float r = 1.0f - a * d;
  float sn, cs;
  sincosf(th, &sn, &cs);
  p[i] = a;
  q[2 * i] = r * cs;
  q[2 * i + 1] = r * sn;
  g[2 * i] = Elem<T>::ld(gamma + 2 * i) * scale;
  g[2 * i + 1] = Elem<T>::ld(gamma + 2 * i + 1) * scale;
}

// k[row, l] = Re(sum_n p gamma q^l), through the polar form of q
__global__ void cema_kernel_kernel(const float* __restrict__ p, const float* __restrict__ q,
                                   const float* __restrict__ g, int N, int L, float* __restrict__ out) {
  extern __shared__ float sm[];  // [N] x {p*gr, p*gi, log r, arg}
  const int r = blockIdx.y;
  for (int n = threadIdx.x; n < N; n += blockDim.x) {
    const float qr = q[2 * (r * N + n)], qi = q[2 * (r * N + n) + 1];
    const float pn = p[r * N + n];
    sm[4 * n + 0] = pn * g[2 * (r * N + n)];
    sm[4 * n + 1] = pn * g[2 * (r * N + n) + 1];
    const float mag = sqrtf(qr * qr + qi * qi);
    sm[4 * n + 2] = mag > 0.f ? logf(mag) : -1e30f;
    sm[4 * n + 3] = atan2f(qi, qr);
  }
  __syncthreads();
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= L) return;
  float acc = 0.f;
  for (int n = 0; n < N; ++n) {
    const float m = l == 0 ? 1.f : expf((float)l * sm[4 * n + 2]);
    float sn, cs;
    sincosf((float)l * sm[4 * n + 3], &sn, &cs);
    acc += m * (sm[4 * n + 0] * cs - sm[4 * n + 1] * sn);
  }
  out[(size_t)r * L + l] = acc;
}

struct CemaArgs {
  const void* x;
  void* y;
  int B, D, L, N;
  long long xsb, xsd, xsl, ysb, ysd, ysl;
  const float *p, *q, *g, *omega;  // q, g interleaved (re, im)
  const unsigned char* mask;
  const float* h_in;  // (B, D, N, 2) or NULL
  float* h_out;
  int ksize;  // kernel support; >= L when not truncated
  int bidir, shift, silu;
};

// q^k for a complex q by repeated squaring
__device__ __forceinline__ void cpow(float qr, float qi, int k, float& outr, float& outi) {
  float rr = 1.f, ri = 0.f;
  while (k > 0) {
    if (k & 1) {
      const float t = rr * qr - ri * qi;
      ri = rr * qi + ri * qr;
      rr = t;
    }
    const float t = qr * qr - qi * qi;
    qi = 2.f * qr * qi;
    qr = t;
    k >>= 1;
  }
  outr = rr;
  outi = ri;
}

template <typename T, int NP, bool kTrunc, bool kMask>
__global__ void __launch_bounds__(128) cema_scan_kernel(CemaArgs a) {
  constexpr int U = 4;
  const int sub = threadIdx.x & 3;
  const long long row = (long long)blockIdx.x * 32 + (threadIdx.x >> 2);
  const bool live = row < (long long)a.B * a.D;  // dead rows keep running for the shuffles
  const int d = live ? (int)(row % a.D) : 0;
  const int b = live ? (int)(row / a.D) : 0;
  const int L = a.L;
  const T* xp = reinterpret_cast<const T*>(a.x) + b * a.xsb + d * a.xsd;
  T* yp = reinterpret_cast<T*>(a.y) + b * a.ysb + d * a.ysd;
  const unsigned char* mp = kMask ? a.mask + (size_t)b * L : nullptr;  // compile-time: see ema_scan_rows_kernel
  const float om = __ldg(a.omega + d);
  const size_t srow = ((size_t)b * a.D + d) * a.N;

  for (int half = 0; half < (a.bidir ? 2 : 1); ++half) {
    const bool rev = half == 1;
    const bool pre_output = rev && a.shift;  // anti-causal half starting at lag 1: emit, then update
    const bool last = half == (a.bidir ? 1 : 0);
    const size_t prow = (size_t)(d + half * a.D) * a.N;
    float pp[NP], qr[NP], qi[NP], gr[NP], gi[NP], hr[NP], hi[NP], wr[kTrunc ? NP : 1], wi[kTrunc ? NP : 1];
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      const int n = k * 4 + sub;
      const bool ok = n < a.N;
      pp[k] = ok ? __ldg(a.p + prow + n) : 0.f;
      qr[k] = ok ? __ldg(a.q + 2 * (prow + n)) : 0.f;
      qi[k] = ok ? __ldg(a.q + 2 * (prow + n) + 1) : 0.f;
      gr[k] = ok ? __ldg(a.g + 2 * (prow + n)) : 0.f;
      gi[k] = ok ? __ldg(a.g + 2 * (prow + n) + 1) : 0.f;
      const bool hin = ok && live && a.h_in != nullptr;
      hr[k] = hin ? __ldg(a.h_in + 2 * (srow + n)) : 0.f;
      hi[k] = hin ? __ldg(a.h_in + 2 * (srow + n) + 1) : 0.f;
      if (kTrunc) {  // p q^ksize: what a sample leaving the window still contributes
        cpow(qr[k], qi[k], a.ksize, wr[k], wi[k]);
        wr[k] *= pp[k];
        wi[k] *= pp[k];
      }
    }
    for (int u0 = 0; u0 < L; u0 += U) {
      float xv[U], xm[U], xd[U], old[U];
#pragma unroll
      for (int j = 0; j < U; ++j) {
        const int u = u0 + j;
        xv[j] = xm[j] = xd[j] = old[j] = 0.f;
        if (u < L && live) {
          const int t = rev ? L - 1 - u : u;
          xv[j] = Elem<T>::ld(xp + t * a.xsl);
          xm[j] = (kMask && __ldg(mp + t) != 0) ? 0.f : xv[j];
          if (kTrunc) {
            const int td = rev ? t + a.ksize : t - a.ksize;
            if (td >= 0 && td < L && !(kMask && __ldg(mp + td) != 0)) xd[j] = Elem<T>::ld(xp + td * a.xsl);
          }
          if (half == 1 && sub == 0) old[j] = Elem<T>::ld_shared(yp + t * a.ysl);  // written by the first half
        }
      }
#pragma unroll
      for (int j = 0; j < U; ++j) {
        const int u = u0 + j;
        if (u < L) {
          float part = 0.f;
#pragma unroll
          for (int k = 0; k < NP; ++k) {
            if (pre_output) part += gr[k] * hr[k] - gi[k] * hi[k];
            float nr = fmaf(qr[k], hr[k], fmaf(-qi[k], hi[k], pp[k] * xm[j]));
            float ni = fmaf(qi[k], hr[k], qr[k] * hi[k]);
            if (kTrunc) {
              nr = fmaf(-wr[k], xd[j], nr);
              ni = fmaf(-wi[k], xd[j], ni);
            }
            hr[k] = nr;
            hi[k] = ni;
            if (!pre_output) part += gr[k] * nr - gi[k] * ni;
          }
          part += __shfl_xor_sync(0xffffffffu, part, 1);
          part += __shfl_xor_sync(0xffffffffu, part, 2);
          if (live && sub == 0) {
            const int t = rev ? L - 1 - u : u;
            float v = half == 0 ? fmaf(om, xv[j], part) : old[j] + part;
            if (last && a.silu) v = siluf_(v);
            Elem<T>::st(yp + t * a.ysl, v);
          }
        }
      }
    }
    if (half == 0 && a.h_out && live) {
#pragma unroll
      for (int k = 0; k < NP; ++k) {
        const int n = k * 4 + sub;
        if (n < a.N) {
          a.h_out[2 * (srow + n)] = hr[k];
          a.h_out[2 * (srow + n) + 1] = hi[k];
        }
      }
    }
  }
}

// Decode step: one thread per (batch, channel); state read and written once.
template <typename T>
__global__ void __launch_bounds__(128) cema_step_kernel(const T* x, T* y, int B, int D, int N, const float* p,
                                                        const float* q, const float* g, const float* omega,
                                                        const float* h_in, float* h_out, int silu) {
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (long long)B * D) return;
  const int d = (int)(gid % D);
  const float xv = Elem<T>::ld(x + gid);
  float acc = 0.f;
  for (int n = 0; n < N; ++n) {
    const size_t c = (size_t)d * N + n, s = (size_t)gid * N + n;
    const float qr = __ldg(q + 2 * c), qi = __ldg(q + 2 * c + 1);
    const float hr = h_in ? h_in[2 * s] : 0.f, hi = h_in ? h_in[2 * s + 1] : 0.f;
    const float nr = fmaf(qr, hr, fmaf(-qi, hi, __ldg(p + c) * xv));
    const float ni = fmaf(qi, hr, qr * hi);
    h_out[2 * s] = nr;
    h_out[2 * s + 1] = ni;
    acc += __ldg(g + 2 * c) * nr - __ldg(g + 2 * c + 1) * ni;
  }
  float v = fmaf(__ldg(omega + d), xv, acc);
  if (silu) v = siluf_(v);
  Elem<T>::st(y + gid, v);
}

// The same step with LN = N / 2 lanes per (batch, channel): a lane owns two complex poles (one
// 16-byte state vector), so a warp moves whole contiguous state rows, and a thread walks BB
// batch entries with its coefficients in registers.  h_in may be NULL and may alias h_out.
// With use_norm the TimestepNorm update of the token runs first (redundantly in the LN lanes;
// lane 0 stores the statistics), as in the real layer's step kernel.
template <typename T, int LN, int BB, bool kAfter>
__global__ void __launch_bounds__(128) cema_step_lanes_kernel(const T* __restrict__ x, T* __restrict__ y,
                                                              T* __restrict__ xn_out, int B, int D,
                                                              const long long* count, float* mean, float* var,
                                                              const float* __restrict__ gamma,
                                                              const float* __restrict__ beta, float eps,
                                                              const float* __restrict__ p,
                                                              const float* __restrict__ q,
                                                              const float* __restrict__ g,
                                                              const float* __restrict__ omega, const float* h_in,
                                                              float* h_out, int silu, int use_norm,
                                                              long long* count_next) {
  if (kAfter) {   // (in the step of a block; the next launch may begin once all that came before this one is done)
    pdl_wait();
    pdl_next();
  }
  constexpr int N = LN * 2;
  const int sub = threadIdx.x % LN;
  const int d = blockIdx.x * (128 / LN) + threadIdx.x / LN;
  const bool live = d < D;  // dead lanes stay for the shuffles
  const int b0 = blockIdx.y * BB;
  float4 qv = make_float4(0.f, 0.f, 0.f, 0.f), gv = qv;
  float2 pv = make_float2(0.f, 0.f);
  float om = 0.f, gam = 1.f, bet = 0.f;
  if (live) {
    qv = __ldg(reinterpret_cast<const float4*>(q + (size_t)d * N * 2) + sub);
    gv = __ldg(reinterpret_cast<const float4*>(g + (size_t)d * N * 2) + sub);
    pv = __ldg(reinterpret_cast<const float2*>(p + (size_t)d * N) + sub);
    om = __ldg(omega + d);
    if (use_norm) {
      gam = __ldg(gamma + d);
      bet = __ldg(beta + d);
    }
  }
  float4 hv[BB];
  float xv[BB], mu[BB], vr[BB], coef[BB];
#pragma unroll
  for (int j = 0; j < BB; ++j) {
    const int b = b0 + j;
    const size_t gid = (size_t)b * D + d;
    hv[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    xv[j] = mu[j] = 0.f;
    vr[j] = coef[j] = 1.f;
    if (live && b < B) {
      if (h_in) hv[j] = *(reinterpret_cast<const float4*>(h_in + gid * N * 2) + sub);
      xv[j] = Elem<T>::ld(x + gid);
      if (use_norm) {
        mu[j] = mean[gid];
        vr[j] = var[gid];
        coef[j] = __frcp_rn((float)(count[b] + 1));
      }
    }
  }
#pragma unroll
  for (int j = 0; j < BB; ++j) {
    const int b = b0 + j;
    const size_t gid = (size_t)b * D + d;
    float xin = xv[j];
    float m1 = 0.f, m2 = 0.f;
    if (use_norm) {
      const float d1 = xin - mu[j];
      m1 = fmaf(coef[j], d1, mu[j]);
      const float d2 = fmaf(d1, xin - m1, -vr[j]);
      m2 = fmaf(coef[j], d2, vr[j]);
      xin = fmaf((xin - m1) * rsqrtf(m2 + eps), gam, bet);
    }
    const float4 h = hv[j];
    float4 hn;
    hn.x = fmaf(qv.x, h.x, fmaf(-qv.y, h.y, pv.x * xin));
    hn.y = fmaf(qv.y, h.x, qv.x * h.y);
    hn.z = fmaf(qv.z, h.z, fmaf(-qv.w, h.w, pv.y * xin));
    hn.w = fmaf(qv.w, h.z, qv.z * h.w);
    float acc = (gv.x * hn.x - gv.y * hn.y) + (gv.z * hn.z - gv.w * hn.w);
#pragma unroll
    for (int o = 1; o < LN; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (live && b < B) {
      *(reinterpret_cast<float4*>(h_out + gid * N * 2) + sub) = hn;
      if (sub == 0) {
        float v = fmaf(om, xin, acc);
        if (silu) v = siluf_(v);
        Elem<T>::st(y + gid, v);
        if (use_norm) {
          mean[gid] = m1;
          var[gid] = m2;
          if (xn_out) Elem<T>::st(xn_out + gid, xin);
        }
      }
    }
  }
  // the counts after this step go to a second array (never the one every CTA is reading)
  if (count_next && d == 0 && sub == 0) {
#pragma unroll
    for (int j = 0; j < BB; ++j)
      if (b0 + j < B) count_next[b0 + j] = count[b0 + j] + 1;
  }
}

// One thread per sequence bumps the counts after the element kernel has read them.
__global__ void cema_count_step_kernel(long long* count, int B) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < B) count[b] += 1;
}

template <typename T>
static bool launch_cema_step_lanes(const T* x, T* y, T* xn_out, int B, int D, int N, const long long* count,
                                   float* mean, float* var, const float* gamma, const float* beta, float eps,
                                   const float* p, const float* q, const float* g, const float* omega,
                                   const float* h_in, float* h_out, int silu, void* stream,
                                   long long* count_next = nullptr, bool after = false) {
  const int use_norm = count != nullptr;
  if (N != 2 && N != 4 && N != 8 && N != 16 && N != 32) return false;
  if (!aligned_to(h_out, 16) || (h_in && !aligned_to(h_in, 16)) || !aligned_to(p, 8) || !aligned_to(q, 16) ||
      !aligned_to(g, 16))
    return false;
  constexpr int BB = 4;
  const int ln = N / 2;
  dim3 grid((unsigned)((D + 128 / ln - 1) / (128 / ln)), (unsigned)((B + BB - 1) / BB));
  if (grid.y > 65535) return false;
#define MEGA_CEMA_STEP_LANES(LNV) \
  do {                                                                                                    \
    if (after)                                                                                            \
      launch_after(cema_step_lanes_kernel<T, LNV, BB, true>, grid, 128, 0, stream, x, y, xn_out, B, D, count, mean, var, gamma, \
         beta, eps, p, q, g, omega, h_in, h_out, silu, use_norm, count_next);   \
    else                                                                                                  \
      launch(cema_step_lanes_kernel<T, LNV, BB, false>, grid, 128, 0, stream, x, y, xn_out, B, D, count, mean, var, gamma, \
         beta, eps, p, q, g, omega, h_in, h_out, silu, use_norm, count_next);        \
  } while (0)
  if (ln == 1) MEGA_CEMA_STEP_LANES(1);
  else if (ln == 2) MEGA_CEMA_STEP_LANES(2);
  else if (ln == 4) MEGA_CEMA_STEP_LANES(4);
  else if (ln == 8) MEGA_CEMA_STEP_LANES(8);
  else MEGA_CEMA_STEP_LANES(16);
#undef MEGA_CEMA_STEP_LANES
  return true;
}

bool cema_step_lanes_try(int dtype, const void* x, void* y, void* xn_out, int B, int D, int N, const long long* count,
                         float* mean, float* var, const float* gamma, const float* beta, float eps, const float* p,
                         const float* q, const float* g, const float* omega, const float* h_in, float* h_out, int silu,
                         void* stream, long long* count_next, bool after) {
  switch (dtype) {
#define MEGA_CEMA_STEP_CASE(DT, TY)                                                                                    \
  case DT:                                                                                                             \
    return launch_cema_step_lanes<TY>((const TY*)x, (TY*)y, (TY*)xn_out, B, D, N, count, mean, var, gamma, beta, eps,  \
                                      p, q, g, omega, h_in, h_out, silu, stream, count_next, after);
    MEGA_CEMA_STEP_CASE(MEGA_F32, float)
    MEGA_CEMA_STEP_CASE(MEGA_BF16, __nv_bfloat16)
    MEGA_CEMA_STEP_CASE(MEGA_F16, __half)
#undef MEGA_CEMA_STEP_CASE
    default: return false;
  }
}

// ---------------------------------------------------------------------------------------------
// backward of the complex layer.  h is holomorphic in q and linear in p, so with the complex
// sensitivities s = dh/dq (s_t = q s_{t-1} + h_{t-1}) and r = dh/dp (r_t = q r_{t-1} + x_t):
//   dL/dp = Re(gamma sum_t dy_t r_t),  dL/dq_re = Re(gamma sum_t dy_t s_t),  dL/dq_im = -Im(same),
//   dL/dgamma_re = sum_t dy_t Re h_t,  dL/dgamma_im = -sum_t dy_t Im h_t,
// and the input gradient is dx_t = sum_n p_n Re(lambda_{n,t}), lambda_t = gamma dy_t + q lambda_{t+1}.
// Same structure as the real layer's kernel: four lanes per (batch, channel) row, no stored history.
// ---------------------------------------------------------------------------------------------
struct CemaBwdArgs {
  const void *dy, *x;
  void* dx;
  int B, D, L, N;
  long long gsb, gsd, gsl, xsb, xsd, xsl, dsb, dsd, dsl;
  const float *p, *q, *g, *omega;
  const unsigned char* mask;
  float *dp, *dq, *dg, *domega;
  int bidir, shift;
  int ksize;  // kTrunc: support of the truncated kernel
};

// kTrunc: sliding-window states as in the real layer's backward kernel, with complex
// Q = q^ksize: h, r take x~_t - Q x~_{t-ksize}, s loses p ksize q^(ksize-1) x~_{t-ksize}, and
// lambda takes g dy_t - (g Q) dy_{t+ksize}.
template <typename T, int NP, bool kMask, bool kTrunc>
__global__ void __launch_bounds__(128) cema_bwd_kernel(CemaBwdArgs a) {
  constexpr int U = 8;
  const int sub = threadIdx.x & 3;
  const long long row = (long long)blockIdx.x * 32 + (threadIdx.x >> 2);
  const bool live = row < (long long)a.B * a.D;
  const int d = live ? (int)(row % a.D) : 0;
  const int b = live ? (int)(row / a.D) : 0;
  const int L = a.L;
  const T* xp = reinterpret_cast<const T*>(a.x) + b * a.xsb + d * a.xsd;
  const T* gp = reinterpret_cast<const T*>(a.dy) + b * a.gsb + d * a.gsd;
  T* dxp = reinterpret_cast<T*>(a.dx) + b * a.dsb + d * a.dsd;
  const unsigned char* mp = kMask ? a.mask + (size_t)b * L : nullptr;
  const float om = __ldg(a.omega + d);
  float aw = 0.f;

  for (int half = 0; half < (a.bidir ? 2 : 1); ++half) {
    const bool rev = half == 1;
    const bool shift = rev && a.shift;
    const size_t prow = (size_t)(d + half * a.D) * a.N;
    float pp[NP], qr[NP], qi[NP], gr[NP], gi[NP];
    float hr[NP], hi[NP], sr[NP], si[NP], rr[NP], ri[NP];
    float ahr[NP], ahi[NP], asr[NP], asi[NP], arr[NP], ari[NP];
    constexpr int NT = kTrunc ? NP : 1;
    float qwr[NT], qwi[NT], tqr[NT], tqi[NT], gqr[NT], gqi[NT];  // Q, p ksize q^(ksize-1), g Q
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      const int n = k * 4 + sub;
      const bool ok = n < a.N;
      pp[k] = ok ? __ldg(a.p + prow + n) : 0.f;
      qr[k] = ok ? __ldg(a.q + 2 * (prow + n)) : 0.f;
      qi[k] = ok ? __ldg(a.q + 2 * (prow + n) + 1) : 0.f;
      gr[k] = ok ? __ldg(a.g + 2 * (prow + n)) : 0.f;
      gi[k] = ok ? __ldg(a.g + 2 * (prow + n) + 1) : 0.f;
      if (kTrunc) {
        const float rho = hypotf(qr[k], qi[k]);
        float m1r = 0.f, m1i = 0.f;  // q^(ksize-1)
        if (rho > 0.f) {
          const float mag = expf((float)(a.ksize - 1) * logf(rho));
          float sn, cs;
          sincosf((float)(a.ksize - 1) * atan2f(qi[k], qr[k]), &sn, &cs);
          m1r = mag * cs;
          m1i = mag * sn;
        }
        qwr[k] = m1r * qr[k] - m1i * qi[k];
        qwi[k] = m1r * qi[k] + m1i * qr[k];
        tqr[k] = pp[k] * (float)a.ksize * m1r;
        tqi[k] = pp[k] * (float)a.ksize * m1i;
        gqr[k] = gr[k] * qwr[k] - gi[k] * qwi[k];
        gqi[k] = gr[k] * qwi[k] + gi[k] * qwr[k];
      }
      hr[k] = hi[k] = sr[k] = si[k] = rr[k] = ri[k] = 0.f;
      ahr[k] = ahi[k] = asr[k] = asi[k] = arr[k] = ari[k] = 0.f;
    }
    for (int u0 = 0; u0 < L; u0 += U) {
      float xv[U], gv[U], xd[kTrunc ? U : 1];
#pragma unroll
      for (int j = 0; j < U; ++j) {
        const int u = u0 + j;
        xv[j] = gv[j] = 0.f;
        if (kTrunc) xd[j] = 0.f;
        if (u < L && live) {
          const int t = rev ? L - 1 - u : u;
          const float xt = Elem<T>::ld(xp + t * a.xsl);
          gv[j] = Elem<T>::ld(gp + t * a.gsl);
          if (half == 0) aw = fmaf(gv[j], xt, aw);
          xv[j] = (kMask && __ldg(mp + t) != 0) ? 0.f : xt;
          if (kTrunc && u >= a.ksize) {  // the sample leaving the window
            const int td = rev ? t + a.ksize : t - a.ksize;
            if (!(kMask && __ldg(mp + td) != 0)) xd[j] = Elem<T>::ld(xp + td * a.xsl);
          }
        }
      }
#pragma unroll
      for (int j = 0; j < U; ++j) {
        if (u0 + j < L) {
          const float dy = gv[j], xm = xv[j];
          const float xo = kTrunc ? xd[j] : 0.f;
#pragma unroll
          for (int k = 0; k < NP; ++k) {
            if (shift) {
              ahr[k] = fmaf(dy, hr[k], ahr[k]); ahi[k] = fmaf(dy, hi[k], ahi[k]);
              asr[k] = fmaf(dy, sr[k], asr[k]); asi[k] = fmaf(dy, si[k], asi[k]);
              arr[k] = fmaf(dy, rr[k], arr[k]); ari[k] = fmaf(dy, ri[k], ari[k]);
            }
            float nsr = fmaf(qr[k], sr[k], fmaf(-qi[k], si[k], hr[k]));
            float nsi = fmaf(qi[k], sr[k], fmaf(qr[k], si[k], hi[k]));
            float nhr = fmaf(qr[k], hr[k], fmaf(-qi[k], hi[k], pp[k] * xm));
            float nhi = fmaf(qi[k], hr[k], qr[k] * hi[k]);
            float nrr = fmaf(qr[k], rr[k], fmaf(-qi[k], ri[k], xm));
            float nri = fmaf(qi[k], rr[k], qr[k] * ri[k]);
            if (kTrunc) {
              nsr = fmaf(-tqr[k], xo, nsr);
              nsi = fmaf(-tqi[k], xo, nsi);
              nhr = fmaf(-pp[k] * qwr[k], xo, nhr);
              nhi = fmaf(-pp[k] * qwi[k], xo, nhi);
              nrr = fmaf(-qwr[k], xo, nrr);
              nri = fmaf(-qwi[k], xo, nri);
            }
            sr[k] = nsr; si[k] = nsi; hr[k] = nhr; hi[k] = nhi; rr[k] = nrr; ri[k] = nri;
            if (!shift) {
              ahr[k] = fmaf(dy, nhr, ahr[k]); ahi[k] = fmaf(dy, nhi, ahi[k]);
              asr[k] = fmaf(dy, nsr, asr[k]); asi[k] = fmaf(dy, nsi, asi[k]);
              arr[k] = fmaf(dy, nrr, arr[k]); ari[k] = fmaf(dy, nri, ari[k]);
            }
          }
        }
      }
    }
    float lr[NP], li[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      const int n = k * 4 + sub;
      lr[k] = li[k] = 0.f;
      if (n < a.N && live) {
        atomicAdd(a.dg + 2 * (prow + n), ahr[k]);
        atomicAdd(a.dg + 2 * (prow + n) + 1, -ahi[k]);
        atomicAdd(a.dp + prow + n, gr[k] * arr[k] - gi[k] * ari[k]);
        atomicAdd(a.dq + 2 * (prow + n), gr[k] * asr[k] - gi[k] * asi[k]);
        atomicAdd(a.dq + 2 * (prow + n) + 1, -(gr[k] * asi[k] + gi[k] * asr[k]));
      }
    }
    for (int u0 = L - 1; u0 >= 0; u0 -= U) {
      float gv[U], old[U], gd[kTrunc ? U : 1];
      bool mk[U];
#pragma unroll
      for (int j = 0; j < U; ++j) {
        const int u = u0 - j;
        gv[j] = old[j] = 0.f;
        if (kTrunc) gd[j] = 0.f;
        mk[j] = false;
        if (u >= 0 && live) {
          const int t = rev ? L - 1 - u : u;
          gv[j] = Elem<T>::ld(gp + t * a.gsl);
          if (kTrunc && u + a.ksize < L) gd[j] = Elem<T>::ld(gp + (rev ? t - a.ksize : t + a.ksize) * a.gsl);
          mk[j] = kMask && __ldg(mp + t) != 0;
          if (half == 1 && sub == 0) old[j] = Elem<T>::ld_shared(dxp + t * a.dsl);  // written by the first half
        }
      }
#pragma unroll
      for (int j = 0; j < U; ++j) {
        const int u = u0 - j;
        if (u >= 0) {
          float part = 0.f;
#pragma unroll
          for (int k = 0; k < NP; ++k) {
            // g dy_t (- g Q dy_{t+ksize})
            float inr = gr[k] * gv[j], ini = gi[k] * gv[j];
            if (kTrunc) {
              inr = fmaf(-gqr[k], gd[j], inr);
              ini = fmaf(-gqi[k], gd[j], ini);
            }
            if (shift) {
              part = fmaf(pp[k], lr[k], part);
              const float nr = fmaf(qr[k], lr[k], fmaf(-qi[k], li[k], inr));
              const float ni = fmaf(qi[k], lr[k], fmaf(qr[k], li[k], ini));
              lr[k] = nr; li[k] = ni;
            } else {
              const float cr = lr[k] + inr, ci = li[k] + ini;
              part = fmaf(pp[k], cr, part);
              lr[k] = qr[k] * cr - qi[k] * ci;
              li[k] = qi[k] * cr + qr[k] * ci;
            }
          }
          part += __shfl_xor_sync(0xffffffffu, part, 1);
          part += __shfl_xor_sync(0xffffffffu, part, 2);
          if (live && sub == 0) {
            const int t = rev ? L - 1 - u : u;
            const float v = mk[j] ? 0.f : part;
            Elem<T>::st(dxp + t * a.dsl, half == 0 ? fmaf(om, gv[j], v) : old[j] + v);
          }
        }
      }
    }
  }
  if (live && sub == 0) atomicAdd(a.domega + d, aw);
}

// Chain rule to the raw parameters: rho = 1 - sigmoid(alpha) sigmoid(delta), phi_n = (n + 1)
// sigmoid(theta) 2 pi / N, q = rho e^{i phi}: dL/drho = G . e^{i phi}, dL/dphi = G . (i q) with
// G = (dL/dq_re, dL/dq_im) and "." the real dot product.  One thread per parameter row.
__global__ void cema_coeffs_bwd_kernel(const float* alpha, const float* delta, const float* theta, const float* q,
                                       const float* dp, const float* dq, const float* dg, int K, int N,
                                       float scale, float* dalpha, float* ddelta, float* dtheta, float* dgamma) {
  // (a warp per row, a lane per pole: a thread per row took 23 us at K = 1024)
  const int k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), n = threadIdx.x & 31;
  if (k >= K) return;
  const float st = 1.f / (1.f + __expf(-theta[k]));
  const float wave = 6.283185307179586f / (float)N;
  float dth = 0.f;
  if (n < N) {
    const int i = k * N + n;
    const float a = 1.f / (1.f + __expf(-alpha[i])), dl = 1.f / (1.f + __expf(-delta[i]));
    const float qr = q[2 * i], qi = q[2 * i + 1];
    const float rho = 1.f - a * dl;
    const float cs = rho != 0.f ? qr / rho : 1.f, sn = rho != 0.f ? qi / rho : 0.f;
    const float gr_ = dq[2 * i], gi_ = dq[2 * i + 1];
    const float drho = gr_ * cs + gi_ * sn;
    const float dphi = -gr_ * qi + gi_ * qr;
    dalpha[i] = (dp[i] - drho * dl) * a * (1.f - a);
    ddelta[i] = -drho * a * dl * (1.f - dl);
    dth = dphi * (float)(n + 1);
    dgamma[2 * i] = dg[2 * i] * scale;
    dgamma[2 * i + 1] = dg[2 * i + 1] * scale;
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) dth += __shfl_xor_sync(0xffffffffu, dth, s);
  if (n == 0) dtheta[k] = dth * wave * st * (1.f - st);
}

}  // namespace mega

using namespace mega;

extern "C" int mega_cema_coeffs(const void* alpha, const void* delta, const void* theta, const void* gamma,
                                int param_dtype, int K, int N, float* p, float* q, float* gamma_hat,
                                mega_stream_t stream) {
  if (!alpha || !delta || !theta || !gamma || !p || !q || !gamma_hat) return MEGA_ERR_NULL;
  if (!valid_dtype(param_dtype)) return MEGA_ERR_DTYPE;
  if (K <= 0) return MEGA_ERR_SHAPE;
  if (N < 1 || N > MEGA_MAX_NDIM) return MEGA_ERR_NDIM;
  const unsigned grid = (unsigned)((K * N + 255) / 256);
  MEGA_DISPATCH_DTYPE(param_dtype, launch(cema_coeffs_kernel<T>, grid, 256, 0, stream, (const T*)alpha,
                                          (const T*)delta, (const T*)theta, (const T*)gamma, K, N,
                                          sqrtf(1.0f / (float)N), p, q, gamma_hat));
  return check_launch("cema_coeffs");
}

extern "C" int mega_cema_kernel(const float* p, const float* q, const float* gamma_hat, int K, int N, int L,
                                float* kernel_out, mega_stream_t stream) {
  if (!p || !q || !gamma_hat || !kernel_out) return MEGA_ERR_NULL;
  if (K <= 0 || L <= 0 || K > 65535) return MEGA_ERR_SHAPE;
  if (N < 1 || N > MEGA_MAX_NDIM) return MEGA_ERR_NDIM;
  dim3 grid((L + 255) / 256, K);
  launch(cema_kernel_kernel, grid, 256, 4 * N * sizeof(float), stream, p, q, gamma_hat, N, L, kernel_out);
  return check_launch("cema_kernel");
}

extern "C" int mega_cema_fwd(const void* x, void* y, int dtype, int B, int D, int L, int64_t xsb, int64_t xsd,
                             int64_t xsl, int64_t ysb, int64_t ysd, int64_t ysl, const float* p, const float* q,
                             const float* gamma_hat, const float* omega, int N, const uint8_t* pad_mask,
                             const float* h_in, float* h_out, unsigned flags, int truncation,
                             mega_stream_t stream) {
  if (!x || !y || !p || !q || !gamma_hat || !omega) return MEGA_ERR_NULL;
  if (!valid_dtype(dtype)) return MEGA_ERR_DTYPE;
  if (B <= 0 || D <= 0 || L <= 0) return MEGA_ERR_SHAPE;
  if (N < 1 || N > MEGA_MAX_NDIM) return MEGA_ERR_NDIM;
  if (!aligned_to(x, elem_size(dtype)) || !aligned_to(y, elem_size(dtype))) return MEGA_ERR_ALIGN;
  const bool bidir = flags & MEGA_EMA_BIDIRECTIONAL;
  const bool trunc = truncation > 0 && truncation < L;
  if (bidir && (h_in || h_out)) return MEGA_ERR_UNSUPPORTED;
  if (!bidir && trunc) return MEGA_ERR_UNSUPPORTED;
  if (x == y && (bidir || trunc || xsb != ysb || xsd != ysd || xsl != ysl)) return MEGA_ERR_STRIDE;
  if (!trunc && x != y) {
    ScanArgs ca{};
    ca.x = x; ca.y = y; ca.B = B; ca.D = D; ca.L = L; ca.N = N;
    ca.xsb = xsb; ca.xsl = xsl; ca.ysb = ysb; ca.ysl = ysl;
    ca.p = p; ca.q = q; ca.g = gamma_hat; ca.omega = omega; ca.mask = pad_mask; ca.h_in = h_in; ca.h_out = h_out;
    ca.cplx = 1;
    ca.bidir = bidir ? 1 : 0;
    ca.shift = (flags & MEGA_EMA_NO_SHIFT) ? 0 : 1;
    ca.silu = (flags & MEGA_EMA_SILU) ? 1 : 0;
    if (chunk_ema_fwd_try(dtype, dtype, ca, xsd, ysd, (cudaStream_t)stream)) return check_launch("cema_fwd(chunk)");
    if (!bidir && N <= 16 && !scan_cluster_first(dtype, ca, xsd, ysd)) {
      StreamArgs sa{};
      sa.B = B; sa.L = L; sa.D = D; sa.N = N;
      sa.p = p; sa.q = q; sa.g = gamma_hat; sa.omega = omega; sa.h_in = h_in; sa.h_out = h_out; sa.mask = pad_mask;
      sa.silu = (flags & MEGA_EMA_SILU) ? 1 : 0;
      sa.cplx = 1;
      if (mma_cl_try(dtype, x, y, nullptr, xsb, xsl, xsd, ysb, ysl, ysd, false, sa, (cudaStream_t)stream))
        return check_launch("cema_fwd(mma)");
    }
    if (scan_ema_fwd_try(dtype, ca, xsd, ysd, (cudaStream_t)stream)) return check_launch("cema_fwd(scan)");
  }
  CemaArgs a{};
  a.x = x; a.y = y; a.B = B; a.D = D; a.L = L; a.N = N;
  a.xsb = xsb; a.xsd = xsd; a.xsl = xsl; a.ysb = ysb; a.ysd = ysd; a.ysl = ysl;
  a.p = p; a.q = q; a.g = gamma_hat; a.omega = omega; a.mask = pad_mask; a.h_in = h_in; a.h_out = h_out;
  a.ksize = trunc ? truncation : L;
  a.bidir = bidir ? 1 : 0;
  a.shift = (flags & MEGA_EMA_NO_SHIFT) ? 0 : 1;
  a.silu = (flags & MEGA_EMA_SILU) ? 1 : 0;
  const unsigned grid = (unsigned)(((long long)B * D + 31) / 32);
  const int np = N <= 4 ? 1 : N <= 8 ? 2 : N <= 16 ? 4 : 8;
#define MEGA_CEMA_LAUNCH(NPV)                                                                   \
  if (trunc && pad_mask) launch(cema_scan_kernel<T, NPV, true, true>, grid, 128, 0, stream, a);   \
  else if (trunc) launch(cema_scan_kernel<T, NPV, true, false>, grid, 128, 0, stream, a);         \
  else if (pad_mask) launch(cema_scan_kernel<T, NPV, false, true>, grid, 128, 0, stream, a);      \
  else launch(cema_scan_kernel<T, NPV, false, false>, grid, 128, 0, stream, a)
  MEGA_DISPATCH_DTYPE(dtype, {
    if (np == 1) { MEGA_CEMA_LAUNCH(1); }
    else if (np == 2) { MEGA_CEMA_LAUNCH(2); }
    else if (np == 4) { MEGA_CEMA_LAUNCH(4); }
    else { MEGA_CEMA_LAUNCH(8); }
  });
#undef MEGA_CEMA_LAUNCH
  return check_launch("cema_fwd");
}

extern "C" int mega_cema_step(const void* x, void* y, int dtype, int B, int D, const float* p, const float* q,
                              const float* gamma_hat, const float* omega, int N, const float* h_in,
                              float* h_out, unsigned flags, mega_stream_t stream) {
  if (!x || !y || !p || !q || !gamma_hat || !omega || !h_out) return MEGA_ERR_NULL;
  if (!valid_dtype(dtype)) return MEGA_ERR_DTYPE;
  if (B <= 0 || D <= 0) return MEGA_ERR_SHAPE;
  if (N < 1 || N > MEGA_MAX_NDIM) return MEGA_ERR_NDIM;
  const unsigned grid = (unsigned)(((long long)B * D + 127) / 128);
  const int silu = (flags & MEGA_EMA_SILU) ? 1 : 0;
  bool lanes = false;
  MEGA_DISPATCH_DTYPE(dtype, lanes = launch_cema_step_lanes<T>((const T*)x, (T*)y, (T*)nullptr, B, D, N, nullptr,
                                                              nullptr, nullptr, nullptr, nullptr, 0.f, p, q,
                                                              gamma_hat, omega, h_in, h_out, silu, stream));
  if (lanes) return check_launch("cema_step(lanes)");
  MEGA_DISPATCH_DTYPE(dtype, launch(cema_step_kernel<T>, grid, 128, 0, stream, (const T*)x, (T*)y, B, D, N, p, q,
                                    gamma_hat, omega, h_in, h_out, (flags & MEGA_EMA_SILU) ? 1 : 0));
  return check_launch("cema_step");
}

extern "C" int mega_tsn_cema_step(const void* x, void* y, void* xn_out, int dtype, int B, int D, int64_t* count,
                                  int64_t* count_next, float* mean, float* var, const float* gamma,
                                  const float* beta, double eps,
                                  const float* p, const float* q, const float* gamma_hat, const float* omega, int N,
                                  float* h, unsigned flags, mega_stream_t stream) {
  if (!x || !y || !count || !mean || !var || !gamma || !beta || !p || !q || !gamma_hat || !omega || !h)
    return MEGA_ERR_NULL;
  if (!valid_dtype(dtype)) return MEGA_ERR_DTYPE;
  if (B <= 0 || D <= 0) return MEGA_ERR_SHAPE;
  if (N < 1 || N > MEGA_MAX_NDIM) return MEGA_ERR_NDIM;
  const int silu = (flags & MEGA_EMA_SILU) ? 1 : 0;
  // a distinct count_next array takes the bumped counts from the element kernel itself
  long long* next = (count_next && count_next != count) ? (long long*)count_next : nullptr;
  const bool lanes = cema_step_lanes_try(dtype, x, y, xn_out, B, D, N, (const long long*)count, mean, var, gamma, beta,
                                         (float)eps, p, q, gamma_hat, omega, h, h, silu, stream, next);
  if (!lanes) return MEGA_ERR_UNSUPPORTED;  // pole counts other than 2, 4, 8, 16, 32, or unaligned states
  if (!next) launch(cema_count_step_kernel, (unsigned)((B + 127) / 128), 128, 0, stream, (long long*)count, B);
  return check_launch("tsn_cema_step");
}

extern "C" int mega_tsn_cema_fwd(const void* x, void* y, void* xn_out, int dtype, int B, int L, int D, int64_t xsb,
                                 int64_t xsl, int64_t xsd, int64_t ysb, int64_t ysl, int64_t ysd,
                                 const int64_t* prev_count, const float* prev_mean, const float* prev_var,
                                 const float* gamma, const float* beta, double eps, int64_t* count_out,
                                 float* mean_out, float* var_out, const float* p, const float* q,
                                 const float* gamma_hat, const float* omega, int N, const uint8_t* pad_mask,
                                 const float* h_in, float* h_out, unsigned flags, mega_stream_t stream) {
  if (!x || !y || !prev_count || !prev_mean || !prev_var || !gamma || !beta || !count_out || !mean_out ||
      !var_out || !p || !q || !gamma_hat || !omega)
    return MEGA_ERR_NULL;
  // every thread block of a sequence reads its incoming count; one of them writes the new one
  if ((const void*)count_out == (const void*)prev_count) return MEGA_ERR_UNSUPPORTED;
  if (!valid_dtype(dtype)) return MEGA_ERR_DTYPE;
  if (B <= 0 || L <= 0 || D <= 0) return MEGA_ERR_SHAPE;
  if (N < 1 || N > MEGA_MAX_NDIM) return MEGA_ERR_NDIM;
  if (flags & MEGA_EMA_BIDIRECTIONAL) return MEGA_ERR_UNSUPPORTED;
  if (x == y) return MEGA_ERR_UNSUPPORTED;
  if (N <= 16) {
    StreamArgs sa{};
    sa.B = B; sa.L = L; sa.D = D; sa.N = N;
    sa.prev_count = (const long long*)prev_count; sa.prev_mean = prev_mean; sa.prev_var = prev_var;
    sa.gamma = gamma; sa.beta = beta; sa.eps = (float)eps;
    sa.count_out = (long long*)count_out; sa.mean_out = mean_out; sa.var_out = var_out;
    sa.p = p; sa.q = q; sa.g = gamma_hat; sa.omega = omega; sa.h_in = h_in; sa.h_out = h_out; sa.mask = pad_mask;
    sa.silu = (flags & MEGA_EMA_SILU) ? 1 : 0;
    sa.cplx = 1;
    if (norm_ema_split_try(dtype, x, y, xn_out, xsb, xsl, xsd, ysb, ysl, ysd, sa, (cudaStream_t)stream))
      return check_launch("tsn_cema_fwd(split)");
    // (a state exported at a length that the tensor-core kernel's steps of 32 do not divide stays with the forms that run
    // in fp32 throughout: a head on that kernel rounds its operands to bf16, and the state was 1e-3 off instead of 1e-6)
    if (mma_cl_try(dtype, x, y, xn_out, xsb, xsl, xsd, ysb, ysl, ysd, true, sa, (cudaStream_t)stream))
      return check_launch("tsn_cema_fwd(mma)");
    if (stream_cl_try(dtype, x, y, xn_out, xsb, xsl, xsd, ysb, ysl, ysd, true, sa, (cudaStream_t)stream))
      return check_launch("tsn_cema_fwd(stream)");
  }
  // outside the streamed kernel's envelope: the two operators in turn (the EMA runs in place)
  void* mid = xn_out ? xn_out : y;
  int rc = mega_timestep_norm_fwd(x, mid, dtype, B, L, D, xsb, xsl, xsd, ysb, ysl, ysd, prev_count, prev_mean,
                                  prev_var, gamma, beta, pad_mask, D, eps, count_out, mean_out, var_out, stream);
  if (rc != MEGA_OK) return rc;
  return mega_cema_fwd(mid, y, dtype, B, D, L, ysb, ysd, ysl, ysb, ysd, ysl, p, q, gamma_hat, omega, N, pad_mask,
                       h_in, h_out, flags, 0, stream);
}

extern "C" int mega_cema_bwd(const void* dy, const void* x, void* dx, int dtype, int B, int D, int L, int64_t gsb,
                             int64_t gsd, int64_t gsl, int64_t xsb, int64_t xsd, int64_t xsl, int64_t dsb,
                             int64_t dsd, int64_t dsl, const float* p, const float* q, const float* gamma_hat,
                             const float* omega, int N, const uint8_t* pad_mask, unsigned flags, int truncation,
                             float* dp, float* dq, float* dgamma_hat, float* domega, mega_stream_t stream) {
  if (!dy || !x || !dx || !p || !q || !gamma_hat || !omega || !dp || !dq || !dgamma_hat || !domega)
    return MEGA_ERR_NULL;
  if (!valid_dtype(dtype)) return MEGA_ERR_DTYPE;
  if (B <= 0 || D <= 0 || L <= 0) return MEGA_ERR_SHAPE;
  if (N < 1 || N > MEGA_MAX_NDIM) return MEGA_ERR_NDIM;
  if (flags & MEGA_EMA_SILU) return MEGA_ERR_UNSUPPORTED;
  const bool trunc = truncation > 0 && truncation < L;
  if (trunc && !(flags & MEGA_EMA_BIDIRECTIONAL)) return MEGA_ERR_UNSUPPORTED;  // as the forward
  const size_t es = elem_size(dtype);
  if (!aligned_to(dy, es) || !aligned_to(x, es) || !aligned_to(dx, es)) return MEGA_ERR_ALIGN;
  const bool bidir = (flags & MEGA_EMA_BIDIRECTIONAL) != 0;
  const size_t K = (size_t)(bidir ? 2 : 1) * D;
  cudaStream_t s = (cudaStream_t)stream;
  if (!zero_arrays(s, {{dp, K * N}, {dq, 2 * K * N}, {dgamma_hat, 2 * K * N}, {domega, (size_t)D}}))
    return check_launch("cema_bwd(memset)");
  if (!trunc && dx != dy && dx != x) {
    ScanArgs ca{};
    ca.x = x; ca.y = dx; ca.dy = dy; ca.B = B; ca.D = D; ca.L = L; ca.N = N;
    ca.xsb = xsb; ca.xsl = xsl; ca.ysb = dsb; ca.ysl = dsl; ca.gsb = gsb; ca.gsl = gsl;
    ca.p = p; ca.q = q; ca.g = gamma_hat; ca.omega = omega; ca.mask = pad_mask;
    ca.cplx = 1;
    ca.bidir = bidir ? 1 : 0;
    ca.shift = (flags & MEGA_EMA_NO_SHIFT) ? 0 : 1;
    ca.dp = dp; ca.dq = dq; ca.dg = dgamma_hat; ca.domega = domega;
    if (chunk_ema_bwd_try(dtype, ca, xsd, dsd, gsd, s)) return check_launch("cema_bwd(chunk)");
    if (scan_ema_bwd_try(dtype, ca, xsd, dsd, gsd, s)) return check_launch("cema_bwd(scan)");
  }
  CemaBwdArgs a{};
  a.dy = dy; a.x = x; a.dx = dx; a.B = B; a.D = D; a.L = L; a.N = N;
  a.gsb = gsb; a.gsd = gsd; a.gsl = gsl; a.xsb = xsb; a.xsd = xsd; a.xsl = xsl;
  a.dsb = dsb; a.dsd = dsd; a.dsl = dsl;
  a.p = p; a.q = q; a.g = gamma_hat; a.omega = omega; a.mask = pad_mask;
  a.dp = dp; a.dq = dq; a.dg = dgamma_hat; a.domega = domega;
  a.bidir = bidir ? 1 : 0;
  a.shift = (flags & MEGA_EMA_NO_SHIFT) ? 0 : 1;
  a.ksize = trunc ? truncation : L;
  const unsigned grid = (unsigned)(((long long)B * D + 31) / 32);
  const int np = N <= 4 ? 1 : N <= 8 ? 2 : N <= 16 ? 4 : 8;
#define MEGA_CEMA_BWD(NPV)                                                          \
  if (trunc) {                                                                             \
    if (pad_mask) launch(cema_bwd_kernel<T, NPV, true, true>, grid, 128, 0, stream, a);     \
    else launch(cema_bwd_kernel<T, NPV, false, true>, grid, 128, 0, stream, a);             \
  } else if (pad_mask) launch(cema_bwd_kernel<T, NPV, true, false>, grid, 128, 0, stream, a); \
  else launch(cema_bwd_kernel<T, NPV, false, false>, grid, 128, 0, stream, a)
  MEGA_DISPATCH_DTYPE(dtype, {
    if (np == 1) { MEGA_CEMA_BWD(1); }
    else if (np == 2) { MEGA_CEMA_BWD(2); }
    else if (np == 4) { MEGA_CEMA_BWD(4); }
    else { MEGA_CEMA_BWD(8); }
  });
#undef MEGA_CEMA_BWD
  return check_launch("cema_bwd");
}

extern "C" int mega_cema_coeffs_bwd(const float* alpha, const float* delta, const float* theta, const float* q,
                                    const float* dp, const float* dq, const float* dgamma_hat, int K, int N,
                                    float* dalpha, float* ddelta, float* dtheta, float* dgamma,
                                    mega_stream_t stream) {
  if (!alpha || !delta || !theta || !q || !dp || !dq || !dgamma_hat || !dalpha || !ddelta || !dtheta || !dgamma)
    return MEGA_ERR_NULL;
  if (K <= 0) return MEGA_ERR_SHAPE;
  if (N < 1 || N > MEGA_MAX_NDIM) return MEGA_ERR_NDIM;
  launch(cema_coeffs_bwd_kernel, (unsigned)((K + 3) / 4), 128, 0, stream, alpha, delta, theta, q, dp, dq,
         dgamma_hat, K, N, rsqrtf((float)N), dalpha, ddelta, dtheta, dgamma);
  return check_launch("cema_coeffs_bwd");
}
