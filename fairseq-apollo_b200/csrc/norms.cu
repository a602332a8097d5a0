// TimestepNorm (plain + grouped) and SequenceNorm (plain + grouped, any memory order).
//
// TimestepNorm is a causal cumulative normalisation: the statistics at step t are the Welford
// moments of the unmasked prefix (plus a prior that acts as prev_count pseudo-samples).
// SequenceNorm normalises with the masked moments of the whole sequence.
#include <mutex>

#include "common.cuh"
#include "scan_norm.cuh"
#include "stream_bwd.cuh"
#include "stream_cl.cuh"
#include "tmem_ema.cuh"

namespace mega {

struct TsnArgs {
  const void* x;
  void* y;
  int B, L, D, G;
  long long xsb, xsl, xsd, ysb, ysl, ysd;
  const long long* prev_count;
  const float *prev_mean, *prev_var, *gamma, *beta;
  const unsigned char* mask;
  float eps;
  long long* count_out;
  float *mean_out, *var_out;
  // training-mode saves (all NULL in inference): per-step statistics, fp32, contiguous (B, L, G);
  // group_mean only for the grouped form
  float *cummean, *cumrstd, *group_mean;
};

// Welford step with the update rule of the reference (fairseq/csrc/utils.h:56-65).
__device__ __forceinline__ void welford_step(float coef, float x, float mean, float var, float& m1,
                                             float& m2) {
  const float d1 = x - mean;
  m1 = fmaf(coef, d1, mean);
  const float d2 = fmaf(d1, x - m1, -var);
  m2 = fmaf(coef, d2, var);
}

// One thread per (batch, feature), feature fastest; sequential over time.  The presence of a
// mask and of the training saves are template parameters: a run-time test of those pointers
// inside the unrolled load batch turns it into branchy code whose loads no longer overlap
// (measured: 4x slower with the mask test, 2x with the save test, even when both are null).
template <typename T, bool kMask, bool kSave>
__global__ void __launch_bounds__(128) tsn_plain_kernel(TsnArgs a) {
  long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (long long)a.B * a.D) return;
  const int d = (int)(gid % a.D);
  const int b = (int)(gid / a.D);
  const T* xp = reinterpret_cast<const T*>(a.x) + b * a.xsb + d * a.xsd;
  T* yp = reinterpret_cast<T*>(a.y) + b * a.ysb + d * a.ysd;
  const unsigned char* mp = kMask ? a.mask + (size_t)b * a.L : nullptr;
  float* cmp = kSave ? a.cummean + (size_t)b * a.L * a.D + d : nullptr;
  float* crp = kSave ? a.cumrstd + (size_t)b * a.L * a.D + d : nullptr;
  // the count as a 32-bit step counter on top of the incoming count (64-bit integer to float
  // conversions inside the serial loop are slow)
  const long long cnt0 = a.prev_count[b];
  const float cnt0f = (float)cnt0;
  int seen = 0;
  float mean = a.prev_mean[gid], var = a.prev_var[gid];
  const float w = __ldg(a.gamma + d), bb = __ldg(a.beta + d);
  constexpr int U = 32;  // loads in flight per thread: B x D threads are few, latency is hidden per thread
  for (int t0 = 0; t0 < a.L; t0 += U) {
    float xv[U];
    bool mk[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = t0 + u;
      xv[u] = 0.f; mk[u] = true;
      if (t < a.L) {
        xv[u] = Elem<T>::ld(xp + t * a.xsl);
        mk[u] = kMask ? __ldg(mp + t) != 0 : false;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int t = t0 + u;
      if (t < a.L) {
        float m1, m2;
        const float coef = rcp_approx(cnt0f + (float)(seen + 1));
        welford_step(coef, xv[u], mean, var, m1, m2);
        const float rstd = rsqrt_approx(m2 + a.eps);
        const float out = mk[u] ? 0.f : fmaf((xv[u] - m1) * rstd, w, bb);
        Elem<T>::st(yp + t * a.ysl, out);
        if (!mk[u]) { mean = m1; var = m2; ++seen; }
        if (kSave) {  // the running mean AFTER step t (unchanged by a padded step)
          cmp[(size_t)t * a.D] = mean;
          crp[(size_t)t * a.D] = rstd;
        }
      }
    }
  }
  a.mean_out[gid] = mean;
  a.var_out[gid] = var;
  if (d == 0) a.count_out[b] = cnt0 + seen;
}

// Grouped: one warp per (batch, group); per step the group's D/G features are reduced to
// (mean, var), combined into the running state with weight 1, then normalised.
template <typename T>
__global__ void __launch_bounds__(128) tsn_group_kernel(TsnArgs a) {
  const int lane = threadIdx.x & 31;
  const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (wid >= (long long)a.B * a.G) return;
  const int g = (int)(wid % a.G);
  const int b = (int)(wid / a.G);
  const int gs = a.D / a.G;
  const T* xp = reinterpret_cast<const T*>(a.x) + b * a.xsb + (long long)g * gs * a.xsd;
  T* yp = reinterpret_cast<T*>(a.y) + b * a.ysb + (long long)g * gs * a.ysd;
  const unsigned char* mp = a.mask ? a.mask + (size_t)b * a.L : nullptr;
  long long cnt = a.prev_count[b];
  float mean = a.prev_mean[wid], var = a.prev_var[wid];
  const float inv_gs = 1.0f / (float)gs;
  for (int t = 0; t < a.L; ++t) {
    const T* xr = xp + t * a.xsl;
    float s = 0.f;
    for (int k = lane; k < gs; k += 32) s += Elem<T>::ld(xr + k * a.xsd);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float gm = s * inv_gs;
    float v = 0.f;
    for (int k = lane; k < gs; k += 32) {
      const float dlt = Elem<T>::ld(xr + k * a.xsd) - gm;
      v = fmaf(dlt, dlt, v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const float gv = v * inv_gs;
    // WelfordCombine(cnt, mean, var, 1, gm, gv)  (fairseq/csrc/utils.h:67-76)
    const float m0 = (float)(cnt + 1);
    const float c1 = (float)cnt / m0, c2 = 1.0f / m0;
    const float dl = gm - mean;
    const float m1 = c1 * mean + c2 * gm;
    const float m2 = c1 * var + c2 * gv + (c1 * dl) * (c2 * dl);
    const float rstd = rsqrtf(m2 + a.eps);
    const bool mk = mp != nullptr && mp[t] != 0;
    T* yr = yp + t * a.ysl;
    for (int k = lane; k < gs; k += 32) {
      const int f = g * gs + k;
      const float xv = Elem<T>::ld(xr + k * a.xsd);
      const float out = mk ? 0.f : fmaf((xv - m1) * rstd, __ldg(a.gamma + f), __ldg(a.beta + f));
      Elem<T>::st(yr + k * a.ysd, out);
    }
    if (!mk) { mean = m1; var = m2; ++cnt; }
    if (a.cummean && lane == 0) {
      const size_t o = ((size_t)b * a.L + t) * a.G + g;
      a.cummean[o] = mean;
      a.cumrstd[o] = rstd;
      a.group_mean[o] = gm;
    }
  }
  if (lane == 0) {
    a.mean_out[wid] = mean;
    a.var_out[wid] = var;
    if (g == 0) a.count_out[b] = cnt;
  }
}

// ---------------------------------------------------------------------------
// SequenceNorm
// ---------------------------------------------------------------------------
struct SqnArgs {
  const void* x;
  void* y;
  int B, D, L, G;
  long long xsb, xsd, xsl, ysb, ysd, ysl;
  const float *gamma, *beta;
  const unsigned char* mask;
  float eps;
  long long* count_out;
  float *mean_out, *rstd_out;
};

__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float r = 0.f;
  const int nw = (blockDim.x + 31) >> 5;
  for (int i = 0; i < nw; ++i) r += red[i];
  return r;
}

// One CTA per (batch, group): the group's gs channels x L positions.  Two reduction passes
// (mean, then centred second moment) and a normalisation pass; when the segment fits the
// dynamic shared memory it is cached there after the first read.
template <typename T>
__global__ void __launch_bounds__(256) sqn_segment_kernel(SqnArgs a, int cache_elems) {
  extern __shared__ float cache[];
  __shared__ float red[8];
  const int g = blockIdx.x % a.G;
  const int b = blockIdx.x / a.G;
  const int gs = a.D / a.G;
  const long long n = (long long)gs * a.L;
  const bool len_fast = a.xsl <= a.xsd;  // iterate the contiguous axis fastest
  const T* xp = reinterpret_cast<const T*>(a.x) + b * a.xsb + (long long)g * gs * a.xsd;
  T* yp = reinterpret_cast<T*>(a.y) + b * a.ysb + (long long)g * gs * a.ysd;
  const unsigned char* mp = a.mask ? a.mask + (size_t)b * a.L : nullptr;
  const bool cached = n <= cache_elems;

  float s = 0.f;
  for (long long i = threadIdx.x; i < n; i += blockDim.x) {
    const int j = len_fast ? (int)(i / a.L) : (int)(i % gs);
    const int t = len_fast ? (int)(i % a.L) : (int)(i / gs);
    const float xv = Elem<T>::ld(xp + j * a.xsd + t * a.xsl);
    if (cached) cache[i] = xv;
    const bool mk = mp != nullptr && mp[t] != 0;
    if (!mk) s += xv;
  }
  __shared__ int valid_steps;
  if (threadIdx.x == 0) valid_steps = 0;
  __syncthreads();
  int c = 0;
  for (int t = threadIdx.x; t < a.L; t += blockDim.x) c += (mp == nullptr || mp[t] == 0) ? 1 : 0;
  if (c) atomicAdd(&valid_steps, c);
  __syncthreads();
  const float tot = (float)valid_steps * (float)gs;
  const float sum = block_sum(s, red);
  const float mean = tot > 0.f ? sum / tot : 0.f;
  float v = 0.f;
  for (long long i = threadIdx.x; i < n; i += blockDim.x) {
    const int j = len_fast ? (int)(i / a.L) : (int)(i % gs);
    const int t = len_fast ? (int)(i % a.L) : (int)(i / gs);
    const float xv = cached ? cache[i] : Elem<T>::ld(xp + j * a.xsd + t * a.xsl);
    const bool mk = mp != nullptr && mp[t] != 0;
    if (!mk) { const float dl = xv - mean; v = fmaf(dl, dl, v); }
  }
  const float var = tot > 0.f ? block_sum(v, red) / tot : 0.f;
  const float rstd = rsqrtf(var + a.eps);
  for (long long i = threadIdx.x; i < n; i += blockDim.x) {
    const int j = len_fast ? (int)(i / a.L) : (int)(i % gs);
    const int t = len_fast ? (int)(i % a.L) : (int)(i / gs);
    const float xv = cached ? cache[i] : Elem<T>::ld(xp + j * a.xsd + t * a.xsl);
    const bool mk = mp != nullptr && mp[t] != 0;
    const int f = g * gs + j;
    const float out = mk ? 0.f : fmaf((xv - mean) * rstd, __ldg(a.gamma + f), __ldg(a.beta + f));
    Elem<T>::st(yp + j * a.ysd + t * a.ysl, out);
  }
  if (threadIdx.x == 0) {
    a.mean_out[blockIdx.x] = mean;
    a.rstd_out[blockIdx.x] = rstd;
    if (g == 0) a.count_out[b] = (long long)valid_steps;
  }
}

// Plain SequenceNorm on channel-contiguous memory: one thread per (batch, channel) column,
// masked Welford over time, then a second sweep that normalises.
template <typename T>
__global__ void __launch_bounds__(128) sqn_column_kernel(SqnArgs a) {
  long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (long long)a.B * a.D) return;
  const int d = (int)(gid % a.D);
  const int b = (int)(gid / a.D);
  const T* xp = reinterpret_cast<const T*>(a.x) + b * a.xsb + d * a.xsd;
  T* yp = reinterpret_cast<T*>(a.y) + b * a.ysb + d * a.ysd;
  const unsigned char* mp = a.mask ? a.mask + (size_t)b * a.L : nullptr;
  long long cnt = 0;
  float mean = 0.f, var = 0.f;
  for (int t = 0; t < a.L; ++t) {
    const bool mk = mp != nullptr && mp[t] != 0;
    if (!mk) {
      const float xv = Elem<T>::ld(xp + t * a.xsl);
      float m1, m2;
      welford_step(__frcp_rn((float)(cnt + 1)), xv, mean, var, m1, m2);
      mean = m1; var = m2; ++cnt;
    }
  }
  const float rstd = rsqrtf(var + a.eps);
  const float w = __ldg(a.gamma + d), bb = __ldg(a.beta + d);
  for (int t = 0; t < a.L; ++t) {
    const bool mk = mp != nullptr && mp[t] != 0;
    const float xv = Elem<T>::ld(xp + t * a.xsl);
    Elem<T>::st(yp + t * a.ysl, mk ? 0.f : fmaf((xv - mean) * rstd, w, bb));
  }
  a.mean_out[gid] = mean;
  a.rstd_out[gid] = rstd;
  if (d == 0) a.count_out[b] = cnt;
}

// ---------------------------------------------------------------------------
// parameters of a norm module in one launch each way (as torch operations: a dozen launches of a few values)
// ---------------------------------------------------------------------------
// fp32 effective scale (weight + 1) and bias; with B > 0 also the priors as running statistics of B sequences.  One of these
// runs in front of every inference call, so it is launched ahead of the end of what comes before it (layer of 16 x 4096 x
// 1024 bf16: 142 us with it, 140 without; 144 where it waits).
template <typename T>
__global__ void norm_prepare_kernel(const long long* prior_count, const T* prior_mean, const T* prior_logv, const T* weight,
                                    const T* bias, int B, int G, int D, long long* count, float* mean, float* var,
                                    float* gamma, float* beta) {
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < D && blockIdx.y == 0) {
    gamma[i] = Elem<T>::ld(weight + i) + 1.f;
    beta[i] = Elem<T>::ld(bias + i);
  }
  if (i < G) {
    const float m = Elem<T>::ld(prior_mean + i), v = expf(Elem<T>::ld(prior_logv + i));
    for (int b = blockIdx.y; b < B; b += gridDim.y) {
      mean[(size_t)b * G + i] = m;
      var[(size_t)b * G + i] = v;
    }
  }
  if (i < B && blockIdx.y == 0) count[i] = prior_count[0];
}
// their gradients in the parameters' type: the affine pair converted, the priors' summed over the batch
template <typename T>
__global__ void norm_finish_kernel(const float* dprev_mean, const float* dprev_var, const T* prior_logv, const float* dgamma,
                                   const float* dbeta, int B, int G, int D, T* dprior_mean, T* dprior_logv, T* dweight,
                                   T* dbias) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < D) {
    Elem<T>::st(dweight + i, dgamma[i]);
    Elem<T>::st(dbias + i, dbeta[i]);
  }
  if (i < G && B > 0) {
    float m = 0.f, v = 0.f;
    for (int b = 0; b < B; ++b) {
      m += dprev_mean[(size_t)b * G + i];
      v += dprev_var[(size_t)b * G + i];
    }
    Elem<T>::st(dprior_mean + i, m);
    Elem<T>::st(dprior_logv + i, v * expf(Elem<T>::ld(prior_logv + i)));
  }
}

// ---------------------------------------------------------------------------
// gates
// ---------------------------------------------------------------------------
template <typename T, int OP>
__global__ void gate_kernel(const T* a, long long lda, const T* b, long long ldb, const T* c, long long ldc,
                            const T* d, long long ldd, T* y, long long ldy, long long rows, int cols) {
  const long long n = rows * cols;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / cols;
    const int col = (int)(i % cols);
    float out;
    if (OP == 0) {  // silu(a [+ b])
      float v = Elem<T>::ld(a + r * lda + col);
      if (b) v += Elem<T>::ld(b + r * ldb + col);
      out = v * sigmoid_of<T>(v);
    } else if (OP == 1) {  // a * silu(b)
      const float v = Elem<T>::ld(b + r * ldb + col);
      out = Elem<T>::ld(a + r * lda + col) * (v * sigmoid_of<T>(v));
    } else {  // a = residual, b = u, c = hx, d = h_lin
      const float res = Elem<T>::ld(a + r * lda + col);
      const float u = sigmoid_of<T>(Elem<T>::ld(b + r * ldb + col));
      const float v = Elem<T>::ld(c + r * ldc + col) + Elem<T>::ld(d + r * ldd + col), h = v * sigmoid_of<T>(v);
      out = fmaf(u, h - res, res);
    }
    Elem<T>::st(y + r * ldy + col, out);
  }
}

// The same gates, 16 bytes per access (8 bf16 / fp16 or 4 fp32 values), for column counts, row pitches and base
// addresses that are multiples of 16 bytes.  A block is blockDim.x vectors of blockDim.y rows, kU times; all loads first,
// and no division (with one per vector, and a grid-stride loop: 126 us where this takes 84 for silu on (65536, 2048) bf16).
// Memory-bound: 2, 3 and 5 streams at 6.4 - 6.9 TB/s (some of it from L2: a copy moves 6.5); two MUFU operations a value cost
// silu 4 us of the 84.
template <typename T, int OP, int kU>
__global__ void __launch_bounds__(256) gate_vec_kernel(const T* a, long long lda, const T* b, long long ldb, const T* c,
                                                       long long ldc, const T* d, long long ldd, T* y, long long ldy,
                                                       long long rows, int cols) {
  constexpr int kN = 16 / (int)sizeof(T);
  const int col = (blockIdx.y * blockDim.x + threadIdx.x) * kN;
  if (col >= cols) return;
  const long long r0 = (long long)blockIdx.x * blockDim.y * kU + threadIdx.y;
  uint4 va[kU], vb[kU], vc[OP == 2 ? kU : 1], vd[OP == 2 ? kU : 1];
#pragma unroll
  for (int u = 0; u < kU; ++u) {
    const long long r = r0 + u * blockDim.y;
    if (r < rows) {
      va[u] = *reinterpret_cast<const uint4*>(a + r * lda + col);
      if (OP != 0 || b != nullptr) vb[u] = *reinterpret_cast<const uint4*>(b + r * ldb + col);
      if (OP == 2) {
        vc[OP == 2 ? u : 0] = *reinterpret_cast<const uint4*>(c + r * ldc + col);
        vd[OP == 2 ? u : 0] = *reinterpret_cast<const uint4*>(d + r * ldd + col);
      }
    }
  }
#pragma unroll
  for (int u = 0; u < kU; ++u) {
    const long long r = r0 + u * blockDim.y;
    if (r >= rows) break;
    const T *fa = reinterpret_cast<const T*>(&va[u]), *fb = reinterpret_cast<const T*>(&vb[u]),
            *fc = reinterpret_cast<const T*>(&vc[OP == 2 ? u : 0]), *fd = reinterpret_cast<const T*>(&vd[OP == 2 ? u : 0]);
    uint4 out;
    T* o = reinterpret_cast<T*>(&out);
#pragma unroll
    for (int k = 0; k < kN; ++k) {
      const float x = Elem<T>::ld_shared(fa + k);
      if (OP == 0) {  // silu(a [+ b])
        const float v = b != nullptr ? x + Elem<T>::ld_shared(fb + k) : x;
        Elem<T>::st(o + k, v * sigmoid_of<T>(v));
      } else if (OP == 1) {  // a * silu(b)
        const float v = Elem<T>::ld_shared(fb + k);
        Elem<T>::st(o + k, x * (v * sigmoid_of<T>(v)));
      } else {  // a = residual, b = u, c = hx, d = h_lin
        const float v = Elem<T>::ld_shared(fb + k);
        const float g = sigmoid_of<T>(v);
        const float hs = Elem<T>::ld_shared(fc + k) + Elem<T>::ld_shared(fd + k);
        const float h = hs * sigmoid_of<T>(hs);
        Elem<T>::st(o + k, fmaf(g, h - x, x));
      }
    }
    *reinterpret_cast<uint4*>(y + r * ldy + col) = out;
  }
}

// One warp per row: z / max(||z||_2, eps), then the two affine rows (query, key).
template <typename T>
__global__ void gate_qk_kernel(const T* z, long long ldz, const float* gamma, const float* beta, T* qo,
                               long long ldq, T* ko, long long ldk, long long rows, int cols, float eps) {
  const int lane = threadIdx.x & 31;
  const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long r = (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5); r < rows; r += warps) {
    const T* zr = z + r * ldz;
    float ss = 0.f;
    for (int c = lane; c < cols; c += 32) {
      const float v = Elem<T>::ld(zr + c);
      ss = fmaf(v, v, ss);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float inv = 1.f / fmaxf(sqrtf(ss), eps);
    for (int c = lane; c < cols; c += 32) {
      const float v = Elem<T>::ld(zr + c) * inv;
      Elem<T>::st(qo + r * ldq + c, fmaf(v, gamma[c] + 1.f, beta[c]));
      Elem<T>::st(ko + r * ldk + c, fmaf(v, gamma[cols + c] + 1.f, beta[cols + c]));
    }
  }
}

// The same with the rotary position embedding of the block applied to both results (pairs of
// features (2j, 2j + 1) of row r rotated by the angle of position r % period and frequency j;
// rot (positions, cols / 2, 2) holds (cos, sin)): a lane owns whole pairs, the rotation runs in fp32
// on the unrounded affine results.
template <typename T>
__global__ void gate_qk_rotary_kernel(const T* z, long long ldz, const float* gamma, const float* beta,
                                      const float* rot, int period, int q_offset, int out_period, T* qo, long long ldq, T* ko,
                                      long long ldk, T* kraw, long long rows, int cols, float eps) {
  const int lane = threadIdx.x & 31;
  const int half = cols >> 1;
  const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long r = (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5); r < rows; r += warps) {
    const T* zr = z + r * ldz;
    float ss = 0.f;
    for (int j = lane; j < half; j += 32) {
      const float a = Elem<T>::ld(zr + 2 * j), b = Elem<T>::ld(zr + 2 * j + 1);
      ss = fmaf(a, a, fmaf(b, b, ss));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float inv = 1.f / fmaxf(sqrtf(ss), eps);
    const int pos = (int)(r % period);
    const long long at = r / period * out_period + pos;
    const float2* rk = reinterpret_cast<const float2*>(rot) + (size_t)pos * half;
    const float2* rq = reinterpret_cast<const float2*>(rot) + (size_t)(pos + q_offset) * half;
    for (int j = lane; j < half; j += 32) {
      const int c = 2 * j;
      const float a = Elem<T>::ld(zr + c) * inv, b = Elem<T>::ld(zr + c + 1) * inv;
      const float qa = fmaf(a, gamma[c] + 1.f, beta[c]), qb = fmaf(b, gamma[c + 1] + 1.f, beta[c + 1]);
      const float ka = fmaf(a, gamma[cols + c] + 1.f, beta[cols + c]);
      const float kb = fmaf(b, gamma[cols + c + 1] + 1.f, beta[cols + c + 1]);
      const float2 wq = __ldg(rq + j), wk = __ldg(rk + j);
      Elem<T>::st(qo + at * ldq + c, qa * wq.x - qb * wq.y);
      Elem<T>::st(qo + at * ldq + c + 1, qa * wq.y + qb * wq.x);
      Elem<T>::st(ko + at * ldk + c, ka * wk.x - kb * wk.y);
      Elem<T>::st(ko + at * ldk + c + 1, ka * wk.y + kb * wk.x);
      if (kraw) {
        Elem<T>::st(kraw + r * cols + c, ka);
        Elem<T>::st(kraw + r * cols + c + 1, kb);
      }
    }
  }
}

// The same, 16 bytes per access, for 16-bit types and 64, 128 or 256 features: kLanes lanes take a row, eight features
// each.  Rows of a chunk may be written at a pitch of their own (out_period >= period rows per chunk), and the keys also
// as they are before the rotation (kraw, contiguous rows, or null), which is what a decoding cache keeps.  Memory-bound.
template <typename T, int kLanes>
__global__ void __launch_bounds__(256) gate_qk_rotary_vec_kernel(const T* z, long long ldz, const float* gamma, const float* beta,
                                                                 const float* rot, int period, int q_offset, int out_period, T* qo,
                                                                 long long ldq, T* ko, long long ldk, T* kraw, long long rows,
                                                                 float eps) {
  constexpr int kCols = kLanes * 8, kPer = 32 / kLanes;
  const int lane = threadIdx.x & 31, sub = lane % kLanes, c = 8 * sub;
  const long long first = ((long long)blockIdx.x * 8 + (threadIdx.x >> 5)) * (2 * kPer) + lane / kLanes;
  uint4 in[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {   // (two rows at once: more bytes in flight)
    const long long r = first + u * kPer;
    in[u] = make_uint4(0u, 0u, 0u, 0u);
    if (r < rows) in[u] = *reinterpret_cast<const uint4*>(z + r * ldz + c);
  }
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const long long r = first + u * kPer;
    const T* e = reinterpret_cast<const T*>(&in[u]);
    float f[8], ss = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      f[i] = Elem<T>::ld_shared(e + i);
      ss = fmaf(f[i], f[i], ss);
    }
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (r >= rows) continue;   // (no break: the lanes of the other rows of the warp shuffle again)
    const float inv = 1.f / fmaxf(sqrtf(ss), eps);
    const long long chunk = r / period;
    const int pos = (int)(r - chunk * period);
    const float4* rk = reinterpret_cast<const float4*>(rot + (size_t)pos * kCols + c);
    const float4* rq = reinterpret_cast<const float4*>(rot + (size_t)(pos + q_offset) * kCols + c);
    uint4 qv, kv, kw;
    T *qp = reinterpret_cast<T*>(&qv), *kp = reinterpret_cast<T*>(&kv), *wp = reinterpret_cast<T*>(&kw);
#pragma unroll
    for (int i = 0; i < 8; i += 4) {
      const float4 g0 = __ldg(reinterpret_cast<const float4*>(gamma + c + i)), g1 = __ldg(reinterpret_cast<const float4*>(gamma + kCols + c + i));
      const float4 b0 = __ldg(reinterpret_cast<const float4*>(beta + c + i)), b1 = __ldg(reinterpret_cast<const float4*>(beta + kCols + c + i));
      const float4 wq = __ldg(rq + i / 4), wk = __ldg(rk + i / 4);
      const float x0 = f[i] * inv, x1 = f[i + 1] * inv, x2 = f[i + 2] * inv, x3 = f[i + 3] * inv;
      const float q0 = fmaf(x0, g0.x + 1.f, b0.x), q1 = fmaf(x1, g0.y + 1.f, b0.y), q2 = fmaf(x2, g0.z + 1.f, b0.z), q3 = fmaf(x3, g0.w + 1.f, b0.w);
      const float k0 = fmaf(x0, g1.x + 1.f, b1.x), k1 = fmaf(x1, g1.y + 1.f, b1.y), k2 = fmaf(x2, g1.z + 1.f, b1.z), k3 = fmaf(x3, g1.w + 1.f, b1.w);
      Elem<T>::st(qp + i, q0 * wq.x - q1 * wq.y); Elem<T>::st(qp + i + 1, q0 * wq.y + q1 * wq.x);
      Elem<T>::st(qp + i + 2, q2 * wq.z - q3 * wq.w); Elem<T>::st(qp + i + 3, q2 * wq.w + q3 * wq.z);
      Elem<T>::st(kp + i, k0 * wk.x - k1 * wk.y); Elem<T>::st(kp + i + 1, k0 * wk.y + k1 * wk.x);
      Elem<T>::st(kp + i + 2, k2 * wk.z - k3 * wk.w); Elem<T>::st(kp + i + 3, k2 * wk.w + k3 * wk.z);
      Elem<T>::st(wp + i, k0); Elem<T>::st(wp + i + 1, k1); Elem<T>::st(wp + i + 2, k2); Elem<T>::st(wp + i + 3, k3);
    }
    const long long at = chunk * out_period + pos;
    *reinterpret_cast<uint4*>(qo + at * ldq + c) = qv;
    *reinterpret_cast<uint4*>(ko + at * ldk + c) = kv;
    if (kraw) *reinterpret_cast<uint4*>(kraw + r * kCols + c) = kw;
  }
}

}  // namespace mega

using namespace mega;

static int tsn_fwd_common(const void* x, void* y, int dtype, int B, int L, int D, int64_t xsb, int64_t xsl,
                          int64_t xsd, int64_t ysb, int64_t ysl, int64_t ysd, const int64_t* prev_count,
                          const float* prev_mean, const float* prev_var, const float* gamma, const float* beta,
                          const uint8_t* pad_mask, int num_groups, double eps, int64_t* count_out,
                          float* mean_out, float* var_out, float* cummean, float* cumrstd, float* group_mean,
                          mega_stream_t stream) {
  if (!x || !y || !prev_count || !prev_mean || !prev_var || !gamma || !beta || !count_out || !mean_out ||
      !var_out)
    return MEGA_ERR_NULL;
  // every thread block of a sequence reads its incoming count; one of them writes the new one
  if ((const void*)count_out == (const void*)prev_count) return MEGA_ERR_UNSUPPORTED;
  if (!valid_dtype(dtype)) return MEGA_ERR_DTYPE;
  if (B <= 0 || L <= 0 || D <= 0) return MEGA_ERR_SHAPE;
  const int G = (num_groups <= 0 || num_groups == D) ? D : num_groups;
  if (D % G != 0) return MEGA_ERR_SHAPE;
  if (!aligned_to(x, elem_size(dtype)) || !aligned_to(y, elem_size(dtype))) return MEGA_ERR_ALIGN;
  TsnArgs a{};
  a.x = x; a.y = y; a.B = B; a.L = L; a.D = D; a.G = G;
  a.xsb = xsb; a.xsl = xsl; a.xsd = xsd; a.ysb = ysb; a.ysl = ysl; a.ysd = ysd;
  a.prev_count = (const long long*)prev_count; a.prev_mean = prev_mean; a.prev_var = prev_var;
  a.gamma = gamma; a.beta = beta; a.mask = pad_mask; a.eps = (float)eps;
  a.count_out = (long long*)count_out; a.mean_out = mean_out; a.var_out = var_out;
  a.cummean = cummean; a.cumrstd = cumrstd; a.group_mean = group_mean;
  if (G == D) {
    if (x != y) {
      StreamArgs sa{};
      sa.B = B; sa.L = L; sa.D = D; sa.N = 0;
      sa.prev_count = a.prev_count; sa.prev_mean = prev_mean; sa.prev_var = prev_var; sa.gamma = gamma;
      sa.beta = beta; sa.eps = (float)eps; sa.count_out = a.count_out; sa.mean_out = mean_out; sa.var_out = var_out;
      sa.mask = pad_mask;
      sa.cummean = cummean; sa.cumrstd = cumrstd;
      // The walk of tmem_ema.cu (bf16, where there are enough sequences and channels: 16 x 4096 x 1024 67 us, 64 x 4096 x 2048 518) and
      // the scan (97, 641) take their statistics in fp32 (variances 1e-6 off), the tensor-core form from bf16 and tf32 operands
      // (3e-4; 142, and 4305 us at 64 x 32768 x 2048 where the scan takes 4969).
      if (!cummean && g_options[OPT_MMA_TILE].load() == 0 && g_options[OPT_DISABLE_MMA].load() == 0) {
        ScanNormArgs na{};
        na.x = x; na.y = y; na.B = B; na.D = D; na.L = L;
        na.xsb = xsb; na.xsl = xsl; na.ysb = ysb; na.ysl = ysl;
        na.prev_count = a.prev_count; na.prev_mean = prev_mean; na.prev_var = prev_var; na.gamma = gamma; na.beta = beta;
        na.mask = pad_mask; na.eps = (float)eps; na.count_out = a.count_out; na.mean_out = mean_out; na.var_out = var_out;
        // (statistics updated in place the scan does not take, and the tensor-core form has a shorter start, 13 x 53 x 32 7 us for 10; the
        // walk has it all the same, for what lasts is the variance)
        const int form = g_options[OPT_SPLIT].load();
        if (xsd == 1 && ysd == 1 && form != 3 && (form == 4 || tmem_norm_us(sa) < 0.9 * scan_norm_us(na)) &&
            tmem_norm_try(dtype, x, y, xsb, xsl, ysb, ysl, sa, (cudaStream_t)stream))
          return check_launch("timestep_norm_fwd(tmem)");
        if (scan_norm_fwd_try(dtype, na, xsd, ysd, (cudaStream_t)stream)) return check_launch("timestep_norm_fwd(scan)");
      }
      // (statistics updated in place where the walk of tmem_ema.cu, which may do so, is not the faster one; a form of the tensor-core
      // kernel asked for by name; or the streamed kernel)
      if (!cummean && mma_cl_try(dtype, x, y, nullptr, xsb, xsl, xsd, ysb, ysl, ysd, true, sa, (cudaStream_t)stream))
        return check_launch("timestep_norm_fwd(mma)");
      if (stream_cl_try(dtype, x, y, nullptr, xsb, xsl, xsd, ysb, ysl, ysd, false, sa, (cudaStream_t)stream))
        return check_launch("timestep_norm_fwd(stream)");
    }
    const unsigned grid = (unsigned)(((long long)B * D + 127) / 128);
    MEGA_DISPATCH_DTYPE(dtype, {
      if (pad_mask && cummean) launch(tsn_plain_kernel<T, true, true>, grid, 128, 0, stream, a);
      else if (pad_mask) launch(tsn_plain_kernel<T, true, false>, grid, 128, 0, stream, a);
      else if (cummean) launch(tsn_plain_kernel<T, false, true>, grid, 128, 0, stream, a);
      else launch(tsn_plain_kernel<T, false, false>, grid, 128, 0, stream, a);
    });
  } else {
    GroupNormArgs ga{};
    ga.B = B; ga.L = L; ga.D = D; ga.G = G;
    ga.prev_count = a.prev_count; ga.prev_mean = prev_mean; ga.prev_var = prev_var; ga.gamma = gamma; ga.beta = beta;
    ga.mask = pad_mask; ga.eps = (float)eps; ga.count_out = a.count_out; ga.mean_out = mean_out; ga.var_out = var_out;
    ga.cummean = cummean; ga.cumrstd = cumrstd; ga.group_mean = group_mean;
    if (group_norm_try(dtype, x, y, xsb, xsl, xsd, ysb, ysl, ysd, ga, (cudaStream_t)stream))
      return check_launch("timestep_norm_fwd(group)");
    const unsigned grid = (unsigned)(((long long)B * G * 32 + 127) / 128);
    MEGA_DISPATCH_DTYPE(dtype, launch(tsn_group_kernel<T>, grid, 128, 0, stream, a));
  }
  return check_launch("timestep_norm_fwd");
}

extern "C" int mega_timestep_norm_fwd(const void* x, void* y, int dtype, int B, int L, int D, int64_t xsb,
                                      int64_t xsl, int64_t xsd, int64_t ysb, int64_t ysl, int64_t ysd,
                                      const int64_t* prev_count, const float* prev_mean,
                                      const float* prev_var, const float* gamma, const float* beta,
                                      const uint8_t* pad_mask, int num_groups, double eps,
                                      int64_t* count_out, float* mean_out, float* var_out,
                                      mega_stream_t stream) {
  return tsn_fwd_common(x, y, dtype, B, L, D, xsb, xsl, xsd, ysb, ysl, ysd, prev_count, prev_mean, prev_var,
                        gamma, beta, pad_mask, num_groups, eps, count_out, mean_out, var_out, nullptr, nullptr,
                        nullptr, stream);
}

extern "C" int mega_timestep_norm_fwd_train(const void* x, void* y, int dtype, int B, int L, int D, int64_t xsb,
                                            int64_t xsl, int64_t xsd, int64_t ysb, int64_t ysl, int64_t ysd,
                                            const int64_t* prev_count, const float* prev_mean,
                                            const float* prev_var, const float* gamma, const float* beta,
                                            const uint8_t* pad_mask, int num_groups, double eps,
                                            int64_t* count_out, float* mean_out, float* var_out, float* cummean,
                                            float* cumrstd, float* group_mean, mega_stream_t stream) {
  if (!cummean || !cumrstd) return MEGA_ERR_NULL;
  const bool grouped = num_groups > 0 && num_groups != D;
  if (grouped && !group_mean) return MEGA_ERR_NULL;
  return tsn_fwd_common(x, y, dtype, B, L, D, xsb, xsl, xsd, ysb, ysl, ysd, prev_count, prev_mean, prev_var,
                        gamma, beta, pad_mask, num_groups, eps, count_out, mean_out, var_out, cummean, cumrstd,
                        grouped ? group_mean : nullptr, stream);
}

extern "C" int mega_sequence_norm_fwd(const void* x, void* y, int dtype, int B, int D, int L, int64_t xsb,
                                      int64_t xsd, int64_t xsl, int64_t ysb, int64_t ysd, int64_t ysl,
                                      const float* gamma, const float* beta, const uint8_t* pad_mask,
                                      int num_groups, double eps, int64_t* count_out, float* mean_out,
                                      float* rstd_out, mega_stream_t stream) {
  if (!x || !y || !gamma || !beta || !count_out || !mean_out || !rstd_out) return MEGA_ERR_NULL;
  if (!valid_dtype(dtype)) return MEGA_ERR_DTYPE;
  if (B <= 0 || L <= 0 || D <= 0) return MEGA_ERR_SHAPE;
  const int G = (num_groups <= 0 || num_groups == D) ? D : num_groups;
  if (D % G != 0) return MEGA_ERR_SHAPE;
  if (!aligned_to(x, elem_size(dtype)) || !aligned_to(y, elem_size(dtype))) return MEGA_ERR_ALIGN;
  SqnArgs a{};
  a.x = x; a.y = y; a.B = B; a.D = D; a.L = L; a.G = G;
  a.xsb = xsb; a.xsd = xsd; a.xsl = xsl; a.ysb = ysb; a.ysd = ysd; a.ysl = ysl;
  a.gamma = gamma; a.beta = beta; a.mask = pad_mask; a.eps = (float)eps;
  a.count_out = (long long*)count_out; a.mean_out = mean_out; a.rstd_out = rstd_out;
  if (G == D && xsd == 1 && xsl != 1 && x != y) {
    ScanNormArgs na{};
    na.x = x; na.y = y; na.B = B; na.D = D; na.L = L;
    na.xsb = xsb; na.xsl = xsl; na.ysb = ysb; na.ysl = ysl;
    na.gamma = gamma; na.beta = beta; na.mask = pad_mask; na.eps = (float)eps;
    na.count_out = a.count_out; na.mean_out = mean_out; na.var_out = rstd_out;
    if (scan_sqn_fwd_try(dtype, na, xsd, ysd, (cudaStream_t)stream)) return check_launch("sequence_norm_fwd(scan)");
  }
  if (G == D && xsd == 1 && xsl != 1) {
    const unsigned grid = (unsigned)(((long long)B * D + 127) / 128);
    MEGA_DISPATCH_DTYPE(dtype, launch(sqn_column_kernel<T>, grid, 128, 0, stream, a));
  } else {
    if ((long long)B * G > 0x7fffffffLL) return MEGA_ERR_SHAPE;
    const long long n = (long long)(D / G) * L;
    // cache the segment in shared memory when it fits (opt-in limit, leaves room for 1 KB of statics)
    static bool attr_ok = false;
    static std::once_flag once;
    std::call_once(once, [] {
      attr_ok = cudaFuncSetAttribute(sqn_segment_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) == cudaSuccess &&
                cudaFuncSetAttribute(sqn_segment_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) == cudaSuccess &&
                cudaFuncSetAttribute(sqn_segment_kernel<__half>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) == cudaSuccess;
      cudaGetLastError();
    });
    const int cap = (attr_ok ? 200 : 40) * 1024 / 4;
    const int cache_elems = n <= cap ? (int)n : 0;
    MEGA_DISPATCH_DTYPE(dtype, launch(sqn_segment_kernel<T>, (unsigned)(B * G), 256,
                                      (size_t)cache_elems * sizeof(float), stream, a, cache_elems));
  }
  return check_launch("sequence_norm_fwd");
}

static int gate_common(int op, const void* a, int64_t lda, const void* b, int64_t ldb, const void* c,
                       int64_t ldc, const void* d, int64_t ldd, void* y, int64_t ldy, int dtype,
                       int64_t rows, int cols, mega_stream_t stream) {
  if (!valid_dtype(dtype)) return MEGA_ERR_DTYPE;
  if (rows <= 0 || cols <= 0) return MEGA_ERR_SHAPE;
  const long long n = rows * cols;
  {
    // 16-byte path: every operand present has a 16-byte aligned base and pitch, cols a multiple of the vector
    const int vn = 16 / elem_size(dtype);
    const long long es = elem_size(dtype);
    auto ok16 = [&](const void* p, long long ld) { return p == nullptr || (aligned_to(p, 16) && (ld * es) % 16 == 0); };
    const int vpr = cols / vn;
    int bx = 32;
    while (bx < vpr && bx < 256) bx *= 2;
    constexpr int kU = 4;
    const int by = 256 / bx;
    const long long gx = (rows + by * kU - 1) / (by * kU);
    if (cols % vn == 0 && ok16(a, lda) && ok16(b, ldb) && ok16(c, ldc) && ok16(d, ldd) && ok16(y, ldy) && gx < 0x7fffffffLL) {
      const dim3 gridv((unsigned)gx, (unsigned)((vpr + bx - 1) / bx)), blockv(bx, by);
      MEGA_DISPATCH_DTYPE(dtype, {
        auto run = [&](auto kernel) {
          launch(kernel, gridv, blockv, 0, stream, (const T*)a, lda, (const T*)b, ldb, (const T*)c, ldc, (const T*)d, ldd, (T*)y, ldy,
                 rows, cols);
        };
        if (op == 0) run(gate_vec_kernel<T, 0, kU>);
        else if (op == 1) run(gate_vec_kernel<T, 1, kU>);
        else run(gate_vec_kernel<T, 2, kU>);
      });
      return check_launch("gate");
    }
  }
  const unsigned grid = (unsigned)((n + 255) / 256 > 148 * 16 ? 148 * 16 : (n + 255) / 256);
  MEGA_DISPATCH_DTYPE(dtype, {
    if (op == 0)
      launch(gate_kernel<T, 0>, grid, 256, 0, stream, (const T*)a, lda, (const T*)b, ldb, (const T*)c, ldc,
             (const T*)d, ldd, (T*)y, ldy, rows, cols);
    else if (op == 1)
      launch(gate_kernel<T, 1>, grid, 256, 0, stream, (const T*)a, lda, (const T*)b, ldb, (const T*)c, ldc,
             (const T*)d, ldd, (T*)y, ldy, rows, cols);
    else
      launch(gate_kernel<T, 2>, grid, 256, 0, stream, (const T*)a, lda, (const T*)b, ldb, (const T*)c, ldc,
             (const T*)d, ldd, (T*)y, ldy, rows, cols);
  });
  return check_launch("gate");
}

extern "C" int mega_gate_silu(const void* a, int64_t ld_a, const void* b, int64_t ld_b, void* y,
                              int64_t ld_y, int dtype, int64_t rows, int cols, mega_stream_t stream) {
  if (!a || !y) return MEGA_ERR_NULL;
  return gate_common(0, a, ld_a, b, ld_b, nullptr, 0, nullptr, 0, y, ld_y, dtype, rows, cols, stream);
}

extern "C" int mega_gate_mul_silu(const void* a, int64_t ld_a, const void* r, int64_t ld_r, void* y,
                                  int64_t ld_y, int dtype, int64_t rows, int cols, mega_stream_t stream) {
  if (!a || !r || !y) return MEGA_ERR_NULL;
  return gate_common(1, a, ld_a, r, ld_r, nullptr, 0, nullptr, 0, y, ld_y, dtype, rows, cols, stream);
}

extern "C" int mega_gate_output(const void* residual, int64_t ld_res, const void* u, int64_t ld_u,
                                const void* hx, int64_t ld_hx, const void* h_lin, int64_t ld_h, void* out,
                                int64_t ld_out, int dtype, int64_t rows, int cols, mega_stream_t stream) {
  if (!residual || !u || !hx || !h_lin || !out) return MEGA_ERR_NULL;
  return gate_common(2, residual, ld_res, u, ld_u, hx, ld_hx, h_lin, ld_h, out, ld_out, dtype, rows, cols,
                     stream);
}

extern "C" int mega_gate_qk(const void* z, int64_t ld_z, const float* gamma, const float* beta, void* q,
                            int64_t ld_q, void* k, int64_t ld_k, int dtype, int64_t rows, int cols, double eps,
                            mega_stream_t stream) {
  if (!z || !gamma || !beta || !q || !k) return MEGA_ERR_NULL;
  if (!valid_dtype(dtype)) return MEGA_ERR_DTYPE;
  if (rows <= 0 || cols <= 0) return MEGA_ERR_SHAPE;
  if (ld_z < cols || ld_q < cols || ld_k < cols) return MEGA_ERR_STRIDE;
  const long long blocks = (rows + 7) / 8;  // 8 warps per block, one row per warp and pass
  const unsigned grid = (unsigned)(blocks > 148 * 8 ? 148 * 8 : blocks);
  MEGA_DISPATCH_DTYPE(dtype, launch(gate_qk_kernel<T>, grid, 256, 0, stream, (const T*)z, (long long)ld_z, gamma,
                                    beta, (T*)q, (long long)ld_q, (T*)k, (long long)ld_k, (long long)rows, cols,
                                    (float)eps));
  return check_launch("gate_qk");
}

extern "C" int mega_gate_qk_rotary_cache(const void* z, int64_t ld_z, const float* gamma, const float* beta, const float* rot,
                                         int positions, int period, int q_offset, int out_period, void* q, int64_t ld_q, void* k,
                                         int64_t ld_k, void* k_raw, int dtype, int64_t rows, int cols, double eps,
                                         mega_stream_t stream) {
  if (!z || !gamma || !beta || !rot || !q || !k) return MEGA_ERR_NULL;
  if (!valid_dtype(dtype)) return MEGA_ERR_DTYPE;
  if (rows <= 0 || cols <= 0 || (cols & 1) || period <= 0 || out_period < period || q_offset < 0 || period + q_offset > positions)
    return MEGA_ERR_SHAPE;
  if (ld_z < cols || ld_q < cols || ld_k < cols) return MEGA_ERR_STRIDE;
  if (!aligned_to(rot, 8)) return MEGA_ERR_ALIGN;
  const bool vec = elem_size(dtype) == 2 && (cols == 64 || cols == 128 || cols == 256) && ld_z % 8 == 0 && ld_q % 8 == 0 &&
                   ld_k % 8 == 0 && aligned_to(z, 16) && aligned_to(q, 16) && aligned_to(k, 16) && aligned_to(k_raw, 16) &&
                   aligned_to(gamma, 16) && aligned_to(beta, 16) && aligned_to(rot, 16);
  if (vec) {
    const int per = 8 * 2 * (256 / cols);   // rows of a block: eight warps
    const unsigned grid = (unsigned)((rows + per - 1) / per);
#define MEGA_QK(T)                                                                                                        \
  {                                                                                                                       \
    auto run = [&](auto kernel) {                                                                                         \
      launch(kernel, grid, 256, 0, stream, (const T*)z, (long long)ld_z, gamma, beta, rot, period, q_offset, out_period, (T*)q, \
             (long long)ld_q, (T*)k, (long long)ld_k, (T*)k_raw, (long long)rows, (float)eps);                            \
    };                                                                                                                    \
    if (cols == 64) run(gate_qk_rotary_vec_kernel<T, 8>);                                                                 \
    else if (cols == 128) run(gate_qk_rotary_vec_kernel<T, 16>);                                                          \
    else run(gate_qk_rotary_vec_kernel<T, 32>);                                                                           \
  }
    if (dtype == MEGA_BF16) MEGA_QK(__nv_bfloat16) else MEGA_QK(__half)
#undef MEGA_QK
    return check_launch("gate_qk_rotary");
  }
  const long long blocks = (rows + 7) / 8;  // 8 warps per block, one row per warp and pass
  const unsigned grid = (unsigned)(blocks > 148 * 8 ? 148 * 8 : blocks);
  MEGA_DISPATCH_DTYPE(dtype, launch(gate_qk_rotary_kernel<T>, grid, 256, 0, stream, (const T*)z, (long long)ld_z, gamma,
                                    beta, rot, period, q_offset, out_period, (T*)q, (long long)ld_q, (T*)k, (long long)ld_k,
                                    (T*)k_raw, (long long)rows, cols, (float)eps));
  return check_launch("gate_qk_rotary");
}

extern "C" int mega_gate_qk_rotary(const void* z, int64_t ld_z, const float* gamma, const float* beta, const float* rot,
                                   int positions, int period, int q_offset, void* q, int64_t ld_q, void* k,
                                   int64_t ld_k, int dtype, int64_t rows, int cols, double eps, mega_stream_t stream) {
  return mega_gate_qk_rotary_cache(z, ld_z, gamma, beta, rot, positions, period, q_offset, period, q, ld_q, k, ld_k, nullptr, dtype,
                                   rows, cols, eps, stream);
}

extern "C" int mega_norm_prepare(const int64_t* prior_count, const void* prior_mean, const void* prior_logv, const void* weight,
                                 const void* bias, int dtype, int B, int G, int D, int64_t* count, float* mean, float* var,
                                 float* gamma, float* beta, mega_stream_t stream) {
  if (!weight || !bias || !gamma || !beta) return MEGA_ERR_NULL;
  if (B > 0 && (!prior_count || !prior_mean || !prior_logv || !count || !mean || !var)) return MEGA_ERR_NULL;
  if (!valid_dtype(dtype)) return MEGA_ERR_DTYPE;
  if (D <= 0 || B < 0 || (B > 0 && G <= 0)) return MEGA_ERR_SHAPE;
  int n = D > B ? D : B;
  if (B > 0 && G > n) n = G;
  const dim3 grid((n + 127) / 128, B > 8 ? 8 : B > 0 ? B : 1);
  MEGA_DISPATCH_DTYPE(dtype, launch_after(norm_prepare_kernel<T>, grid, dim3(128), 0, stream,
                                    (const long long*)prior_count, (const T*)prior_mean, (const T*)prior_logv,
                                    (const T*)weight, (const T*)bias, B, B > 0 ? G : 0, D, (long long*)count, mean, var, gamma,
                                    beta));
  return check_launch("norm_prepare");
}

extern "C" int mega_norm_finish(const float* dprev_mean, const float* dprev_var, const void* prior_logv, const float* dgamma,
                                const float* dbeta, int dtype, int B, int G, int D, void* dprior_mean, void* dprior_logv,
                                void* dweight, void* dbias, mega_stream_t stream) {
  if (!dgamma || !dbeta || !dweight || !dbias) return MEGA_ERR_NULL;
  if (B > 0 && (!dprev_mean || !dprev_var || !prior_logv || !dprior_mean || !dprior_logv)) return MEGA_ERR_NULL;
  if (!valid_dtype(dtype)) return MEGA_ERR_DTYPE;
  if (D <= 0 || B < 0 || (B > 0 && (G <= 0 || G > D))) return MEGA_ERR_SHAPE;
  MEGA_DISPATCH_DTYPE(dtype, launch(norm_finish_kernel<T>, (unsigned)((D + 127) / 128), 128, 0, stream, dprev_mean, dprev_var,
                                    (const T*)prior_logv, dgamma, dbeta, B, B > 0 ? G : 0, D, (T*)dprior_mean,
                                    (T*)dprior_logv, (T*)dweight, (T*)dbias));
  return check_launch("norm_finish");
}
