// Grouped TimestepNorm, forward and backward, parallel over time (channel-contiguous activations).
//
// The norm pools the statistics of the D / G channels of a group at every step and combines them over the
// steps.  Only that combination is serial, it is one value per step and group, and it is associative, so
// a pass is three launches: (1) the moments of every (step, group), a vector of 16 bytes per lane and
// shuffles inside the group; (2) a scan over the steps, one block per sequence and 2 or 8 groups, 256 or 128
// threads along time: each walks its run of steps, the runs are combined across the threads (Chan's rule for
// counts, means and squared deviations), each walks its run again from what came before; (3) the
// elementwise part.  The backward is the same with the reverse scan written as plain suffix sums: with
// V = dL/dvar / n and U = dL/dmean / n at count n the recurrence of the reference
// (fairseq/csrc/ops/timestep_norm.cc:318-446) becomes
//   V_{n-1} = V_n - r^3 ds / (2 n),   U_{n-1} = U_n - r db / n - 2 (ux - pu) / n * V_{n-1}.
// Bound: HBM, x twice (once from L2 when it fits) and y once.  B = 4, L = 4096, D = 1024, 32 groups, bf16:
// the walk over the steps inside one block per 64 channels took 1906 us forward and 2591 us backward.
// Group sizes: powers of two from one vector to 256 channels; others use the generic kernel.
#include "common.cuh"
#include "scratch.cuh"
#include "stream_bwd.cuh"

namespace mega {

namespace {

constexpr int kRowsPerBlock = 32;   // rows (sequence, step) of a block of the moment and elementwise kernels
// The scan's blocks take 2 groups with 256 threads along time while there are no more of them than SMs, else 8 with 128: it is
// issue slots and latency, so it goes over as many SMs as there are pairs (4 sequences of 32 groups at L = 4096: 36 us forward
// and 20 backward against 48 + 12 and 23 + 21; one group would read a sector of 32 bytes for each float), but beyond the SMs half
// of a sector is read twice (forward and backward of 10 sequences of 12 groups at L = 2805: 174 us against 186; of 27 of 24 at
// 1256 218 against 195).
bool by_pairs(int B, int G) { return (long long)B * ((G + 1) / 2) <= 148; }

template <typename T>
struct Vec {
  static constexpr int kN = 16 / (int)sizeof(T);
  static __device__ __forceinline__ void load(const T* p, float (&f)[kN]) {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
    const T* e = reinterpret_cast<const T*>(&v);
#pragma unroll
    for (int k = 0; k < kN; ++k) f[k] = Elem<T>::ld_shared(e + k);
  }
  static __device__ __forceinline__ void store(T* p, const float (&f)[kN]) {
    uint4 v;
    T* e = reinterpret_cast<T*>(&v);
#pragma unroll
    for (int k = 0; k < kN; ++k) Elem<T>::st(e + k, f[k]);
    *reinterpret_cast<uint4*>(p) = v;
  }
};

// sum over `width` neighbouring lanes (a power of two)
__device__ __forceinline__ float lanes_sum(float v, int width) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    if (o < width) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---- forward ---------------------------------------------------------------------------------
// A warp takes rows; lane l of pass k owns the vector 32 k + l of the row.
template <typename T>
__global__ void __launch_bounds__(256) group_moments_kernel(const T* x, long long xsb, long long xsl, int L, int D, int G,
                                                            long long rows, float* gm_out, float* gv_out) {
  constexpr int kN = Vec<T>::kN;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gs = D / G, width = gs / kN;   // lanes per group (1 .. 32)
  const float inv = 1.f / (float)gs;
  const int nv = D / kN;
  for (int rr = warp; rr < kRowsPerBlock; rr += 8) {
    const long long r = (long long)blockIdx.x * kRowsPerBlock + rr;
    if (r >= rows) return;
    const T* xr = x + (r / L) * xsb + (r % L) * xsl;
    for (int v0 = 0; v0 < nv; v0 += 32) {   // (nv is a multiple of width: a group never straddles the end)
      const int v = v0 + lane;
      float f[kN];
#pragma unroll
      for (int k = 0; k < kN; ++k) f[k] = 0.f;
      if (v < nv) Vec<T>::load(xr + (long long)v * kN, f);
      float s = 0.f;
#pragma unroll
      for (int k = 0; k < kN; ++k) s += f[k];
      const float m = lanes_sum(s, width) * inv;
      float q = 0.f;
#pragma unroll
      for (int k = 0; k < kN; ++k) q = fmaf(f[k] - m, f[k] - m, q);
      q = lanes_sum(q, width) * inv;
      if (v < nv && (lane & (width - 1)) == 0) {
        gm_out[r * G + v / width] = m;
        gv_out[r * G + v / width] = q;
      }
    }
  }
}

// Statistics of a run of steps: count, mean, squared deviations (Chan et al.'s pairwise combination).
struct Run {
  float n, m, s;
};
__device__ __forceinline__ Run combine(Run a, Run b) {
  const float n = a.n + b.n;
  if (b.n == 0.f) return a;
  if (a.n == 0.f) return b;
  const float w = b.n / n, d = b.m - a.m;
  return {n, fmaf(d, w, a.m), a.s + b.s + d * d * a.n * w};
}

template <int kScanG, int kScanT>
__global__ void __launch_bounds__(kScanG* kScanT) group_scan_kernel(const float* gm, const float* gv, int L, int G,
                                                                    const long long* prev_count, const float* prev_mean,
                                                                    const float* prev_var, const unsigned char* mask,
                                                                    float eps, float* cummean, float* cumrstd,
                                                                    long long* count_out, float* mean_out, float* var_out) {
  __shared__ Run part[kScanT][kScanG];
  const int gi = threadIdx.x % kScanG, ti = threadIdx.x / kScanG;
  const int b = blockIdx.y, g = blockIdx.x * kScanG + gi;
  const bool ok = g < G;
  const int per = (L + kScanT - 1) / kScanT;
  const int t0 = min(L, ti * per), t1 = min(L, t0 + per);
  const unsigned char* mp = mask ? mask + (size_t)b * L : nullptr;
  const size_t base = (size_t)b * L * G + g;
  // (the loads of several steps go out together: one at a time, each waited for the one before, 31 us at L = 4096 and
  // 32 groups)
  constexpr int kFwdB = 8;
  float ms[kFwdB], vs[kFwdB];
  bool skip[kFwdB];
  auto fetch = [&](int k) {
#pragma unroll
    for (int j = 0; j < kFwdB; ++j) {
      const int t = min(k + j, t1 - 1);
      ms[j] = __ldg(gm + base + (size_t)t * G);
      vs[j] = __ldg(gv + base + (size_t)t * G);
      skip[j] = k + j >= t1 || (mp && mp[t]);
    }
  };
  // own run: sums about its first value
  Run r{0.f, 0.f, 0.f};
  if (ok) {
    float c = 0.f, s1 = 0.f, s2 = 0.f, n = 0.f;
    for (int k = t0; k < t1; k += kFwdB) {
      fetch(k);
#pragma unroll
      for (int j = 0; j < kFwdB; ++j) {
        if (skip[j]) continue;
        if (n == 0.f) c = ms[j];
        const float d = ms[j] - c;
        s1 += d;
        s2 += fmaf(d, d, vs[j]);
        n += 1.f;
      }
    }
    if (n > 0.f) r = {n, c + s1 / n, not_negative(s2 - s1 * s1 / n)};
  }
  part[ti][gi] = r;
  __syncthreads();
  // inclusive scan over the threads along time (seven or eight rounds)
#pragma unroll
  for (int o = 1; o < kScanT; o <<= 1) {
    Run mine = part[ti][gi];
    if (ti >= o) mine = combine(part[ti - o][gi], mine);
    __syncthreads();
    part[ti][gi] = mine;
    __syncthreads();
  }
  const long long cnt0 = prev_count[b];
  const size_t at = (size_t)b * G + (ok ? g : 0);
  const float mean0 = prev_mean[at], var0 = prev_var[at];
  __syncthreads();   // (mean_out and var_out may be prev_mean and prev_var: all threads have read them)
  if (!ok) return;
  const Run prior{(float)cnt0, mean0, var0 * (float)cnt0};
  Run in = prior;
  if (ti > 0) in = combine(prior, part[ti - 1][gi]);
  // second walk, sums about the mean that came in (or the first value when nothing did)
  // (the thread's own steps counted from zero: one by one they would be lost on a count beyond 2^24)
  float c = in.m, s1 = 0.f, s2 = 0.f, seen = 0.f;
  const float n0 = in.n;
  float n = n0;
  float mean = in.n > 0.f ? in.m : prior.m, var = in.n > 0.f ? in.s / in.n : var0;
  for (int k = t0; k < t1; k += kFwdB) {
    fetch(k);
#pragma unroll
    for (int j = 0; j < kFwdB; ++j) {
      if (!skip[j]) {
        if (n == 0.f) c = ms[j];
        const float d = ms[j] - c;
        s1 += d;
        s2 += fmaf(d, d, vs[j]);
        seen += 1.f;
        n = n0 + seen;
        const float inv = 1.f / n, u = s1 * inv;
        mean = c + u;
        var = not_negative(fmaf(-u, u, (in.s + s2) * inv));
      }
      if (k + j < t1) {
        const size_t i = base + (size_t)(k + j) * G;
        cummean[i] = mean;
        cumrstd[i] = rsqrtf(var + eps);
      }
    }
  }
  if (ti == kScanT - 1) {
    const Run all = part[ti][gi];
    const Run fin = combine(prior, all);
    mean_out[(size_t)b * G + g] = fin.n > 0.f ? fin.m : prior.m;
    var_out[(size_t)b * G + g] = fin.n > 0.f ? fin.s / fin.n : var0;
    if (g == 0) count_out[b] = cnt0 + (long long)(all.n + 0.5f);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) group_apply_kernel(const T* x, T* y, long long xsb, long long xsl, long long ysb,
                                                          long long ysl, int L, int D, int G, long long rows,
                                                          const float* cummean, const float* cumrstd, const float* gamma,
                                                          const float* beta, const unsigned char* mask) {
  constexpr int kN = Vec<T>::kN;
  const int nv = D / kN, width = D / G / kN;
  const long long total = rows * nv;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < total; i += (long long)gridDim.x * 256) {
    const long long r = i / nv;
    const int v = (int)(i - r * nv);
    const long long b = r / L, t = r - b * L;
    float f[kN], o[kN];
    Vec<T>::load(x + b * xsb + t * xsl + (long long)v * kN, f);
    const float m = __ldg(cummean + r * G + v / width), rs = __ldg(cumrstd + r * G + v / width);
    const bool mk = mask && mask[r];
#pragma unroll
    for (int k = 0; k < kN; ++k)
      o[k] = mk ? 0.f : fmaf((f[k] - m) * rs, __ldg(gamma + v * kN + k), __ldg(beta + v * kN + k));
    Vec<T>::store(y + b * ysb + t * ysl + (long long)v * kN, o);
  }
}

// ---- backward ----------------------------------------------------------------------------------
// ds = sum dy (x - u) w, db = sum dy w per (step, group); per-channel sums for dgamma and dbeta: a thread
// owns one vector of channels and every eighth row of the block.
template <typename T>
__global__ void __launch_bounds__(256) group_bwd_sums_kernel(const T* dy, const T* x, long long gsb, long long gsl,
                                                             long long xsb, long long xsl, int L, int D, int G,
                                                             long long rows, const float* cummean, const float* cumrstd,
                                                             const float* gamma, const unsigned char* mask, float* ds_out,
                                                             float* db_out, float* dgamma, float* dbeta) {
  constexpr int kN = Vec<T>::kN;
  __shared__ float red[8][32 * kN + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nv = D / kN, width = D / G / kN;
  const int v = blockIdx.y * 32 + lane;
  const bool ok = v < nv;
  float w[kN], wg[kN], bg[kN];
#pragma unroll
  for (int k = 0; k < kN; ++k) {
    w[k] = ok ? __ldg(gamma + v * kN + k) : 0.f;
    wg[k] = bg[k] = 0.f;
  }
  for (int rr = warp; rr < 4 * kRowsPerBlock; rr += 8) {
    const long long r = (long long)blockIdx.x * (4 * kRowsPerBlock) + rr;
    if (r >= rows) break;
    const bool mk = mask && mask[r];
    float ds = 0.f, db = 0.f;
    if (ok && !mk) {
      const long long b = r / L, t = r - b * L;
      float fx[kN], fy[kN];
      Vec<T>::load(x + b * xsb + t * xsl + (long long)v * kN, fx);
      Vec<T>::load(dy + b * gsb + t * gsl + (long long)v * kN, fy);
      const float u = __ldg(cummean + r * G + v / width), rs = __ldg(cumrstd + r * G + v / width);
#pragma unroll
      for (int k = 0; k < kN; ++k) {
        const float e = fx[k] - u, p = fy[k] * w[k];
        ds = fmaf(p, e, ds);
        db += p;
        wg[k] = fmaf(fy[k] * e, rs, wg[k]);
        bg[k] += fy[k];
      }
    }
    ds = lanes_sum(ds, width);
    db = lanes_sum(db, width);
    if (ok && (lane & (width - 1)) == 0) {
      ds_out[r * G + v / width] = ds;
      db_out[r * G + v / width] = db;
    }
  }
  for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
    for (int k = 0; k < kN; ++k) red[warp][lane * kN + k] = pass == 0 ? wg[k] : bg[k];
    __syncthreads();
    for (int c = threadIdx.x; c < 32 * kN; c += 256) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) s += red[i][c];
      const int d = blockIdx.y * 32 * kN + c;
      if (d < D) atomicAdd((pass == 0 ? dgamma : dbeta) + d, s);
    }
    __syncthreads();
  }
}

// Reverse scan.  A run of steps maps (V, U) to (V + sv, U + su + sw V); runs compose associatively.
struct Map {
  float n, sv, su, sw;   // n: unmasked steps of the run
};
// `late` runs first (it lies later in time), then `early`
__device__ __forceinline__ Map compose(Map late, Map early) {
  return {late.n + early.n, late.sv + early.sv, late.su + early.su + early.sw * late.sv, late.sw + early.sw};
}

template <int kScanG, int kScanT>
__global__ void __launch_bounds__(kScanG* kScanT) group_bwd_scan_kernel(const float* ds, const float* db, int L, int G,
                                                                        const float* cummean, const float* cumrstd,
                                                                        const float* group_mean, const float* prev_mean,
                                                                        const long long* count, const float* dmean,
                                                                        const float* dvar, const unsigned char* mask,
                                                                        float* dux, float* dvx, float* dprev_mean,
                                                                        float* dprev_var) {
  __shared__ Map part[kScanT][kScanG];
  __shared__ float cnts[kScanT];
  const int gi = threadIdx.x % kScanG, ti = threadIdx.x / kScanG;   // ti = 0 owns the latest steps
  const int b = blockIdx.y, g = blockIdx.x * kScanG + gi;
  const bool ok = g < G;
  const int per = (L + kScanT - 1) / kScanT;
  const int hi = max(0, L - ti * per), lo = max(0, hi - per);       // steps hi - 1 down to lo
  const unsigned char* mp = mask ? mask + (size_t)b * L : nullptr;
  const size_t base = (size_t)b * L * G + g;
  // unmasked steps of the later runs, for this run's counts
  if (gi == 0) {
    int c = 0;
    if (mp) {
      for (int t = lo; t < hi; ++t) c += mp[t] ? 0 : 1;
    } else {
      c = hi - lo;
    }
    cnts[ti] = (float)c;
  }
  __syncthreads();
  float later = mp ? 0.f : (float)min(L, ti * per);
  if (mp)
    for (int i = 0; i < ti; ++i) later += cnts[i];
  const float n_end = (float)count[b];
  const float n_in = n_end - later;   // count after this run's last step (its own steps are counted apart: see the forward)
  auto prev_u = [&](int t) -> float { return t > 0 ? __ldg(cummean + base + (size_t)(t - 1) * G) : prev_mean[(size_t)b * G + g]; };
  constexpr int kBwdB = 4;   // (steps whose loads go out together)
  float lr[kBwdB], le[kBwdB], ls[kBwdB], lb[kBwdB];
  bool skip[kBwdB];
  auto fetch = [&](int k) {   // steps k, k - 1, ...
#pragma unroll
    for (int j = 0; j < kBwdB; ++j) {
      const int t = max(k - j, lo);
      const size_t i = base + (size_t)t * G;
      lr[j] = __ldg(cumrstd + i);
      le[j] = 2.f * (__ldg(group_mean + i) - prev_u(t));
      ls[j] = __ldg(ds + i);
      lb[j] = __ldg(db + i);
      skip[j] = k - j < lo || (mp && mp[t]);
    }
  };
  Map m{0.f, 0.f, 0.f, 0.f};
  if (ok) {
    for (int k = hi - 1; k >= lo; k -= kBwdB) {
      fetch(k);
#pragma unroll
      for (int j = 0; j < kBwdB; ++j) {
        if (skip[j]) continue;
        const float rs = lr[j], inv = 1.f / (n_in - m.n), e = le[j] * inv;
        m.sv -= 0.5f * (rs * rs * rs) * ls[j] * inv;
        m.su -= fmaf(e, m.sv, rs * lb[j] * inv);
        m.sw -= e;
        m.n += 1.f;
      }
    }
  }
  part[ti][gi] = m;
  __syncthreads();
#pragma unroll
  for (int o = 1; o < kScanT; o <<= 1) {
    Map mine = part[ti][gi];
    if (ti >= o) mine = compose(part[ti - o][gi], mine);
    __syncthreads();
    part[ti][gi] = mine;
    __syncthreads();
  }
  if (!ok) return;
  const float v0 = (dvar && n_end > 0.f) ? dvar[(size_t)b * G + g] / n_end : 0.f;
  const float u0 = (dmean && n_end > 0.f) ? dmean[(size_t)b * G + g] / n_end : 0.f;
  float V = v0, U = u0;
  if (ti > 0) {
    const Map p = part[ti - 1][gi];
    V = v0 + p.sv;
    U = u0 + p.su + p.sw * v0;
  }
  float done = 0.f;
  for (int k = hi - 1; k >= lo; k -= kBwdB) {
    fetch(k);
#pragma unroll
    for (int j = 0; j < kBwdB; ++j) {
      float ou = 0.f, ov = 0.f;
      if (!skip[j]) {
        const float rs = lr[j], n = n_in - done, inv = 1.f / n, e = le[j];
        V -= 0.5f * (rs * rs * rs) * ls[j] * inv;
        const float h = U - rs * lb[j] * inv;
        ov = V;
        ou = fmaf((n - 1.f) * inv * e, V, h);
        U = fmaf(-e * inv, V, h);
        done += 1.f;
      }
      if (k - j >= lo) {
        const size_t i = base + (size_t)(k - j) * G;
        dux[i] = ou;
        dvx[i] = ov;
      }
    }
  }
  if (ti == kScanT - 1) {
    const Map all = part[ti][gi];
    const float n0 = n_end - all.n;   // count before the first step
    // (no unmasked step: the incoming gradients pass through)
    dprev_mean[(size_t)b * G + g] = all.n > 0.f ? n0 * U : (dmean ? dmean[(size_t)b * G + g] : 0.f);
    dprev_var[(size_t)b * G + g] = all.n > 0.f ? n0 * V : (dvar ? dvar[(size_t)b * G + g] : 0.f);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) group_bwd_apply_kernel(const T* dy, const T* x, T* dx, long long gsb, long long gsl,
                                                              long long xsb, long long xsl, long long dsb, long long dsl,
                                                              int L, int D, int G, long long rows, const float* cumrstd,
                                                              const float* group_mean, const float* dux, const float* dvx,
                                                              const float* gamma, const unsigned char* mask) {
  constexpr int kN = Vec<T>::kN;
  const int nv = D / kN, width = D / G / kN;
  const float cg = (float)G / (float)D;
  const long long total = rows * nv;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < total; i += (long long)gridDim.x * 256) {
    const long long r = i / nv;
    const int v = (int)(i - r * nv);
    const long long b = r / L, t = r - b * L;
    float fx[kN], fy[kN], o[kN];
    Vec<T>::load(x + b * xsb + t * xsl + (long long)v * kN, fx);
    Vec<T>::load(dy + b * gsb + t * gsl + (long long)v * kN, fy);
    const long long gi = r * G + v / width;
    const float rs = __ldg(cumrstd + gi), ux = __ldg(group_mean + gi);
    const float du = __ldg(dux + gi) * cg, dv = 2.f * __ldg(dvx + gi) * cg;
    const bool mk = mask && mask[r];
#pragma unroll
    for (int k = 0; k < kN; ++k)
      o[k] = mk ? 0.f : fmaf(fy[k] * rs, __ldg(gamma + v * kN + k), fmaf(dv, fx[k] - ux, du));
    Vec<T>::store(dx + b * dsb + t * dsl + (long long)v * kN, o);
  }
}

// group sizes: a power of two of whole vectors, at most 32 of them; rows of whole vectors, 16-byte aligned
static bool group_ok(int dtype, int D, int G) {
  const int n = 16 / elem_size(dtype);
  if (G <= 0 || D % G != 0) return false;
  const int gs = D / G;
  return gs % n == 0 && gs / n <= 32 && (gs & (gs - 1)) == 0;
}
static bool vec_ok(int dtype, const void* p, long long sb, long long sl, long long sd) {
  const long long es = elem_size(dtype);
  return sd == 1 && aligned_to(p, 16) && (sb * es) % 16 == 0 && (sl * es) % 16 == 0;
}
static unsigned apply_grid(long long vecs) {
  const long long want = (vecs + 255) / 256;
  return (unsigned)(want > 148 * 16 ? 148 * 16 : want);
}

}  // namespace

bool group_norm_try(int dtype, const void* x, void* y, long long xsb, long long xsl, long long xsd, long long ysb,
                    long long ysl, long long ysd, const GroupNormArgs& a, cudaStream_t s) {
  if (g_options[OPT_DISABLE_STREAM].load() != 0) return false;
  if (!group_ok(dtype, a.D, a.G) || !vec_ok(dtype, x, xsb, xsl, xsd) || !vec_ok(dtype, y, ysb, ysl, ysd) || a.B > 65535)
    return false;
  const long long rows = (long long)a.B * a.L;
  const size_t n = (size_t)rows * a.G;
  const bool save = a.cummean != nullptr;
  Scratch sc(Scratch::padded(n * sizeof(float)) * (save ? 1 : 4), s);
  if (!sc) return false;
  float* gv = sc.take<float>(n);
  float* gm = save ? a.group_mean : sc.take<float>(n);
  float* cm = save ? a.cummean : sc.take<float>(n);
  float* cr = save ? a.cumrstd : sc.take<float>(n);
  const unsigned grid_m = (unsigned)((rows + kRowsPerBlock - 1) / kRowsPerBlock);
  const bool pairs = by_pairs(a.B, a.G);
  const dim3 grid_s(pairs ? (a.G + 1) / 2 : (a.G + 7) / 8, a.B);
  switch (dtype) {
#define MEGA_GROUP_CASE(DT, TY)                                                                                       \
  case DT:                                                                                                            \
    launch(group_moments_kernel<TY>, grid_m, 256, 0, (void*)s, (const TY*)x, xsb, xsl, a.L, a.D, a.G, rows, gm, gv);   \
    launch(pairs ? group_scan_kernel<2, 256> : group_scan_kernel<8, 128>, grid_s, pairs ? 512 : 1024, 0, (void*)s, gm, gv, a.L, a.G, a.prev_count, a.prev_mean,       \
           a.prev_var, a.mask, a.eps, cm, cr, a.count_out, a.mean_out, a.var_out);                                     \
    launch(group_apply_kernel<TY>, apply_grid(rows * (a.D / Vec<TY>::kN)), 256, 0, (void*)s, (const TY*)x, (TY*)y, xsb, \
           xsl, ysb, ysl, a.L, a.D, a.G, rows, cm, cr, a.gamma, a.beta, a.mask);                                       \
    return true;
    MEGA_GROUP_CASE(MEGA_F32, float)
    MEGA_GROUP_CASE(MEGA_BF16, __nv_bfloat16)
    MEGA_GROUP_CASE(MEGA_F16, __half)
#undef MEGA_GROUP_CASE
    default: return false;
  }
}

bool group_norm_bwd_try(int dtype, const void* dy, const void* x, void* dx, long long gsb, long long gsl, long long gsd,
                        long long xsb, long long xsl, long long xsd, long long dsb, long long dsl, long long dsd,
                        const GroupNormBwdArgs& a, cudaStream_t s) {
  if (g_options[OPT_DISABLE_STREAM].load() != 0) return false;
  if (!group_ok(dtype, a.D, a.G) || !vec_ok(dtype, x, xsb, xsl, xsd) || !vec_ok(dtype, dy, gsb, gsl, gsd) ||
      !vec_ok(dtype, dx, dsb, dsl, dsd) || a.B > 65535)
    return false;
  const long long rows = (long long)a.B * a.L;
  const size_t n = (size_t)rows * a.G;
  Scratch sc(Scratch::padded(n * sizeof(float)) * 4, s);
  if (!sc) return false;
  float *ds = sc.take<float>(n), *db = sc.take<float>(n), *dux = sc.take<float>(n), *dvx = sc.take<float>(n);
  const bool pairs = by_pairs(a.B, a.G);
  const dim3 grid_s(pairs ? (a.G + 1) / 2 : (a.G + 7) / 8, a.B);
  switch (dtype) {
#define MEGA_GROUP_CASE(DT, TY)                                                                                        \
  case DT: {                                                                                                           \
    const dim3 grid_m((unsigned)((rows + 4 * kRowsPerBlock - 1) / (4 * kRowsPerBlock)),                                \
                      (unsigned)((a.D / Vec<TY>::kN + 31) / 32));                                                      \
    launch(group_bwd_sums_kernel<TY>, grid_m, 256, 0, (void*)s, (const TY*)dy, (const TY*)x, gsb, gsl, xsb, xsl, a.L,  \
           a.D, a.G, rows, a.cummean, a.cumrstd, a.gamma, a.mask, ds, db, a.dgamma, a.dbeta);                          \
    launch(pairs ? group_bwd_scan_kernel<2, 256> : group_bwd_scan_kernel<8, 128>, grid_s, pairs ? 512 : 1024, 0, (void*)s, ds, db, a.L, a.G, a.cummean, a.cumrstd,        \
           a.group_mean, a.prev_mean, a.count, a.dmean, a.dvar, a.mask, dux, dvx, a.dprev_mean, a.dprev_var);          \
    launch(group_bwd_apply_kernel<TY>, apply_grid(rows * (a.D / Vec<TY>::kN)), 256, 0, (void*)s, (const TY*)dy,        \
           (const TY*)x, (TY*)dx, gsb, gsl, xsb, xsl, dsb, dsl, a.L, a.D, a.G, rows, a.cumrstd, a.group_mean, dux, dvx, \
           a.gamma, a.mask);                                                                                           \
    return true;                                                                                                       \
  }
    MEGA_GROUP_CASE(MEGA_F32, float)
    MEGA_GROUP_CASE(MEGA_BF16, __nv_bfloat16)
    MEGA_GROUP_CASE(MEGA_F16, __half)
#undef MEGA_GROUP_CASE
    default: return false;
  }
}

}  // namespace mega
