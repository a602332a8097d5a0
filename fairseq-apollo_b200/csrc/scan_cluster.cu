// The EMA layer in one launch: a cluster of blocks holds 32 channels of a whole sequence in shared memory.
//
// The three launches of scan_ema.cu read the sequence twice and exchange states through memory; at sizes that fit, a
// cluster does the same work with its own shared memory.  Block r of C takes the r-th part of the sequence, its eight
// warps adjacent segments of T steps, a lane one channel with its 16 poles in registers:
//   inputs in (all copies of a warp at once) -> [TimestepNorm: moments of every segment, combined over warps and, through
//   distributed shared memory, over blocks; the segment normalised in place] -> local pole states -> the states that enter
//   each segment, over warps and blocks as before -> outputs.
// Work per element and direction: 16 + 32 FMA real, two to three times that complex.  Bound: latency where the blocks do
// not fill the device, the FMA pipe beyond.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "norm_run.cuh"
#include "poles.cuh"
#include "scan_ema.cuh"
#include "scan_cluster.cuh"
#include "tma.cuh"
#include "walk.cuh"

namespace mega {

namespace {

constexpr int kW = 8;   // warps (segments) of a block

struct ClusterArgs {
  ScanArgs a;
  int T;   // steps of a segment
};

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// a float of another block's shared memory, at the address it has in ours
__device__ __forceinline__ float peer(const float* p, int rank) {
  uint32_t at;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_u32(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
  return v;
}

// Bytes of shared memory: tiles (rows of 32 channels; a normalised one in fp32), what the causal half leaves for the other,
// states [dirs][kW][parts * 16][32], their totals [dirs][parts * 16][32], moments [kW + 1][3][32], masks.
template <typename T, bool kC, bool kNorm, bool kBidir>
struct Layout {
  static constexpr int kRow = kNorm ? 128 : 32 * (int)sizeof(T);
  static constexpr int kParts = kC ? 2 : 1, kDirs = kBidir ? 2 : 1;
  static constexpr int kState = kParts * 16 * 32;   // floats of a state of 32 channels
  int part, st, tot, run, mask, total;
  __host__ __device__ explicit Layout(int T_) {
    part = kW * T_ * kRow;
    st = part + (kBidir ? kW * T_ * 128 : 0);
    tot = st + kDirs * kW * kState * 4;
    run = tot + kDirs * kState * 4;
    mask = run + (kNorm ? (kW + 1) * 3 * 32 * 4 : 0);
    total = mask + kW * ((T_ + 31) / 32) * 4;
  }
};

// calls f(r, pad) for the steps [0, n) of a segment, in order or reversed; mk: their padding bits
template <int kDir, bool kMask, typename F>
__device__ __forceinline__ void steps(int n, const unsigned* mk, F&& f) {
  int k = 0;
  for (; k + kU <= n; k += kU) {
    // (the bits of eight steps: in order they start at a multiple of eight, reversed anywhere)
    unsigned bits = 0u;
    if (kMask) {
      const int lo = kDir > 0 ? k : n - k - kU;
      const unsigned w0 = mk[lo >> 5], w1 = mk[min((lo >> 5) + 1, (n - 1) >> 5)];
      bits = __funnelshift_r(w0, w1, lo & 31);
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int r = kDir > 0 ? k + u : n - 1 - k - u;
      f(r, kMask && ((bits >> (kDir > 0 ? u : kU - 1 - u)) & 1u) != 0);
    }
  }
  for (; k < n; ++k) {
    const int r = kDir > 0 ? k : n - 1 - k;
    f(r, kMask && ((mk[r >> 5] >> (r & 31)) & 1u) != 0);
  }
}

template <bool kC>
__device__ __forceinline__ void put_state(const State<kC>& h, float* dst) {   // dst: [parts * 16][32], the lane's column
#pragma unroll
  for (int j = 0; j < kP2; ++j) {
    float lo, hi;
    unpack2(h.r[j], lo, hi);
    dst[(2 * j) * 32] = lo;
    dst[(2 * j + 1) * 32] = hi;
    if (kC) {
      unpack2(h.i[j], lo, hi);
      dst[(16 + 2 * j) * 32] = lo;
      dst[(16 + 2 * j + 1) * 32] = hi;
    }
  }
}
template <bool kC>
__device__ __forceinline__ void get_state(State<kC>& h, const float* src) {
#pragma unroll
  for (int j = 0; j < kP2; ++j) {
    h.r[j] = pack2(src[(2 * j) * 32], src[(2 * j + 1) * 32]);
    if (kC) h.i[j] = pack2(src[(16 + 2 * j) * 32], src[(16 + 2 * j + 1) * 32]);
  }
}

template <bool kC>
__device__ __forceinline__ float2 power(float2 q, int n) {
  return kC ? ipow(q, n) : make_float2(powf(q.x, (float)n), 0.f);
}
// w H + v
template <bool kC>
__device__ __forceinline__ float2 onward(float2 w, float2 H, float2 v) {
  if (!kC) return make_float2(fmaf(w.x, H.x, v.x), 0.f);
  const float2 p = cmul(w, H);
  return make_float2(p.x + v.x, p.y + v.y);
}

template <typename T, bool kC, bool kMask, bool kState, bool kNorm, bool kBidir>
__global__ void __launch_bounds__(kW * 32, kC ? 1 : 2) scan_cluster_kernel(ClusterArgs s) {
  static_assert(!kBidir || (!kState && !kNorm), "state and norm are causal");
  using Lay = Layout<T, kC, kNorm, kBidir>;
  using In = typename std::conditional<kNorm, float, T>::type;   // what the tile holds
  constexpr int kState_ = Lay::kState;
  extern __shared__ __align__(16) unsigned char smem[];
  const ScanArgs& a = s.a;
  const Lay o(s.T);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rank = (int)cluster_rank(), ranks = gridDim.y;   // (a cluster is one column of the grid)
  const int b = blockIdx.z, d0 = blockIdx.x * 32, left = a.D - d0;
  const bool ok = lane < left;
  const int d = d0 + lane, dc = ok ? d : a.D - 1;
  const int seg = rank * kW + warp;
  const int t0 = min(a.L, seg * s.T), n = min(a.L, t0 + s.T) - t0;
  unsigned char* tile = smem + (size_t)warp * s.T * Lay::kRow;
  float* st = reinterpret_cast<float*>(smem + o.st);
  float* tot = reinterpret_cast<float*>(smem + o.tot);
  unsigned* mk = reinterpret_cast<unsigned*>(smem + o.mask) + warp * ((s.T + 31) / 32);

  // ---- inputs
  {
    // (16-bit inputs of a norm go to the upper half of the tile: their rows are widened from the front)
    constexpr int kPer = 32 * (int)sizeof(T) / 16;   // 16-byte pieces of a row
    const T* x = reinterpret_cast<const T*>(a.x) + b * a.xsb + (long long)t0 * a.xsl + d0;
    const uint32_t at = smem_u32(tile) + (kNorm && sizeof(T) == 2 ? s.T * 64 : 0);
#pragma unroll 4
    for (int id = lane; id < n * kPer; id += 32) {
      const int r = id / kPer, c = (id % kPer) * (16 / (int)sizeof(T));
      const bool in = c < left;
      const int bytes = in ? min(16, (left - c) * (int)sizeof(T)) : 0;   // (nothing behind the last channel is read)
      asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;" ::"r"(at + id * 16),
                   "l"(in ? x + (long long)r * a.xsl + c : x), "r"(bytes)
                   : "memory");
    }
    tile_commit();
  }
  if (kMask) {
    const unsigned char* m = a.mask + (size_t)b * a.L + t0;
    for (int k = 0; k < n; k += 32) {
      const unsigned bits = __ballot_sync(0xffffffffu, k + lane < n && __ldg(m + k + lane) != 0);
      if (lane == 0) mk[k >> 5] = bits;
    }
  }
  Poles<kC> P;
  load_poles<kC>(P, a, dc);
  // (for the states that enter the segments, where a thread takes two poles of a channel; the inputs are still on their way)
  float2 full[Lay::kDirs][2], part[Lay::kDirs][2];   // q^T, q^(L mod T)
#pragma unroll
  for (int dir = 0; dir < Lay::kDirs; ++dir)
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int pole = warp + kW * k;
      const size_t c = (size_t)(dc + dir * a.D) * a.N + pole;
      float2 q = make_float2(0.f, 0.f);
      if (pole < a.N) q = kC ? make_float2(__ldg(a.q + 2 * c), __ldg(a.q + 2 * c + 1)) : make_float2(__ldg(a.q + c), 0.f);
      full[dir][k] = power<kC>(q, s.T);
      part[dir][k] = power<kC>(q, a.L % s.T);
    }
  tile_wait<0>();
  __syncwarp();

  // ---- TimestepNorm: moments, what the segment starts from, and the segment normalised
  Running rs;
  float w = 0.f, bb = 0.f;
  if constexpr (kNorm) {
    w = __ldg(a.gamma + dc);
    bb = __ldg(a.beta + dc);
    const T* raw = reinterpret_cast<const T*>(tile + (sizeof(T) == 2 ? s.T * 64 : 0)) + lane;
    float cnt = 0.f, sum = 0.f, sq = 0.f;
    steps<1, kMask>(n, mk, [&](int r, bool pad) {
      if (!pad) {
        sum += Elem<T>::ld_shared(raw + r * 32);
        cnt += 1.f;
      }
    });
    const float c = cnt > 0.f ? sum / cnt : 0.f;
    steps<1, kMask>(n, mk, [&](int r, bool pad) {
      const float e = pad ? 0.f : Elem<T>::ld_shared(raw + r * 32) - c;
      sq = fmaf(e, e, sq);
    });
    float* run = reinterpret_cast<float*>(smem + o.run);   // [kW + 1][3][32]: the segments', the block's
    run[(warp * 3) * 32 + lane] = cnt;
    run[(warp * 3 + 1) * 32 + lane] = c;
    run[(warp * 3 + 2) * 32 + lane] = sq;
    __syncthreads();
    const long long cnt0 = a.prev_count[b];
    const size_t i = (size_t)b * a.D + dc;
    Run r{0.f, 0.f, 0.f};
    if (ranks > 1) {
      if (warp == 0) {
#pragma unroll
        for (int k = 0; k < kW; ++k)
          r = combine(r, Run{run[(k * 3) * 32 + lane], run[(k * 3 + 1) * 32 + lane], run[(k * 3 + 2) * 32 + lane]});
        float* all = run + kW * 3 * 32 + lane;
        all[0] = r.n;
        all[32] = r.m;
        all[64] = r.s;
      }
      cluster_arrive();
      cluster_wait();
    }
    r = Run{(float)cnt0, __ldg(a.prev_mean + i), __ldg(a.prev_var + i) * (float)cnt0};
    const float* all = run + kW * 3 * 32 + lane;
    Run before[7];   // (at most eight blocks; all reads of the others at once)
#pragma unroll
    for (int k = 0; k < 7; ++k)
      if (k < rank) before[k] = Run{peer(all, k), peer(all + 32, k), peer(all + 64, k)};
#pragma unroll
    for (int k = 0; k < 7; ++k)
      if (k < rank) r = combine(r, before[k]);
    float seen = 0.f;   // unmasked steps of the call before the segment (a float count that starts beyond 2^24 would round them)
#pragma unroll
    for (int k = 0; k < 7; ++k)
      if (k < rank) seen += before[k].n;
    for (int k = 0; k < warp; ++k) {
      r = combine(r, Run{run[(k * 3) * 32 + lane], run[(k * 3 + 1) * 32 + lane], run[(k * 3 + 2) * 32 + lane]});
      seen += run[(k * 3) * 32 + lane];
    }
    r.n = (float)cnt0 + seen;
    rs.start(r);
    if (rank == ranks - 1 && warp == kW - 1 && ok) {
      r = combine(r, Run{cnt, c, sq});
      a.mean_out[i] = r.n > 0.f ? r.m : a.prev_mean[i];
      a.var_out[i] = r.n > 0.f ? r.s / r.n : a.prev_var[i];
      if (d == 0) a.count_out[b] = cnt0 + (long long)(seen + cnt);
    }
  }

  // ---- local states
  State<kC> h;
  h.zero();
  const In* in = reinterpret_cast<const In*>(tile) + lane;
  if constexpr (kNorm) {
    const T* raw = reinterpret_cast<const T*>(tile + (sizeof(T) == 2 ? s.T * 64 : 0)) + lane;
    float* out = reinterpret_cast<float*>(tile) + lane;
    T* xn = a.xn ? reinterpret_cast<T*>(a.xn) + b * a.ysb + (long long)t0 * a.ysl + dc : nullptr;
    for (int k = 0; k < n; k += kU) {
      float v[kU];
      const unsigned bits = kMask ? mk[k >> 5] >> (k & 31) : 0u;
#pragma unroll
      for (int u = 0; u < kU; ++u) v[u] = k + u < n ? Elem<T>::ld_shared(raw + (k + u) * 32) : 0.f;
      __syncwarp();   // (widened rows may cover those that other lanes have just read)
#pragma unroll
      for (int u = 0; u < kU; ++u)
        if (k + u < n) {
          v[u] = normed(rs, v[u], kMask && ((bits >> u) & 1u), w, bb, a.eps);
          out[(k + u) * 32] = v[u];
          advance<kC>(h, P, splat(v[u]));
          if (xn) {
            if (ok) Elem<T>::st(xn, v[u]);
            xn += a.ysl;
          }
        }
    }
  } else {
    steps<1, kMask>(n, mk, [&](int r, bool pad) { advance<kC>(h, P, splat(kMask && pad ? 0.f : Elem<In>::ld_shared(in + r * 32))); });
  }
  put_state<kC>(h, st + warp * kState_ + lane);
  if constexpr (kBidir) {
    load_poles<kC>(P, a, dc + a.D);
    h.zero();
    steps<-1, kMask>(n, mk, [&](int r, bool pad) { advance<kC>(h, P, splat(kMask && pad ? 0.f : Elem<In>::ld_shared(in + r * 32))); });
    put_state<kC>(h, st + (kW + warp) * kState_ + lane);
  }
  __syncthreads();

  // ---- the states that enter each segment
  auto length = [&](int g) { return min(a.L, g * s.T + s.T) - min(a.L, g * s.T); };   // of a segment
  auto value = [&](const float* v) { return make_float2(v[0], kC ? v[16 * 32] : 0.f); };
  if (ranks > 1) {
#pragma unroll
    for (int dir = 0; dir < Lay::kDirs; ++dir)
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int pole = warp + kW * k;
        const float* v = st + dir * kW * kState_ + pole * 32 + lane;
        float2 H = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < kW; ++i) {
          const int g = dir == 0 ? i : kW - 1 - i, len = length(rank * kW + g);
          if (len > 0) H = onward<kC>(len == s.T ? full[dir][k] : part[dir][k], H, value(v + g * kState_));
        }
        float* t = tot + dir * kState_ + pole * 32 + lane;
        t[0] = H.x;
        if (kC) t[16 * 32] = H.y;
      }
    cluster_arrive();
    cluster_wait();
  }
#pragma unroll
  for (int dir = 0; dir < Lay::kDirs; ++dir)
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int pole = warp + kW * k;
      const bool live = pole < a.N;
      const size_t at = ((size_t)b * a.D + dc) * a.N + pole;
      const float gain = kState && live ? __ldg(a.p + (size_t)dc * a.N + pole) : 1.f;
      float2 H = make_float2(0.f, 0.f);
      if (kState && a.h_in && live) H = kC ? make_float2(a.h_in[2 * at], a.h_in[2 * at + 1]) : make_float2(a.h_in[at], 0.f);
      const float* t = tot + dir * kState_ + pole * 32 + lane;
      if (ranks > 1) {
        static_assert(kW == 8, "three squarings");
        float2 whole = full[dir][k];   // q^(steps of a block)
#pragma unroll
        for (int i = 0; i < 3; ++i) whole = kC ? cmul(whole, whole) : make_float2(whole.x * whole.x, 0.f);
        const int before = dir == 0 ? rank : ranks - 1 - rank;
        float2 v[7];
#pragma unroll
        for (int i = 0; i < 7; ++i)
          if (i < before) {
            const int r = dir == 0 ? i : ranks - 1 - i;
            v[i] = make_float2(gain * peer(t, r), kC ? gain * peer(t + 16 * 32, r) : 0.f);
          }
#pragma unroll
        for (int i = 0; i < 7; ++i)
          // (blocks before one with steps are whole; against time, H is zero until the last of them)
          if (i < before) H = onward<kC>(whole, H, v[i]);
      }
      float* v = st + dir * kW * kState_ + pole * 32 + lane;
#pragma unroll
      for (int i = 0; i < kW; ++i) {
        const int g = dir == 0 ? i : kW - 1 - i, len = length(rank * kW + g);
        const float2 own = value(v + g * kState_);
        v[g * kState_] = H.x;
        if (kC) v[g * kState_ + 16 * 32] = H.y;
        if (len > 0) H = onward<kC>(len == s.T ? full[dir][k] : part[dir][k], H, make_float2(gain * own.x, gain * own.y));
      }
      if (kState && a.h_out && live && ok && rank == (a.L - 1) / (kW * s.T)) {   // (the block of the last step)
        a.h_out[kC ? 2 * at : at] = H.x;
        if (kC) a.h_out[2 * at + 1] = H.y;
      }
    }
  __syncthreads();
  if (ranks > 1) cluster_arrive();   // (a block stays until the others have read its totals: the wait is at the end)

  // ---- outputs
  const float om = __ldg(a.omega + dc);
  T* y = reinterpret_cast<T*>(a.y) + b * a.ysb + (long long)t0 * a.ysl + dc;
  if (kBidir) load_poles<kC>(P, a, dc);
  State<kC> c;
  load_weights<kC>(c, a, dc, !kState);
  f32x2 p[kState ? kP2 : 1];
  if (kState) {
#pragma unroll
    for (int j = 0; j < kP2; ++j) {
      const size_t i = (size_t)dc * a.N + 2 * j;
      p[kState ? j : 0] = pack2(2 * j < a.N ? __ldg(a.p + i) : 0.f, 2 * j + 1 < a.N ? __ldg(a.p + i + 1) : 0.f);
    }
  }
  get_state<kC>(h, st + warp * kState_ + lane);
  float* half = reinterpret_cast<float*>(smem + o.part) + (size_t)warp * s.T * 32 + lane;
  steps<1, kMask>(n, mk, [&](int r, bool pad) {
    const float xv = Elem<In>::ld_shared(in + r * 32);
    const f32x2 x2 = splat(kMask && !kNorm && pad ? 0.f : xv);
    if constexpr (kState) advance_gain<kC>(h, P, p, x2);
    else advance<kC>(h, P, x2);
    float v = fmaf(om, xv, dot<kC>(c, h));
    if constexpr (kBidir) {
      half[r * 32] = v;
    } else {
      if (a.silu) v = siluf_(v);
      if (ok) Elem<T>::st(y, v);
      y += a.ysl;
    }
  });
  if constexpr (kBidir) {
    load_poles<kC>(P, a, dc + a.D);
    load_weights<kC>(c, a, dc + a.D, true);
    get_state<kC>(h, st + (kW + warp) * kState_ + lane);
    const bool shift = a.shift != 0;
    y += (long long)(n - 1) * a.ysl;
    steps<-1, kMask>(n, mk, [&](int r, bool pad) {
      float v = half[r * 32];
      if (shift) v += dot<kC>(c, h);
      advance<kC>(h, P, splat(kMask && pad ? 0.f : Elem<In>::ld_shared(in + r * 32)));
      if (!shift) v += dot<kC>(c, h);
      if (a.silu) v = siluf_(v);
      if (ok) Elem<T>::st(y, v);
      y -= a.ysl;
    });
  }
  if (ranks > 1) cluster_wait();
}

template <typename T, bool kC, bool kMask, bool kState, bool kNorm, bool kBidir>
bool launch_cluster(const ClusterArgs& s, int ranks, cudaStream_t st) {
  auto kernel = scan_cluster_kernel<T, kC, kMask, kState, kNorm, kBidir>;
  const int smem = Layout<T, kC, kNorm, kBidir>(s.T).total;
  if (smem > 48 * 1024) allow_smem(reinterpret_cast<const void*>(kernel), smem);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((s.a.D + 31) / 32, ranks, s.a.B);
  cfg.blockDim = dim3(kW * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1;
  at[0].val.clusterDim.y = ranks;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, s);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  g_last_kernel.store("scan_cluster", std::memory_order_relaxed);
  return true;
}

template <typename T, bool kC>
bool launch_form(const ClusterArgs& s, int ranks, cudaStream_t st) {
  const ScanArgs& a = s.a;
  const bool state = a.h_in || a.h_out, norm = a.prev_count != nullptr;
#define MEGA_FORM(ST, NO, BI) \
  (a.mask ? launch_cluster<T, kC, true, ST, NO, BI>(s, ranks, st) : launch_cluster<T, kC, false, ST, NO, BI>(s, ranks, st))
  if constexpr (!kC)
    if (a.bidir) return MEGA_FORM(false, false, true);
  if (norm) return state ? MEGA_FORM(true, true, false) : MEGA_FORM(false, true, false);
  return state ? MEGA_FORM(true, false, false) : MEGA_FORM(false, false, false);
#undef MEGA_FORM
}

}  // namespace

namespace {

// Steps of a segment and blocks of a cluster: the smallest product of rounds and steps (60 steps' worth of time pass
// beside them: copies in, exchange of states).  False when the sequence does not fit, is one of complex poles walked both
// ways (its exchange costs more than the launches it saves), or statistics or states are updated in place.
bool plan(int dtype, const ScanArgs& a, int& T, int& ranks, double& rounds, double& best) {
  if ((a.cplx && a.bidir) || a.B > 65535 || a.N > 16) return false;
  const bool norm = a.prev_count != nullptr;
  // (all blocks of a cluster read the incoming statistics and states, the last one writes the new ones)
  const size_t stats = (size_t)a.B * a.D, states = stats * a.N * (a.cplx ? 2 : 1);
  if (overlap(a.h_in, a.h_out, states)) return false;
  if (norm)
    for (const float* out : {a.mean_out, a.var_out})
      if (overlap(out, a.prev_mean, stats) || overlap(out, a.prev_var, stats)) return false;
  const int dirs = a.bidir ? 2 : 1;
  const int row = (norm ? 128 : 32 * elem_size(dtype)) + (a.bidir ? 128 : 0);
  const double strips = (double)((a.D + 31) / 32) * a.B;
  best = 1e30;
  for (int c = 1; c <= 8; c *= 2) {
    const int t = std::max(16, ((a.L + c * kW - 1) / (c * kW) + kU - 1) / kU * kU);
    const int smem = kW * t * row + dirs * (kW + 1) * (a.cplx ? 2 : 1) * 2048 + (kW + 1) * 384 + kW * (t / 32 + 1) * 4;
    if (smem > 200 * 1024) continue;
    const int per_sm = std::max(1, std::min(227 * 1024 / (smem + 1024), a.cplx ? 1 : 2));
    // (a cluster stays within a group of 16 to 18 SMs: larger ones leave some of them over)
    const double n = std::ceil(strips * c / ((c == 8 ? 112.0 : c == 4 ? 132.0 : 148.0) * per_sm));
    const double cost = n * (t + 60.0) * (strips * c > 148 ? std::min<double>(per_sm, strips * c / 148.0) : 1.0);
    if (cost < best) {
      best = cost;
      T = t;
      ranks = c;
      rounds = n;
    }
    if (t == 16) break;
  }
  return best < 1e30;
}

}  // namespace

// From a grid of shapes on one B200: a fixed part, then the longer of what a segment's steps take and what all elements
// take.  Beyond 8.5 million elements (6.5 of complex poles in more than one round, 4.3 walked both ways: where that grid had
// the two level), or in rounds of long segments, the three launches of scan_ema.cu are as fast.
double scan_cluster_us(int dtype, const ScanArgs& a) {
  int T = 0, ranks = 1;
  double rounds = 0, steps = 0;
  const double n = (double)a.B * a.L * a.D;
  if (!plan(dtype, a, T, ranks, rounds, steps)) return 1e30;
  if (n > (a.cplx && rounds > 1 ? 6.5e6 : a.bidir ? 4.3e6 : 8.5e6) || (rounds > 1 && T > 64)) return 1e30;
  const bool norm = a.prev_count != nullptr;
  const double fixed = a.cplx ? 14.0 : a.bidir ? 12.0 : norm ? 8.0 : 6.0;
  const double step = a.cplx ? (norm ? 0.4 : 0.3) : a.bidir ? 0.4 : norm ? 0.22 : 0.14;
  const double rate = a.cplx ? (norm ? 85e3 : 115e3) : a.bidir ? 100e3 : norm ? 165e3 : 195e3;
  return std::max(fixed + std::max(T * step, n / rate), (a.cplx ? 0.27 : 0.08) * steps);   // (many short rounds: the latter)
}

// The chain costs 24 ns per position pipelined along the sequence, 44 with a mask, and 28 complex beside 54 us of its own
// (filling the pipeline of its tiles), until all elements cost more (1.3 and 0.6 per ns); a tenth in hand for the model.
bool scan_cluster_first(int dtype, const ScanArgs& a, long long xsd, long long ysd) {
  if (dtype != MEGA_BF16 || a.bidir || g_options[OPT_SPLIT].load() == 1 || g_options[OPT_DISABLE_MMA].load() != 0 ||
      g_options[OPT_MMA_TILE].load() != 0 || !scan_ema_fwd_ok(dtype, a, xsd, ysd))
    return false;
  if (a.h_out && !a.mask && !a.cplx && a.L % 32 != 0) return false;   // (that kernel's head, then a tail of under 32 steps)
  const double n = (double)a.B * a.L * a.D;
  const double chain = a.cplx ? 54.0 + a.L * 28e-3 : a.L * (a.mask ? 44e-3 : 24e-3), all = n / (a.cplx ? 600e3 : 1300e3);
  return scan_cluster_us(dtype, a) < 0.9 * (6.0 + std::max(chain, all));
}

bool scan_cluster_try(int dtype, const ScanArgs& a, cudaStream_t st) {
  ClusterArgs s{a, 0};
  int ranks = 1;
  double rounds, steps;
  if (scan_cluster_us(dtype, a) > 1e29 || !plan(dtype, a, s.T, ranks, rounds, steps)) return false;
  switch (dtype) {
    case MEGA_F32: return a.cplx ? launch_form<float, true>(s, ranks, st) : launch_form<float, false>(s, ranks, st);
    case MEGA_BF16: return a.cplx ? launch_form<__nv_bfloat16, true>(s, ranks, st) : launch_form<__nv_bfloat16, false>(s, ranks, st);
    case MEGA_F16: return a.cplx ? launch_form<__half, true>(s, ranks, st) : launch_form<__half, false>(s, ranks, st);
    default: return false;
  }
}

}  // namespace mega
