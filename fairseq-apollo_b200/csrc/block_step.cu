// One decoding step of the causal Mega block: TimestepNorm -> EMA -> SiLU on the running state, the projections,
// one query against the cached keys and values of its chunk, the output projection and the gates.
//
// A step of a few sequences reads every weight once (17 MB at embed 1024, hidden 2048: they stay in L2) and the
// cache once, and computes next to nothing: what it costs is launches, host calls and latency.  Five launches:
//   (1) the single-token step of TimestepNorm -> EMA (fused.cu, cema.cu), which writes mx and the normalised xn;
//   (2) v_proj(xn) and mx_proj(mx) in one launch: 16 output rows per block, the reduction split over its
//       warps; SiLU(v) goes straight into its row of the value cache;
//   (3) query and key from z (normalised, affine, rotary), the key into the cache, 32 scores per block;
//   (4) softmax and the weighted sum of the values, 64 columns per block, times SiLU(r);
//   (5) h_proj and the output gate.
// The products run on mma.sync with the weights as the 16 rows and the sequences as the 8 columns: a lane's
// 16-byte load of a weight row is the A operand of two MMAs once the reduction index is permuted alike on both
// sides, so weights go from memory to the tensor cores through registers alone; with at most 64 columns the
// tensor pipe is idle anyway and a TMEM accumulator would only add its round trip.  Launches 2 to 5 are
// programmatic dependents: their blocks start, and (2) and (5) fetch their weights, while the launch before ends.
// B = 4, embed 1024, hidden 2048, 700 cached keys: 510 us per token through the block's torch operations.
#include "common.cuh"
#include "block_step.cuh"

namespace mega {

namespace {

template <typename T>
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1);
template <>
__device__ __forceinline__ void mma_16816<__nv_bfloat16>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                         uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma_16816<__half>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                  uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

struct BlockStep {
  int B, D, S, E;
  const void *x, *xn, *mx;
  void* out;
  const void *vw, *vb, *mw, *mb, *hw;
  const void *qg, *qb;
  const float* rot;
  int qk16;         // the query / key affine in the activations' type (else fp32)
  float qk_eps;
  void *keys, *krot, *values;
  long long cap;
  int pos;          // keys cached before this step
  void *base, *gated;
  float* scores;    // [B][cap]
};

constexpr int kAhead = 4;   // blocks of 32 reduction indices whose weights are in flight per warp

// 16 rows of W (row-major, K columns) against kNB x 8 activation rows, K split over kW warps; on return thread t < 16 x B
// holds in `v` the product of row t % 16 and sequence t / 16, further ones a grid of the block's threads apart.
template <typename T, int kNB, int kW, typename F>
__device__ __forceinline__ void rows_times(const T* w, const T* act, int B, int K, unsigned char* smem, F&& finish) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
  const int pitch = K + 64 / (int)sizeof(T);   // (the eight rows of a quarter warp on distinct banks)
  T* as = reinterpret_cast<T*>(smem);
  const int nblk = K / 32;
  const T *w0 = w + (size_t)g * K + 8 * q, *w1 = w0 + (size_t)8 * K;
  uint4 wa[kAhead], wb[kAhead];
  auto fetch = [&](int i) {
    const int kb = warp + i * kW;
    if (kb < nblk) {
      wa[i % kAhead] = __ldg(reinterpret_cast<const uint4*>(w0 + kb * 32));
      wb[i % kAhead] = __ldg(reinterpret_cast<const uint4*>(w1 + kb * 32));
    }
  };
#pragma unroll
  for (int i = 0; i < kAhead; ++i) fetch(i);
  pdl_wait();   // the activations are the launch before's
  pdl_next();   // (after the wait: so the next launch may read, before its own, whatever earlier steps left in the caches)
  for (int i = threadIdx.x; i < B * (K / 8); i += kW * 32) {
    const int b = i / (K / 8), c = (i - b * (K / 8)) * 8;
    *reinterpret_cast<uint4*>(as + (size_t)b * pitch + c) = __ldg(reinterpret_cast<const uint4*>(act + (size_t)b * K + c));
  }
  __syncthreads();
  float acc[kNB][4];
#pragma unroll
  for (int n = 0; n < kNB; ++n)
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[n][k] = 0.f;
  const int iters = (nblk - warp + kW - 1) / kW;
  for (int i0 = 0; i0 < iters; i0 += kAhead) {
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int i = i0 + u;
      if (i < iters) {
        const uint4 a = wa[u], c = wb[u];
        const int kb = warp + i * kW;
#pragma unroll
        for (int n = 0; n < kNB; ++n) {
          uint4 b = make_uint4(0u, 0u, 0u, 0u);
          if (8 * n + g < B) b = *reinterpret_cast<const uint4*>(as + (size_t)(8 * n + g) * pitch + kb * 32 + 8 * q);
          mma_16816<T>(acc[n], a.x, c.x, a.y, c.y, b.x, b.y);
          mma_16816<T>(acc[n], a.z, c.z, a.w, c.w, b.z, b.w);
        }
        const int nx = i + kAhead;
        if (nx < iters) {
          wa[u] = __ldg(reinterpret_cast<const uint4*>(w0 + (warp + nx * kW) * 32));
          wb[u] = __ldg(reinterpret_cast<const uint4*>(w1 + (warp + nx * kW) * 32));
        }
      }
    }
  }
  // sums over the warps: [kW][8 kNB sequences][16 rows + 1]
  __syncthreads();
  float* red = reinterpret_cast<float*>(smem);
#pragma unroll
  for (int n = 0; n < kNB; ++n) {
    float* r = red + (size_t)warp * kNB * 8 * 17 + (size_t)(8 * n + 2 * q) * 17;
    r[g] = acc[n][0];
    r[17 + g] = acc[n][1];
    r[g + 8] = acc[n][2];
    r[17 + g + 8] = acc[n][3];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 16 * B; i += kW * 32) {
    const int row = i & 15, b = i >> 4;
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < kW; ++k) v += red[(size_t)k * kNB * 8 * 17 + b * 17 + row];
    finish(row, b, v);
  }
}

template <typename T>
__device__ __forceinline__ float round_to(float v) {
  T t;
  Elem<T>::st(&t, v);
  return Elem<T>::ld_shared(&t);
}

// (2) rows 0 .. E - 1: v_proj; then the rows of mx_proj.
template <typename T, int kNB>
__global__ void __launch_bounds__(256) block_proj_kernel(BlockStep a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int r0 = blockIdx.x * 16;
  const bool isv = r0 < a.E;
  const int F = 2 * a.D + a.S + a.E;
  const T* w = isv ? reinterpret_cast<const T*>(a.vw) + (size_t)r0 * a.D : reinterpret_cast<const T*>(a.mw) + (size_t)(r0 - a.E) * a.D;
  const T* bias = isv ? reinterpret_cast<const T*>(a.vb) + r0 : reinterpret_cast<const T*>(a.mb) + (r0 - a.E);
  rows_times<T, kNB, 8>(w, reinterpret_cast<const T*>(isv ? a.xn : a.mx), a.B, a.D, smem, [&](int row, int b, float v) {
    v = round_to<T>(v + Elem<T>::ld(bias + row));
    if (isv) Elem<T>::st(reinterpret_cast<T*>(a.values) + ((size_t)b * a.cap + a.pos) * a.E + r0 + row, siluf_(v));
    else Elem<T>::st(reinterpret_cast<T*>(a.base) + (size_t)b * F + (r0 - a.E) + row, v);
  });
}

constexpr int kKeys = 32;   // keys per block of the score kernel

// (3)
template <typename T>
__global__ void __launch_bounds__(256) block_score_kernel(BlockStep a) {
  __shared__ float qs[512];
  __shared__ float red[8];
  const int b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // the keys of earlier steps are read ahead of the wait
  const int k0 = blockIdx.x * kKeys;
  const int lanes = a.S / 8;           // lanes of a key (8, 16 or 32)
  const int per = 32 / lanes;          // keys of a warp at once
  const int sub = lane % lanes, first = k0 + warp * per + lane / lanes;
  const T* key = reinterpret_cast<const T*>(a.krot) + (size_t)b * a.cap * a.S + 8 * sub;
  uint4 early[kKeys / 8];
#pragma unroll
  for (int i = 0; i < kKeys / 8; ++i) {
    const int k = first + i * 8 * per;
    early[i] = make_uint4(0u, 0u, 0u, 0u);
    if (i * per < kKeys / 8 && k < a.pos) early[i] = __ldcg(reinterpret_cast<const uint4*>(key + (size_t)k * a.S));
  }
  pdl_wait();
  pdl_next();
  const int S = a.S, F = 2 * a.D + S + a.E, n = a.pos + 1;
  const T* z = reinterpret_cast<const T*>(a.base) + (size_t)b * F + a.D;
  float ss = 0.f;
  for (int c = tid; c < S; c += 256) {
    const float v = Elem<T>::ld_shared(z + c);
    ss = fmaf(v, v, ss);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if (lane == 0) red[warp] = ss;
  __syncthreads();
  ss = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) ss += red[k];
  const float inv = 1.f / fmaxf(sqrtf(ss), a.qk_eps);
  const bool owner = k0 <= a.pos && a.pos < k0 + kKeys;   // this block's keys include the new one
  const float2* rot = reinterpret_cast<const float2*>(a.rot) + (size_t)a.pos * (S / 2);
  for (int j = tid; j < S / 2; j += 256) {
    const int c = 2 * j;
    const float u = Elem<T>::ld_shared(z + c) * inv, v = Elem<T>::ld_shared(z + c + 1) * inv;
    const float2 w = __ldg(rot + j);
    auto affine = [&](float z, int i) {
      const float g = a.qk16 ? Elem<T>::ld(reinterpret_cast<const T*>(a.qg) + i) : __ldg(reinterpret_cast<const float*>(a.qg) + i);
      const float b = a.qk16 ? Elem<T>::ld(reinterpret_cast<const T*>(a.qb) + i) : __ldg(reinterpret_cast<const float*>(a.qb) + i);
      return fmaf(z, g + 1.f, b);
    };
    const float qa = affine(u, c), qb = affine(v, c + 1);
    qs[c] = qa * w.x - qb * w.y;
    qs[c + 1] = qa * w.y + qb * w.x;
    if (owner) {
      const float ka = round_to<T>(affine(u, S + c)), kb = round_to<T>(affine(v, S + c + 1));
      const size_t at = ((size_t)b * a.cap + a.pos) * S + c;
      Elem<T>::st(reinterpret_cast<T*>(a.keys) + at, ka);
      Elem<T>::st(reinterpret_cast<T*>(a.keys) + at + 1, kb);
      Elem<T>::st(reinterpret_cast<T*>(a.krot) + at, ka * w.x - kb * w.y);
      Elem<T>::st(reinterpret_cast<T*>(a.krot) + at + 1, ka * w.y + kb * w.x);
    }
  }
  __syncthreads();   // (also orders the new key's row before its read below)
#pragma unroll
  for (int i = 0; i < kKeys / 8; ++i) {
    const int k = first + i * 8 * per;
    if (i * per >= kKeys / 8) break;
    float s = 0.f;
    if (k < n) {
      const uint4 v = k < a.pos ? early[i] : *reinterpret_cast<const uint4*>(key + (size_t)k * S);
      const T* e = reinterpret_cast<const T*>(&v);
#pragma unroll
      for (int j = 0; j < 8; ++j) s = fmaf(Elem<T>::ld_shared(e + j), qs[8 * sub + j], s);
    }
    for (int o = lanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (sub == 0 && k < n) a.scores[(size_t)b * a.cap + k] = s;
  }
}

// (4) 64 columns of the values per block: 8 lanes of 16 bytes across, 32 keys at once
template <typename T>
__global__ void __launch_bounds__(256) block_attend_kernel(BlockStep a) {
  extern __shared__ __align__(16) unsigned char smem[];
  float* w = reinterpret_cast<float*>(smem);   // [n] weights, then [8][64] partial sums
  __shared__ float red[8];
  pdl_next();
  const int b = blockIdx.y, c0 = blockIdx.x * 64, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = a.pos + 1;
  const int cv = tid & 7, kr = tid >> 3;
  const int col = c0 + 8 * cv;
  const T* val = reinterpret_cast<const T*>(a.values) + (size_t)b * a.cap * a.E + col;
  constexpr int kDeep = 8;
  uint4 r[kDeep];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int u = 0; u < kDeep; ++u) {
      const int k = k0 + 32 * u;
      r[u] = k < n && col < a.E ? __ldcg(reinterpret_cast<const uint4*>(val + (size_t)k * a.E)) : make_uint4(0u, 0u, 0u, 0u);
    }
  };
  fetch(kr);   // (the values are complete: the launch before this one waited for those that write them)
  pdl_wait();
  const float* sc = a.scores + (size_t)b * a.cap;
  float m = -INFINITY;
  for (int k = tid; k < n; k += 256) {
    const float v = __ldcg(sc + k);
    w[k] = v;
    m = fmaxf(m, v);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) red[warp] = m;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 8; ++k) m = fmaxf(m, red[k]);
  __syncthreads();
  float sum = 0.f;
  for (int k = tid; k < n; k += 256) {
    const float e = m == -INFINITY ? 0.f : __expf(w[k] - m);
    w[k] = e;
    sum += e;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) red[warp] = sum;
  __syncthreads();
  sum = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) sum += red[k];
  const float inv = sum > 0.f ? 1.f / sum : 0.f;
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;
  for (int k0 = kr; k0 < n; k0 += 32 * kDeep) {
    if (k0 != kr) fetch(k0);
#pragma unroll
    for (int u = 0; u < kDeep; ++u) {
      const int k = k0 + 32 * u;
      const float wk = k < n ? w[k] : 0.f;
      const T* e = reinterpret_cast<const T*>(&r[u]);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] = fmaf(wk, Elem<T>::ld_shared(e + i), acc[i]);
    }
  }
  // a warp holds four keys' partial sums of the 64 columns
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 8);
    acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 16);
  }
  __syncthreads();
  if (lane < 8) {
#pragma unroll
    for (int i = 0; i < 8; ++i) w[warp * 64 + 8 * lane + i] = acc[i];
  }
  __syncthreads();
  if (tid < 64 && c0 + tid < a.E) {
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) v += w[k * 64 + tid];
    v = round_to<T>(v * inv);
    const int F = 2 * a.D + a.S + a.E;
    const float r = Elem<T>::ld_shared(reinterpret_cast<const T*>(a.base) + (size_t)b * F + a.D + a.S + c0 + tid);
    Elem<T>::st(reinterpret_cast<T*>(a.gated) + (size_t)b * a.E + c0 + tid, v * siluf_(r));
  }
}

// (5)
template <typename T, int kNB>
__global__ void __launch_bounds__(512) block_out_kernel(BlockStep a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int r0 = blockIdx.x * 16;
  const int F = 2 * a.D + a.S + a.E;
  rows_times<T, kNB, 16>(reinterpret_cast<const T*>(a.hw) + (size_t)r0 * a.E, reinterpret_cast<const T*>(a.gated), a.B, a.E, smem,
                         [&](int row, int b, float v) {
                           const int d = r0 + row;
                           const T* base = reinterpret_cast<const T*>(a.base) + (size_t)b * F;
                           const float u = sigmoidf_(Elem<T>::ld_shared(base + d));
                           const float h = siluf_(Elem<T>::ld_shared(base + a.D + a.S + a.E + d) + round_to<T>(v));
                           const float x = Elem<T>::ld(reinterpret_cast<const T*>(a.x) + (size_t)b * a.D + d);
                           Elem<T>::st(reinterpret_cast<T*>(a.out) + (size_t)b * a.D + d, fmaf(u, h - x, x));
                         });
}

// Keys and values of a prompt into the step's buffers, the keys also rotated by their positions.
template <typename T>
__global__ void __launch_bounds__(256) block_fill_kernel(const T* k, long long ksb, long long ksl, const T* v, long long vsb,
                                                         long long vsl, const float* rot, int n, int S, int E, T* keys,
                                                         T* krot, T* values, long long cap) {
  const int b = blockIdx.y, t = blockIdx.x;
  const T* kr = k + b * ksb + t * ksl;
  const T* vr = v + b * vsb + t * vsl;
  const size_t row = (size_t)b * cap + t;
  const float2* w = reinterpret_cast<const float2*>(rot) + (size_t)t * (S / 2);
  for (int j = threadIdx.x; j < S / 2; j += 256) {
    const float x = Elem<T>::ld(kr + 2 * j), y = Elem<T>::ld(kr + 2 * j + 1);
    const float2 c = __ldg(w + j);
    Elem<T>::st(keys + row * S + 2 * j, x);
    Elem<T>::st(keys + row * S + 2 * j + 1, y);
    Elem<T>::st(krot + row * S + 2 * j, x * c.x - y * c.y);
    Elem<T>::st(krot + row * S + 2 * j + 1, x * c.y + y * c.x);
  }
  for (int c = threadIdx.x; c < E; c += 256) values[row * E + c] = vr[c];
}

template <typename T, int kNB>
static void step_launches(const BlockStep& s, cudaStream_t st) {
  const size_t es = sizeof(T);
  auto smem = [&](int K, int warps) {
    const size_t act = (size_t)s.B * (K * es + 64), red = (size_t)warps * kNB * 8 * 17 * 4;
    return act > red ? act : red;
  };
  launch_after(block_proj_kernel<T, kNB>, dim3((2 * s.E + 2 * s.D + s.S) / 16), dim3(256), smem(s.D, 8), st, s);
  launch_after(block_score_kernel<T>, dim3((s.pos + 1 + kKeys - 1) / kKeys, s.B), dim3(256), 0, st, s);
  const size_t ws = (size_t)(s.pos + 1 > 512 ? s.pos + 1 : 512) * 4;
  launch_after(block_attend_kernel<T>, dim3((s.E + 63) / 64, s.B), dim3(256), ws, st, s);
  launch_after(block_out_kernel<T, kNB>, dim3(s.D / 16), dim3(512), smem(s.E, 16), st, s);
}

}  // namespace

}  // namespace mega

using namespace mega;

static size_t step_part(size_t bytes) { return (bytes + 255) & ~size_t(255); }

extern "C" int64_t mega_block_step_work(int dtype, int B, int D, int S, int E, int64_t cap) {
  if (dtype != MEGA_BF16 && dtype != MEGA_F16) return 0;
  const size_t es = 2;
  return (int64_t)(2 * step_part((size_t)B * D * es) + step_part((size_t)B * (2 * D + S + E) * es) + step_part((size_t)B * E * es) +
                   step_part((size_t)B * cap * 4));
}

extern "C" int mega_block_step(const mega_block_step_args* p, mega_stream_t stream) {
  if (!p || !p->x || !p->out || !p->count || !p->count_next || !p->mean || !p->var || !p->norm_gamma || !p->norm_beta ||
      !p->p || !p->q || !p->gamma_hat || !p->omega || !p->h || !p->v_weight || !p->v_bias || !p->mx_weight || !p->mx_bias ||
      !p->h_weight || !p->qk_gamma || !p->qk_beta || !p->rot || !p->keys || !p->keys_rot || !p->values || !p->work)
    return MEGA_ERR_NULL;
  if ((p->dtype != MEGA_BF16 && p->dtype != MEGA_F16) || (p->qk_dtype != MEGA_F32 && p->qk_dtype != p->dtype)) return MEGA_ERR_DTYPE;
  const int B = p->batch, D = p->embed, S = p->zdim, E = p->hdim;
  if (B <= 0 || D <= 0 || S <= 0 || E <= 0 || p->pos < 0 || p->pos >= p->cap || p->pos >= p->positions) return MEGA_ERR_SHAPE;
  // whole MMA tiles; a key is 8, 16 or 32 lanes of 16 bytes; the activations of a block fit its shared memory
  if (B > 64 || D % 32 != 0 || E % 32 != 0 || (S != 64 && S != 128 && S != 256) || p->pos >= 50000 ||
      (size_t)B * ((D > E ? D : E) * 2 + 64) > 200 * 1024)
    return MEGA_ERR_UNSUPPORTED;
  const void* al[] = {p->x, p->out, p->v_weight, p->mx_weight, p->h_weight, p->keys, p->keys_rot, p->values, p->work};
  for (const void* q : al)
    if (!aligned_to(q, 16)) return MEGA_ERR_ALIGN;
  cudaStream_t s = (cudaStream_t)stream;
  char* w = (char*)p->work;
  auto take = [&](size_t bytes) {
    char* r = w;
    w += step_part(bytes);
    return (void*)r;
  };
  BlockStep a{};
  a.B = B; a.D = D; a.S = S; a.E = E;
  void* mx = take((size_t)B * D * 2);
  void* xn = take((size_t)B * D * 2);
  a.base = take((size_t)B * (2 * D + S + E) * 2);
  a.gated = take((size_t)B * E * 2);
  a.scores = (float*)take((size_t)B * p->cap * 4);
  a.x = p->x; a.xn = xn; a.mx = mx; a.out = p->out;
  a.vw = p->v_weight; a.vb = p->v_bias; a.mw = p->mx_weight; a.mb = p->mx_bias; a.hw = p->h_weight;
  a.qg = p->qk_gamma; a.qb = p->qk_beta; a.qk16 = p->qk_dtype != MEGA_F32; a.rot = p->rot; a.qk_eps = (float)p->qk_eps;
  a.keys = p->keys; a.krot = p->keys_rot; a.values = p->values; a.cap = p->cap; a.pos = p->pos;
  const bool ok =
      p->complex_poles
          ? cema_step_lanes_try(p->dtype, p->x, mx, xn, B, D, p->ndim, (const long long*)p->count, p->mean, p->var,
                                p->norm_gamma, p->norm_beta, (float)p->norm_eps, p->p, p->q, p->gamma_hat, p->omega, p->h,
                                p->h, 1, stream, (long long*)p->count_next, true)
          : step_lanes_try(p->dtype, p->x, mx, xn, B, D, p->ndim, (const long long*)p->count, p->mean, p->var, p->norm_gamma,
                           p->norm_beta, (float)p->norm_eps, p->p, p->q, p->gamma_hat, p->omega, p->h, p->h, 1, stream,
                           (long long*)p->count_next, true);
  if (!ok) return MEGA_ERR_UNSUPPORTED;
#define MEGA_BLOCK_STEP(TY)                                \
  if (B <= 8) step_launches<TY, 1>(a, s);                  \
  else if (B <= 16) step_launches<TY, 2>(a, s);            \
  else if (B <= 32) step_launches<TY, 4>(a, s);            \
  else step_launches<TY, 8>(a, s)
  if (p->dtype == MEGA_BF16) { MEGA_BLOCK_STEP(__nv_bfloat16); }
  else { MEGA_BLOCK_STEP(__half); }
#undef MEGA_BLOCK_STEP
  return check_launch("block_step");
}

extern "C" int mega_block_cache_fill(const void* k, int64_t ksb, int64_t ksl, const void* v, int64_t vsb, int64_t vsl,
                                     const float* rot, int positions, int dtype, int B, int n, int S, int E, void* keys,
                                     void* keys_rot, void* values, int64_t cap, mega_stream_t stream) {
  if (!k || !v || !rot || !keys || !keys_rot || !values) return MEGA_ERR_NULL;
  if (dtype != MEGA_BF16 && dtype != MEGA_F16) return MEGA_ERR_DTYPE;
  if (B <= 0 || B > 65535 || n <= 0 || n > cap || n > positions || S <= 0 || (S & 1) || E <= 0) return MEGA_ERR_SHAPE;
  const dim3 grid(n, B);
  if (dtype == MEGA_BF16)
    launch(block_fill_kernel<__nv_bfloat16>, grid, 256, 0, stream, (const __nv_bfloat16*)k, (long long)ksb, (long long)ksl,
           (const __nv_bfloat16*)v, (long long)vsb, (long long)vsl, rot, n, S, E, (__nv_bfloat16*)keys,
           (__nv_bfloat16*)keys_rot, (__nv_bfloat16*)values, (long long)cap);
  else
    launch(block_fill_kernel<__half>, grid, 256, 0, stream, (const __half*)k, (long long)ksb, (long long)ksl, (const __half*)v,
           (long long)vsb, (long long)vsl, rot, n, S, E, (__half*)keys, (__half*)keys_rot, (__half*)values, (long long)cap);
  return check_launch("block_cache_fill");
}
