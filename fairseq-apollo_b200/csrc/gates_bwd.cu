// Training kernels of the Mega block around its projections and attention products: the gates' backward, the query /
// key affine's backward and the softmax with the learned relative bias (moving_average_gated_attention.py:308,
// 322-330, 407-412, 223-280).
//
// Elementwise kernels: a thread owns one 16-byte vector of columns and walks rows, so the column sums (the bias
// gradients of the projections that produced the operands) stay in its registers and cost one block reduction and
// one atomic add per column and block.  Operands may be column slices of a wider matrix (row pitches), which is how
// the four gradients of the mx_proj output land in one matrix without copies.
// Bound: HBM, each operand once (16384 rows, embed 1024, hidden 2048: the torch operations they replace, with their
// slice gradients zero-filled, copied and added, took 1.1 ms of a 3.5 ms training pass).
#include <type_traits>

#include "common.cuh"

namespace mega {

namespace {

template <typename T>
struct Row16 {
  static constexpr int kN = 16 / (int)sizeof(T);
  static __device__ __forceinline__ void load(const T* p, float (&f)[kN]) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
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

// d silu(v) / dv given s = sigmoid(v)  (1 - s is small only where the term it is in is small beside s)
__device__ __forceinline__ float dsilu(float v, float s) { return fmaf(v * s, 1.f - s, s); }

// column sums of a block (32 vectors of columns x 8 rows of threads) into `out`
template <typename T>
__device__ __forceinline__ void add_columns(const float (&s)[Row16<T>::kN], float* out, int cols, float (*red)[32 * Row16<T>::kN + 4]) {
  constexpr int kN = Row16<T>::kN;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kN; ++k) red[ty][tx * kN + k] = s[k];
  __syncthreads();
  for (int c = threadIdx.x; c < 32 * kN; c += 256) {
    float v = 0.f;
#pragma unroll
    for (int y = 0; y < 8; ++y) v += red[y][c];
    const int col = blockIdx.x * 32 * kN + c;
    if (col < cols) atomicAdd(out + col, v);
  }
}

struct GateBwd {
  const void *g, *a, *b, *c, *d;   // gradient of the result, operands
  void *o0, *o1, *o2;              // gradients of the operands
  long long ldg, lda, ldb, ldc, ldd, l0, l1, l2;
  float *s0, *s1;                  // column sums, or null
  long long rows;
  int cols, per;                   // rows of a block
};

// OP 0: y = silu(a): o0 = da.  OP 1: y = a silu(b): o0 = da, o1 = db.  OP 2: out = a + sigmoid(b) (silu(c + d) - a):
// o0 = da, o1 = db, o2 = dc = dd.  s0: column sums of o0 (OP 0) or o1; s1: of o2.
template <typename T, int OP>
__global__ void __launch_bounds__(256) gate_bwd_kernel(GateBwd p) {
  constexpr int kN = Row16<T>::kN;
  __shared__ float red[8][32 * kN + 4];
  const int col = (blockIdx.x * 32 + (threadIdx.x & 31)) * kN;
  const bool ok = col < p.cols;
  float s0[kN], s1[kN];
#pragma unroll
  for (int k = 0; k < kN; ++k) s0[k] = s1[k] = 0.f;
  const long long r1 = min(p.rows, (long long)(blockIdx.y + 1) * p.per);
  for (long long r = (long long)blockIdx.y * p.per + (threadIdx.x >> 5); ok && r < r1; r += 8) {
    float g[kN], a[kN], o0[kN], o1[kN];
    Row16<T>::load(reinterpret_cast<const T*>(p.g) + r * p.ldg + col, g);
    Row16<T>::load(reinterpret_cast<const T*>(p.a) + r * p.lda + col, a);
    if (OP == 0) {
#pragma unroll
      for (int k = 0; k < kN; ++k) {
        o0[k] = g[k] * dsilu(a[k], sigmoid_of<T>(a[k]));
        s0[k] += o0[k];
      }
    } else if (OP == 1) {
      float b[kN];
      Row16<T>::load(reinterpret_cast<const T*>(p.b) + r * p.ldb + col, b);
#pragma unroll
      for (int k = 0; k < kN; ++k) {
        const float s = sigmoid_of<T>(b[k]);
        o0[k] = g[k] * b[k] * s;
        o1[k] = g[k] * a[k] * dsilu(b[k], s);
        s0[k] += o1[k];
      }
      Row16<T>::store(reinterpret_cast<T*>(p.o1) + r * p.l1 + col, o1);
    } else {
      float b[kN], c[kN], d[kN], o2[kN];
      Row16<T>::load(reinterpret_cast<const T*>(p.b) + r * p.ldb + col, b);
      Row16<T>::load(reinterpret_cast<const T*>(p.c) + r * p.ldc + col, c);
      Row16<T>::load(reinterpret_cast<const T*>(p.d) + r * p.ldd + col, d);
#pragma unroll
      for (int k = 0; k < kN; ++k) {
        const float t = c[k] + d[k];
        const Gate u = gate_of<T>(b[k]);
        const float s = sigmoid_of<T>(t);
        o0[k] = g[k] * u.c;
        o1[k] = g[k] * fmaf(t, s, -a[k]) * u.s * u.c;
        o2[k] = g[k] * u.s * dsilu(t, s);
        s0[k] += o1[k];
        s1[k] += o2[k];
      }
      Row16<T>::store(reinterpret_cast<T*>(p.o1) + r * p.l1 + col, o1);
      Row16<T>::store(reinterpret_cast<T*>(p.o2) + r * p.l2 + col, o2);
    }
    Row16<T>::store(reinterpret_cast<T*>(p.o0) + r * p.l0 + col, o0);
  }
  if (p.s0) add_columns<T>(s0, p.s0, p.cols, red);
  if (OP == 2 && p.s1) add_columns<T>(s1, p.s1, p.cols, red);
}

// Query / key affine.  A warp takes rows, lane l owns the feature pairs l + 32 i of every row, so its shares of the
// (2, S) parameter sums and of the column sums stay in registers.
constexpr int kQkPairs = 8;   // at most 512 features

// two adjacent values (rows and pairs start at even elements of aligned arrays)
template <typename T>
__device__ __forceinline__ void load_pair(const T* p, float& a, float& b) {
  using P = typename std::conditional<sizeof(T) == 4, float2, uint32_t>::type;
  const P v = __ldg(reinterpret_cast<const P*>(p));
  a = Elem<T>::ld_shared(reinterpret_cast<const T*>(&v));
  b = Elem<T>::ld_shared(reinterpret_cast<const T*>(&v) + 1);
}
template <typename T>
__device__ __forceinline__ void store_pair(T* p, float a, float b) {
  using P = typename std::conditional<sizeof(T) == 4, float2, uint32_t>::type;
  P v;
  Elem<T>::st(reinterpret_cast<T*>(&v), a);
  Elem<T>::st(reinterpret_cast<T*>(&v) + 1, b);
  *reinterpret_cast<P*>(p) = v;
}

// kP: pairs of a lane (1, 2, 4 or 8): the sums of 64 features are 10 registers, those of 512 are 80 and leave few warps.
template <typename T, int kP>
__global__ void __launch_bounds__(256) gate_qk_bwd_kernel(const T* z, long long ldz, const float* gamma, const float* rot,
                                                          int period, int q_offset, const T* dq, long long ldq, const T* dk,
                                                          long long ldk, T* dz, long long ldd, float* dgamma, float* dbeta,
                                                          float* colsum, long long rows, int cols, float eps) {
  __shared__ float red[8][128];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = cols >> 1;
  float sg0[2 * kP], sg1[2 * kP], sb0[2 * kP], sb1[2 * kP], sz[2 * kP];
#pragma unroll
  for (int i = 0; i < 2 * kP; ++i) sg0[i] = sg1[i] = sb0[i] = sb1[i] = sz[i] = 0.f;
  for (long long r = (long long)blockIdx.x * 8 + warp; r < rows; r += (long long)gridDim.x * 8) {
    float zn[2 * kP], d[2 * kP], gq[2 * kP], gk[2 * kP];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < kP; ++i) {
      const int j = lane + 32 * i;
      if (j < half) {
        load_pair(dq + r * ldq + 2 * j, gq[2 * i], gq[2 * i + 1]);
        load_pair(dk + r * ldk + 2 * j, gk[2 * i], gk[2 * i + 1]);
      }
    }
#pragma unroll
    for (int i = 0; i < kP; ++i) {
      const int j = lane + 32 * i;
      zn[2 * i] = zn[2 * i + 1] = d[2 * i] = d[2 * i + 1] = 0.f;
      if (j < half) {
        load_pair(z + r * ldz + 2 * j, zn[2 * i], zn[2 * i + 1]);
        ss = fmaf(zn[2 * i], zn[2 * i], fmaf(zn[2 * i + 1], zn[2 * i + 1], ss));
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float norm = sqrtf(ss);
    const float inv = 1.f / fmaxf(norm, eps);
    const int pos = (int)(r % period);
    const float2* rk = reinterpret_cast<const float2*>(rot) + (size_t)pos * half;
    const float2* rq = reinterpret_cast<const float2*>(rot) + (size_t)(pos + q_offset) * half;
    float dots = 0.f;
#pragma unroll
    for (int i = 0; i < kP; ++i) {
      const int j = lane + 32 * i;
      if (j < half) {
        const int c = 2 * j;
        float qa = gq[2 * i], qb = gq[2 * i + 1], ka = gk[2 * i], kb = gk[2 * i + 1];
        if (rot) {   // the transposed rotations
          const float2 wq = __ldg(rq + j), wk = __ldg(rk + j);
          const float q0 = qa * wq.x + qb * wq.y, k0 = ka * wk.x + kb * wk.y;
          qb = qb * wq.x - qa * wq.y;
          kb = kb * wk.x - ka * wk.y;
          qa = q0;
          ka = k0;
        }
        zn[2 * i] *= inv;
        zn[2 * i + 1] *= inv;
        sb0[2 * i] += qa;
        sb0[2 * i + 1] += qb;
        sb1[2 * i] += ka;
        sb1[2 * i + 1] += kb;
        sg0[2 * i] = fmaf(qa, zn[2 * i], sg0[2 * i]);
        sg0[2 * i + 1] = fmaf(qb, zn[2 * i + 1], sg0[2 * i + 1]);
        sg1[2 * i] = fmaf(ka, zn[2 * i], sg1[2 * i]);
        sg1[2 * i + 1] = fmaf(kb, zn[2 * i + 1], sg1[2 * i + 1]);
        d[2 * i] = fmaf(qa, __ldg(gamma + c) + 1.f, ka * (__ldg(gamma + cols + c) + 1.f));
        d[2 * i + 1] = fmaf(qb, __ldg(gamma + c + 1) + 1.f, kb * (__ldg(gamma + cols + c + 1) + 1.f));
        dots = fmaf(d[2 * i], zn[2 * i], fmaf(d[2 * i + 1], zn[2 * i + 1], dots));
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dots += __shfl_xor_sync(0xffffffffu, dots, o);
    if (norm < eps) dots = 0.f;   // the divisor is eps itself
#pragma unroll
    for (int i = 0; i < kP; ++i) {
      const int j = lane + 32 * i;
      if (j < half) {
        const float v0 = inv * (d[2 * i] - zn[2 * i] * dots), v1 = inv * (d[2 * i + 1] - zn[2 * i + 1] * dots);
        store_pair(dz + r * ldd + 2 * j, v0, v1);
        sz[2 * i] += v0;
        sz[2 * i + 1] += v1;
      }
    }
  }
  // the block's eight warps, two values of every lane at a time
  auto flush = [&](const float(&s)[2 * kP], float* out) {
    if (!out) return;
#pragma unroll
    for (int i = 0; i < kP; ++i) {
      if (64 * i >= cols) break;
      __syncthreads();
      red[warp][2 * lane] = s[2 * i];
      red[warp][2 * lane + 1] = s[2 * i + 1];
      __syncthreads();
      if (threadIdx.x < 64 && 64 * i + (int)threadIdx.x < cols) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) v += red[w][threadIdx.x];
        atomicAdd(out + 64 * i + threadIdx.x, v);
      }
    }
  };
  flush(sg0, dgamma);
  flush(sg1, dgamma + cols);
  flush(sb0, dbeta);
  flush(sb1, dbeta + cols);
  flush(sz, colsum);
}

// softmax over a row of scores + bias[column - row + span - 1], padded columns out; a fully padded row takes no mask
// Rows of at most 2048 values of 16 bits (1024 fp32) in whole 16-byte pieces: a warp takes one, kN pieces per lane, in
// registers.  Bound by the bias's unaligned loads (a diagonal per row) and the instructions around them.
template <typename T, int kN>
__global__ void __launch_bounds__(256) bias_softmax_warp_kernel(const T* x, T* y, const T* bias, const unsigned char* mask, int rows,
                                                                int cols, int span) {
  constexpr int kV = 16 / (int)sizeof(T);
  using M = typename std::conditional<kV == 8, uint2, unsigned>::type;   // the mask of a piece
  const int lane = threadIdx.x & 31, b = blockIdx.y, r = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (r >= rows) return;
  const T* xr = x + ((size_t)b * rows + r) * cols;
  T* yr = y + ((size_t)b * rows + r) * cols;
  const T* br = bias + (span - 1 - r);
  float v[kN][kV];
  unsigned pad[kN];
  bool live = mask == nullptr;
#pragma unroll
  for (int j = 0; j < kN; ++j) {
    const int c = (lane + 32 * j) * kV;
    pad[j] = 0u;
    if (c < cols) {
      const uint4 raw = *reinterpret_cast<const uint4*>(xr + c);
      if (mask) {
        const M m = __ldg(reinterpret_cast<const M*>(mask + (size_t)b * cols + c));
        const unsigned char* e = reinterpret_cast<const unsigned char*>(&m);
#pragma unroll
        for (int k = 0; k < kV; ++k) pad[j] |= (e[k] != 0 ? 1u : 0u) << k;
        live |= pad[j] != (1u << kV) - 1u;
      }
#pragma unroll
      for (int k = 0; k < kV; ++k) v[j][k] = Elem<T>::ld_shared(reinterpret_cast<const T*>(&raw) + k) + Elem<T>::ld(br + c + k);
    } else {
#pragma unroll
      for (int k = 0; k < kV; ++k) v[j][k] = -INFINITY;
    }
  }
  const bool all = !__any_sync(0xffffffffu, live);   // (padded throughout: as without a mask)
  float m = -INFINITY;
#pragma unroll
  for (int j = 0; j < kN; ++j)
#pragma unroll
    for (int k = 0; k < kV; ++k) {
      if (!all && ((pad[j] >> k) & 1u)) v[j][k] = -INFINITY;
      m = fmaxf(m, v[j][k]);
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < kN; ++j)
#pragma unroll
    for (int k = 0; k < kV; ++k) {
      v[j][k] = m == -INFINITY ? 0.f : exp_of<T>(v[j][k] - m);
      s += v[j][k];
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const float inv = s > 0.f ? 1.f / s : 0.f;
#pragma unroll
  for (int j = 0; j < kN; ++j) {
    const int c = (lane + 32 * j) * kV;
    if (c < cols) {
      uint4 raw;
#pragma unroll
      for (int k = 0; k < kV; ++k) Elem<T>::st(reinterpret_cast<T*>(&raw) + k, v[j][k] * inv);
      *reinterpret_cast<uint4*>(yr + c) = raw;
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(128) bias_softmax_kernel(const T* x, T* y, const T* bias, const unsigned char* mask,
                                                           int rows, int cols, int span) {
  extern __shared__ float row[];
  __shared__ float red[4];
  __shared__ int live;
  const int b = blockIdx.y, r = blockIdx.x, tid = threadIdx.x;
  const T* xr = x + ((size_t)b * rows + r) * cols;
  T* yr = y + ((size_t)b * rows + r) * cols;
  const T* br = bias + (span - 1 - r);
  const unsigned char* mr = mask ? mask + (size_t)b * cols : nullptr;
  if (mr) {
    if (tid == 0) live = 0;
    __syncthreads();
    int any = 0;
    for (int c = tid; c < cols; c += 128) any |= mr[c] == 0;
    if (any) live = 1;
    __syncthreads();
    if (!live) mr = nullptr;
  }
  float m = -INFINITY;
  for (int c = tid; c < cols; c += 128) {
    const float v = (mr && mr[c]) ? -INFINITY : Elem<T>::ld(xr + c) + Elem<T>::ld(br + c);
    row[c] = v;
    m = fmaxf(m, v);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((tid & 31) == 0) red[tid >> 5] = m;
  __syncthreads();
  m = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
  __syncthreads();
  float s = 0.f;
  for (int c = tid; c < cols; c += 128) {
    const float e = m == -INFINITY ? 0.f : exp_of<T>(row[c] - m);
    row[c] = e;
    s += e;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((tid & 31) == 0) red[tid >> 5] = s;
  __syncthreads();
  s = (red[0] + red[1]) + (red[2] + red[3]);
  const float inv = s > 0.f ? 1.f / s : 0.f;
  for (int c = tid; c < cols; c += 128) Elem<T>::st(yr + c, row[c] * inv);
}

// dbias[column - row + span - 1] = sum of ds along the diagonals; a thread owns a diagonal of 64 rows of some batches
template <typename T>
__global__ void __launch_bounds__(256) bias_grad_kernel(const T* ds, float* dbias, int batch, int rows, int cols, int span) {
  const int diag = (int)(blockIdx.x * 256 + threadIdx.x) - (rows - 1);   // column - row
  if (diag >= cols) return;
  const int r0 = blockIdx.y * 64, r1 = min(rows, r0 + 64);
  const int lo = max(r0, -diag), hi = min(r1, cols - diag);
  if (lo >= hi) return;
  float s = 0.f;
  for (int b = blockIdx.z; b < batch; b += gridDim.z) {
    const T* p = ds + ((size_t)b * rows + lo) * cols + lo + diag;
    int r = lo;
    for (; r + 8 <= hi; r += 8) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = Elem<T>::ldv(p + (size_t)u * (cols + 1));
#pragma unroll
      for (int u = 0; u < 8; ++u) s += v[u];
      p += (size_t)8 * (cols + 1);
    }
    for (; r < hi; ++r, p += cols + 1) s += Elem<T>::ld(p);
  }
  atomicAdd(dbias + diag + span - 1, s);
}

static int gate_bwd_common(int op, GateBwd p, int dtype, int64_t rows, int cols, mega_stream_t stream) {
  if (!valid_dtype(dtype)) return MEGA_ERR_DTYPE;
  if (rows <= 0 || cols <= 0) return MEGA_ERR_SHAPE;
  const int es = elem_size(dtype), n = 16 / es;
  if (cols % n != 0) return MEGA_ERR_STRIDE;
  const void* ptr[] = {p.g, p.a, p.b, p.c, p.d, p.o0, p.o1, p.o2};
  const long long ld[] = {p.ldg, p.lda, p.ldb, p.ldc, p.ldd, p.l0, p.l1, p.l2};
  for (int i = 0; i < 8; ++i)
    if (ptr[i] && (!aligned_to(ptr[i], 16) || (ld[i] * es) % 16 != 0)) return MEGA_ERR_ALIGN;
  p.rows = rows;
  p.cols = cols;
  const int gx = (cols / n + 31) / 32;
  // enough blocks for two rounds of eight per SM; a block's column sums cost about 32 rows
  long long per = (rows * gx + 148 * 16 - 1) / (148 * 16);
  per = per < 32 ? 32 : per;
  if ((rows + per - 1) / per > 65535) per = (rows + 65534) / 65535;
  p.per = (int)per;
  const dim3 grid(gx, (unsigned)((rows + per - 1) / per));
  MEGA_DISPATCH_DTYPE(dtype, {
    if (op == 0) launch(gate_bwd_kernel<T, 0>, grid, 256, 0, stream, p);
    else if (op == 1) launch(gate_bwd_kernel<T, 1>, grid, 256, 0, stream, p);
    else launch(gate_bwd_kernel<T, 2>, grid, 256, 0, stream, p);
  });
  return check_launch("gate_bwd");
}

struct ToFloat {
  const void* src[8];
  float* dst[8];
  long long n[8];
};
template <typename T>
__global__ void __launch_bounds__(256) to_float_kernel(ToFloat a) {
  const int k = blockIdx.y;
  const T* s = reinterpret_cast<const T*>(a.src[k]);
  for (long long i = blockIdx.x * 256 + threadIdx.x; i < a.n[k]; i += (long long)gridDim.x * 256) a.dst[k][i] = Elem<T>::ld(s + i);
}

}  // namespace

}  // namespace mega

using namespace mega;

extern "C" int mega_gate_silu_bwd(const void* dy, int64_t ld_dy, const void* a, int64_t ld_a, void* da, int64_t ld_da,
                                  float* colsum, int dtype, int64_t rows, int cols, mega_stream_t stream) {
  if (!dy || !a || !da) return MEGA_ERR_NULL;
  GateBwd p{};
  p.g = dy; p.ldg = ld_dy; p.a = a; p.lda = ld_a; p.o0 = da; p.l0 = ld_da; p.s0 = colsum;
  return gate_bwd_common(0, p, dtype, rows, cols, stream);
}

extern "C" int mega_gate_mul_silu_bwd(const void* dy, int64_t ld_dy, const void* a, int64_t ld_a, const void* r, int64_t ld_r,
                                      void* da, int64_t ld_da, void* dr, int64_t ld_dr, float* colsum_r, int dtype,
                                      int64_t rows, int cols, mega_stream_t stream) {
  if (!dy || !a || !r || !da || !dr) return MEGA_ERR_NULL;
  GateBwd p{};
  p.g = dy; p.ldg = ld_dy; p.a = a; p.lda = ld_a; p.b = r; p.ldb = ld_r;
  p.o0 = da; p.l0 = ld_da; p.o1 = dr; p.l1 = ld_dr; p.s0 = colsum_r;
  return gate_bwd_common(1, p, dtype, rows, cols, stream);
}

extern "C" int mega_gate_output_bwd(const void* dout, int64_t ld_do, const void* residual, int64_t ld_res, const void* u,
                                    int64_t ld_u, const void* hx, int64_t ld_hx, const void* h_lin, int64_t ld_h, void* dres,
                                    int64_t ld_dres, void* du, int64_t ld_du, void* dhx, int64_t ld_dhx, float* colsum_u,
                                    float* colsum_hx, int dtype, int64_t rows, int cols, mega_stream_t stream) {
  if (!dout || !residual || !u || !hx || !h_lin || !dres || !du || !dhx) return MEGA_ERR_NULL;
  GateBwd p{};
  p.g = dout; p.ldg = ld_do; p.a = residual; p.lda = ld_res; p.b = u; p.ldb = ld_u; p.c = hx; p.ldc = ld_hx; p.d = h_lin;
  p.ldd = ld_h; p.o0 = dres; p.l0 = ld_dres; p.o1 = du; p.l1 = ld_du; p.o2 = dhx; p.l2 = ld_dhx;
  p.s0 = colsum_u; p.s1 = colsum_hx;
  return gate_bwd_common(2, p, dtype, rows, cols, stream);
}

extern "C" int mega_gate_qk_bwd(const void* z, int64_t ld_z, const float* gamma, const float* rot, int positions, int period,
                                int q_offset, const void* dq, int64_t ld_dq, const void* dk, int64_t ld_dk, void* dz,
                                int64_t ld_dz, float* dgamma, float* dbeta, float* colsum, int dtype, int64_t rows, int cols,
                                double eps, mega_stream_t stream) {
  if (!z || !gamma || !dq || !dk || !dz || !dgamma || !dbeta) return MEGA_ERR_NULL;
  if (!valid_dtype(dtype)) return MEGA_ERR_DTYPE;
  if (rows <= 0 || cols <= 0 || (cols & 1)) return MEGA_ERR_SHAPE;
  if (rot && (period <= 0 || q_offset < 0 || period + q_offset > positions)) return MEGA_ERR_SHAPE;
  if (cols > 64 * kQkPairs) return MEGA_ERR_UNSUPPORTED;
  // (pairs of values are read and written at once)
  if (ld_z < cols || ld_dq < cols || ld_dk < cols || ld_dz < cols) return MEGA_ERR_STRIDE;
  const size_t pair = 2 * elem_size(dtype);
  if (!aligned_to(z, pair) || !aligned_to(dq, pair) || !aligned_to(dk, pair) || !aligned_to(dz, pair) || !aligned_to(rot, 8) ||
      ((ld_z | ld_dq | ld_dk | ld_dz) & 1))
    return MEGA_ERR_ALIGN;
  const long long want = (rows + 31) / 32;   // four rows per warp at least
  const unsigned grid = (unsigned)(want > 148 * 4 ? 148 * 4 : want);
  MEGA_DISPATCH_DTYPE(dtype, {
    auto run = [&](auto kernel) {
      launch(kernel, grid, 256, 0, stream, (const T*)z, (long long)ld_z, gamma, rot, rot ? period : 1, q_offset, (const T*)dq,
             (long long)ld_dq, (const T*)dk, (long long)ld_dk, (T*)dz, (long long)ld_dz, dgamma, dbeta, colsum, (long long)rows, cols,
             (float)eps);
    };
    if (cols <= 64) run(gate_qk_bwd_kernel<T, 1>);
    else if (cols <= 128) run(gate_qk_bwd_kernel<T, 2>);
    else if (cols <= 256) run(gate_qk_bwd_kernel<T, 4>);
    else run(gate_qk_bwd_kernel<T, kQkPairs>);
  });
  return check_launch("gate_qk_bwd");
}

extern "C" int mega_attention_bias_softmax_fwd(const void* x, void* y, const void* bias, int span, const uint8_t* pad_mask,
                                               int dtype, int64_t batch, int rows, int cols, mega_stream_t stream) {
  if (!x || !y || !bias) return MEGA_ERR_NULL;
  if (!valid_dtype(dtype)) return MEGA_ERR_DTYPE;
  if (batch <= 0 || batch > 65535 || rows <= 0 || cols <= 0 || span < rows || span < cols) return MEGA_ERR_SHAPE;
  if (cols > 48 * 1024) return MEGA_ERR_UNSUPPORTED;   // a row lives in shared memory
  const dim3 grid(rows, (unsigned)batch);
  const int kv = 16 / elem_size(dtype);
  if (cols % kv == 0 && cols <= 8 * 32 * kv && aligned_to(x, 16) && aligned_to(y, 16) && aligned_to(pad_mask, kv)) {
    const dim3 gridw((rows + 7) / 8, (unsigned)batch);
    const int vecs = (cols / kv + 31) / 32;
    MEGA_DISPATCH_DTYPE(dtype, {
      auto run = [&](auto kernel) {
        launch(kernel, gridw, 256, 0, stream, (const T*)x, (T*)y, (const T*)bias, pad_mask, rows, cols, span);
      };
      if (vecs <= 1) run(bias_softmax_warp_kernel<T, 1>);
      else if (vecs <= 2) run(bias_softmax_warp_kernel<T, 2>);
      else if (vecs <= 4) run(bias_softmax_warp_kernel<T, 4>);
      else run(bias_softmax_warp_kernel<T, 8>);
    });
    return check_launch("attention_bias_softmax_fwd");
  }
  MEGA_DISPATCH_DTYPE(dtype, launch(bias_softmax_kernel<T>, grid, 128, (size_t)cols * 4, stream, (const T*)x, (T*)y,
                                    (const T*)bias, pad_mask, rows, cols, span));
  return check_launch("attention_bias_softmax_fwd");
}

extern "C" int mega_attention_bias_grad(const void* ds, float* dbias, int span, int dtype, int64_t batch, int rows, int cols,
                                        mega_stream_t stream) {
  if (!ds || !dbias) return MEGA_ERR_NULL;
  if (!valid_dtype(dtype)) return MEGA_ERR_DTYPE;
  if (batch <= 0 || rows <= 0 || cols <= 0 || span < rows || span < cols) return MEGA_ERR_SHAPE;
  const dim3 grid((rows + cols - 1 + 255) / 256, (rows + 63) / 64, (unsigned)(batch > 4 ? 4 : batch));
  if (grid.y > 65535) return MEGA_ERR_UNSUPPORTED;
  MEGA_DISPATCH_DTYPE(dtype, launch(bias_grad_kernel<T>, grid, 256, 0, stream, (const T*)ds, dbias, (int)batch, rows, cols, span));
  return check_launch("attention_bias_grad");
}

extern "C" int mega_to_float(const void* const* src, float* const* dst, const int64_t* n, int count, int dtype,
                             mega_stream_t stream) {
  if (!src || !dst || !n) return MEGA_ERR_NULL;
  if (dtype != MEGA_BF16 && dtype != MEGA_F16) return MEGA_ERR_DTYPE;
  if (count < 1 || count > 8) return MEGA_ERR_SHAPE;
  ToFloat a{};
  long long most = 0;
  for (int i = 0; i < count; ++i) {
    if (!src[i] || !dst[i]) return MEGA_ERR_NULL;
    if (n[i] < 0) return MEGA_ERR_SHAPE;
    a.src[i] = src[i];
    a.dst[i] = dst[i];
    a.n[i] = n[i];
    if (n[i] > most) most = n[i];
  }
  const long long blocks = most / 256 + 1;
  const dim3 grid((unsigned)(blocks > 256 ? 256 : blocks), count);
  if (dtype == MEGA_BF16) launch(to_float_kernel<__nv_bfloat16>, grid, 256, 0, stream, a);
  else launch(to_float_kernel<__half>, grid, 256, 0, stream, a);
  return check_launch("to_float");
}
