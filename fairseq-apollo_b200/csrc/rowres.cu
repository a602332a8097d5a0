// Row-resident EMA for length-contiguous activations ((B, D, L) memory): causal or bidirectional,
// optionally preceded by a fused per-channel SequenceNorm.
//
// A CTA keeps rows (batch, channel) in shared memory (fp32) and cuts each into segments of 32 positions, which turns the
// layer into three products with matrices of the channel, S the number of segments:
//   local pole states   H = X V      X (S, 32) the row, V (32, poles): q^(31-k), anti-causal q^k
//   outputs             Y = X T + C E   T (32, 32) the taps between positions of a segment, both directions at once;
//                                    C (S, poles) the states that enter a segment, E (poles, 32)
// with omega x added in fp32, and a scan of the S states per pole (C from H): the run that a lane holds, lanes by shuffles,
// warps through a table.
// 96 multiply-adds per element bidirectional, 64 causal.  HBM sees the row once in, once out.
//
// fp32 on the bf16 tensor pipe: a float is exactly the sum of three bf16 values, and six of the nine products (all
// but those below 2^-24 of the largest) are accumulated in fp32.  That is 576 bf16 products per element where the packed
// FMA pipe, at an eleventh of the rate, would spend 96 slots.  The tensor pipe truncates its sums, so what would be large
// in them stays out: omega x, usually the larger part of an output, and the leading products of the outputs, which have an
// accumulator of their own.  Against the float64 recurrence: 1.0e-7 bidirectional, 6.4e-8 causal (the fp32 walk: 1.0e-7 and
// 6.8e-8; omega on T's diagonal, one accumulator and taps summed in fp32: 1.2e-7 and 8.3e-8; each tile's leading products
// added by themselves: 9.3e-8 and 6.1e-8, at 717 us where the case below takes 686).
//
// B = 32, D = 256, L = 16384 fp32 bidirectional after the norm: 1310 us as a walk (FMA, one row per SM), 609 us now (691
// padded by up to half): the tensor pipe is at 48 %, shared memory at 55 %, issue slots at 41 %, the rest is latency, 16
// warps being what the registers allow.  L = 1024, B = 32, D = 128: 42 us.  (L2 flushed in front of each call.)
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "rowres.cuh"
#include "split_mma.cuh"
#include "tma.cuh"

namespace mega {

namespace {

constexpr int kRowNP = 16;    // poles per direction
constexpr int kSeg = 32;      // positions of a segment
constexpr int kMaxThreads = 512;

// q^32 of a pole, then q^(32 g R) for g = 0 .. 8, R the segments a lane holds
constexpr int kQ1 = 0, kQRun = 1, kQRows = 10;

template <bool kBidir>
struct RowSmem {   // byte offsets: the channel's tables first, at addresses that are constants, then the rows
  static constexpr int frag = 0, pw = frag + (kBidir ? 24 : 16) * kBlockBytes, tap = pw + 33 * 32 * 4, q = tap + 64 * 4,
                       tot = q + kQRows * 32 * 4, red = tot + (kMaxThreads / 32) * 32 * 4,
                       rows = red + 3 * (kMaxThreads / 32) * 4;
  static_assert(rows % 16 == 0, "rows are read in pieces of 16 bytes");
  __host__ __device__ static constexpr int mask(int nseg) { return rows + nseg * kSeg * 4; }
  __host__ __device__ static constexpr int total(int nseg) { return mask(nseg) + 2 * nseg * 4; }
};

// d = products of K reduction tiles, all but those of the leading parts, smallest first, then those.  The tensor pipe truncates
// its sums: kApart gives the leading products an accumulator of their own, which an fp32 addition joins.  Block of tile k at
// block + k * stride.
template <int K, bool kApart>
__device__ __forceinline__ void products(float (&d)[4], const uint32_t (&a)[K][3][4], const unsigned char* block, int stride) {
  float l[4] = {0.f, 0.f, 0.f, 0.f};
  d[0] = d[1] = d[2] = d[3] = 0.f;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const Frag b = load_frag(block + k * stride);
    if (kApart) mma(l, a[k][0], b.u.x, b.u.y);
    mma(d, a[k][2], b.u.x, b.u.y);
    mma(d, a[k][0], b.v.x, b.v.y);
    mma(d, a[k][1], b.u.z, b.u.w);
    mma(d, a[k][1], b.u.x, b.u.y);
    mma(d, a[k][0], b.u.z, b.u.w);
  }
  if (kApart) {
#pragma unroll
    for (int i = 0; i < 4; ++i) d[i] += l[i];
  } else {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const uint2 b = *reinterpret_cast<const uint2*>(block + k * stride + (threadIdx.x & 31) * 16);
      mma(d, a[k][0], b.x, b.y);
    }
  }
}
// zero where the mask's bits say so
__device__ __forceinline__ float4 keep(float4 v, unsigned m) {
  return make_float4(m & 1 ? 0.f : v.x, m & 2 ? 0.f : v.y, m & 4 ? 0.f : v.z, m & 8 ? 0.f : v.w);
}
// count, mean, squared deviations (Chan et al.'s pairwise combination)
struct Run {
  float n, mean, m2;
};
__device__ __forceinline__ Run combine(Run a, Run b) {
  const float n = a.n + b.n, w = n > 0.f ? b.n / n : 0.f, d = b.mean - a.mean;
  return {n, fmaf(d, w, a.mean), a.m2 + b.m2 + d * d * a.n * w};
}

__device__ __forceinline__ Run row_run(Run v, float* red, int w, int nw) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v = combine(v, Run{__shfl_xor_sync(0xffffffffu, v.n, o), __shfl_xor_sync(0xffffffffu, v.mean, o),
                       __shfl_xor_sync(0xffffffffu, v.m2, o)});
  if (lane == 0) {
    red[3 * w] = v.n;
    red[3 * w + 1] = v.mean;
    red[3 * w + 2] = v.m2;
  }
  __syncthreads();
  Run r{0.f, 0.f, 0.f};
  for (int i = 0; i < nw; ++i) r = combine(r, Run{red[3 * i], red[3 * i + 1], red[3 * i + 2]});
  return r;
}

// positions in the row buffer are in pieces of four, a lane's runs of 2^rs segments one after another; every other run of 2^rs segments swaps the halves of its segments,
// so that the eight lanes of a 16-byte phase (two segments a run apart, four pieces) hit different banks
__device__ __forceinline__ int piece(int seg, int c, int rs) { return seg * 8 + (c ^ (((seg >> rs) & 1) << 2)); }
// time of slot k of a reduction tile (a lane's four slots are four consecutive positions) and position of column c of
// an output tile (two tiles give a lane four consecutive positions)
__device__ __forceinline__ int slot_time(int kt, int k) { return 16 * kt + 4 * ((k & 7) >> 1) + 2 * (k >> 3) + (k & 1); }
__device__ __forceinline__ int column_pos(int nt, int c) { return 16 * (nt >> 1) + 4 * (c >> 1) + 2 * (nt & 1) + (c & 1); }

// The channel's matrices as B fragments, and its tables of powers.
template <bool kBidir>
__device__ __forceinline__ void prepare_channel(const RowArgs& a, int d, int per_warp, unsigned char* smem) {
  using o = RowSmem<kBidir>;
  float* pw = reinterpret_cast<float*>(smem + o::pw);     // [33][32]: q^k of pole column n
  float* tap = reinterpret_cast<float*>(smem + o::tap);   // lag + 31
  float* qt = reinterpret_cast<float*>(smem + o::q);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
  const int n = lane & 15;
  const bool live = n < a.N && (kBidir || lane < 16);
  const size_t at = (size_t)(d + (lane < 16 ? 0 : a.D)) * a.N + n;
  const float q = live ? __ldg(a.q + at) : 0.f;
  const double c = live ? (double)__ldg(a.p + at) * __ldg(a.g + at) : 0.;
  for (int l = tid; l < 31; l += blockDim.x)
    if (!kBidir) tap[l] = 0.f;
  {
    // (in double, rounded once: few enough to keep their roundings out of the result; the poles' shares of a tap alternate
    // in sign.  Lanes 0 - 15 sum those of the causal half, the others those of the anti-causal one)
    double step = 1., v = 1.;
    for (int i = 0; i < nw; ++i) step *= q;
    for (int i = 0; i < w; ++i) v *= q;
    for (int k = w; k <= 32; k += nw) {
      pw[k * 32 + lane] = (float)v;
      double t = c * v;
#pragma unroll
      for (int s = 8; s > 0; s >>= 1) t += __shfl_xor_sync(0xffffffffu, t, s);
      const int back = a.shift ? k + 1 : k;   // lag of the anti-causal half
      if (kBidir && back == 0) t += __shfl_xor_sync(0xffffffffu, t, 16);
      if (lane == 0 && k < 32) tap[31 + k] = (float)t;
      if (kBidir && lane == 16 && back > 0 && back < 32) tap[31 - back] = (float)t;
      v *= step;
    }
  }
  __syncthreads();
  if (w == 0) {   // powers over segments, and over the run of segments that a lane holds
    double q32 = q;
    for (int i = 0; i < 5; ++i) q32 *= q32;
    double r = q32;
    for (int i = 1; i < 2 * per_warp; i *= 2) r *= r;
    qt[kQ1 * 32 + lane] = (float)q32;
    double v = 1.;
    for (int g = 0; g <= 8; ++g) {
      qt[(kQRun + g) * 32 + lane] = (float)v;
      v *= r;
    }
  }
  constexpr int kStateTiles = kBidir ? 4 : 2, kStateK = kBidir ? 2 : 1;
  constexpr int kV = 2 * kStateTiles, kT = 8, kE = 4 * kStateK;
  for (int e = tid; e < (kV + kT + kE) * 32; e += blockDim.x) {
    const int blk = e >> 5, g = lane >> 2, t = lane & 3;   // (blockDim is a multiple of 32)
    float v[4];   // slots 2t, 2t + 1, 2t + 8, 2t + 9 of column g
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = 2 * t + (i & 1) + 8 * (i >> 1);
      if (blk < kV) {
        const int kt = blk / kStateTiles, pole = 8 * (blk % kStateTiles) + g, time = slot_time(kt, k);
        v[i] = pw[(pole < 16 ? 31 - time : time) * 32 + pole];
      } else if (blk < kV + kT) {
        const int kt = (blk - kV) >> 2, nt = (blk - kV) & 3;
        v[i] = tap[column_pos(nt, g) - slot_time(kt, k) + 31];
      } else {
        const int kt = (blk - kV - kT) >> 2, nt = (blk - kV - kT) & 3, pole = 16 * kt + k, pos = column_pos(nt, g);
        const int m = pole & 15;
        const size_t row = (size_t)(d + (pole < 16 ? 0 : a.D)) * a.N + m;
        const double cp = m < a.N ? (double)__ldg(a.p + row) * __ldg(a.g + row) : 0.;
        v[i] = (float)(cp * pw[(pole < 16 ? pos + 1 : (a.shift ? 31 : 32) - pos) * 32 + pole]);
      }
    }
    store_frag(smem + o::frag + blk * kBlockBytes, v);
  }
}

// Bit i of word s: position 32 s + i of the row is padded or beyond L; the warp's segments.  Returns the bits that any
// of them have, and in all those that all have.  m: the row's bytes or null; first: nothing lies before them.
__device__ __forceinline__ unsigned load_mask(const unsigned char* m, bool first, int L, int base, int segs, unsigned* mk, unsigned& all) {
  const int lane = threadIdx.x & 31;
  const int shift = (int)(reinterpret_cast<uintptr_t>(m) & 3);
  unsigned any = 0u;
  all = ~0u;
  for (int s = base + lane; s < base + segs; s += 32) {
    const int i = kSeg * s;
    unsigned bits = L - i >= kSeg ? 0u : L <= i ? ~0u : ~0u << (L - i);
    if (m && bits != ~0u) {
      if (i + kSeg + 4 <= L && (shift == 0 || !first || i > 0)) {   // nine aligned words hold the segment's bytes
        const unsigned* at = reinterpret_cast<const unsigned*>(m + i - shift);
        unsigned v[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) v[k] = __ldg(at + k);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const unsigned four = __funnelshift_r(v[k], v[k + 1], 8 * shift);
          bits |= ((__vsetgtu4(four, 0u) * 0x01020408u) >> 24 & 15u) << (4 * k);
        }
      } else {
#pragma unroll 8
        for (int k = 0; k < kSeg; ++k)
          if (i + k < L && __ldg(m + i + k) != 0) bits |= 1u << k;
      }
    }
    mk[s] = bits;
    any |= bits;
    all &= bits;
  }
  any = __reduce_or_sync(0xffffffffu, any);
  all = __reduce_and_sync(0xffffffffu, all);
  return any;
}

// the warp's segments in fp32, zero beyond L (padded positions are zeroed where they are read)
template <typename T, int rs>
__device__ __forceinline__ void load_x_row(const T* xg, int L, int base, float* xs) {
  constexpr int rounds = 2 << rs;   // of 32 pieces
  const int lane = threadIdx.x & 31;
  const bool vec = (reinterpret_cast<uintptr_t>(xg) & 15) == 0;
  float* dst = xs + 32 * base;
  const int i0 = kSeg * base;
  if (!vec) {   // (rows that start anywhere: a position per lane)
#pragma unroll 32
    for (int k = 0; k < 4 * rounds; ++k) {
      const int i = i0 + 32 * k + lane;
      float* at = dst + 32 * k + (lane ^ (((k >> rs) & 1) << 4));
      if constexpr (sizeof(T) == 4) {
        if (i < L)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(at)), "l"(xg + i) : "memory");
        else
          *at = 0.f;
      } else {
        *at = i < L ? Elem<T>::ldv(xg + i) : 0.f;
      }
    }
  } else if constexpr (sizeof(T) == 4) {
#pragma unroll 8
    for (int k = 0; k < rounds; ++k) {
      const int i = i0 + 128 * k + 4 * lane;
      const int bytes = max(0, min(16, 4 * (L - i)));
      asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;" ::"r"(
                       smem_u32(dst + 128 * k + 4 * (lane ^ (((k >> (rs - 2)) & 1) << 2)))),
                   "l"(bytes ? xg + i : xg), "r"(bytes)
                   : "memory");
    }
  } else {
#pragma unroll 8
    for (int k = 0; k < rounds / 2; ++k) {
      const int i = i0 + 256 * k + 8 * lane;
      T v[8];
      if (i + 8 <= L) {
        *reinterpret_cast<uint4*>(v) = __ldg(reinterpret_cast<const uint4*>(xg + i));
      } else {
#pragma unroll
        for (int u = 0; u < 8; ++u) Elem<T>::st(v + u, i + u < L ? Elem<T>::ld(xg + i + u) : 0.f);
      }
      const int swap = (((64 * k + 2 * lane) >> (rs + 3)) & 1) << 2;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float4 f;
        f.x = Elem<T>::ld_shared(v + 4 * h); f.y = Elem<T>::ld_shared(v + 4 * h + 1);
        f.z = Elem<T>::ld_shared(v + 4 * h + 2); f.w = Elem<T>::ld_shared(v + 4 * h + 3);
        *reinterpret_cast<float4*>(dst + 4 * ((64 * k + 2 * lane + h) ^ swap)) = f;
      }
    }
  }
}

// The warp's outputs.  kResidual: a padded position's comes without the residual, which is that of the unmasked x.
template <typename T, bool kResidual, int rs>
__device__ __forceinline__ void store_row(const float* xs, const unsigned* mk, unsigned any, int L, int base, float om, int silu,
                                          const T* xg, T* yg) {
  constexpr int rounds = 2 << rs;   // of 32 pieces
  const int lane = threadIdx.x & 31, i0 = kSeg * base;
  const float* src = xs + 32 * base;
  const bool pieces = (reinterpret_cast<uintptr_t>(yg) & (4 * sizeof(T) - 1)) == 0 && !(kResidual && any);
  const int whole = pieces ? min(rounds, max(0, (L - i0) / 128)) : 0;
  auto four = [&](int k) {   // positions per lane
    float4 v = *reinterpret_cast<const float4*>(src + 4 * ((32 * k + lane) ^ (((k >> (rs - 2)) & 1) << 2)));
    if (silu) v = make_float4(siluf_(v.x), siluf_(v.y), siluf_(v.z), siluf_(v.w));
    T* at = yg + i0 + 128 * k + 4 * lane;
    if constexpr (sizeof(T) == 4) {
      *reinterpret_cast<float4*>(at) = v;
    } else {
      uint2 packed;
      T* pt = reinterpret_cast<T*>(&packed);
      Elem<T>::st(pt, v.x); Elem<T>::st(pt + 1, v.y); Elem<T>::st(pt + 2, v.z); Elem<T>::st(pt + 3, v.w);
      *reinterpret_cast<uint2*>(at) = packed;
    }
  };
  if (whole == rounds) {
#pragma unroll 4
    for (int k = 0; k < rounds; ++k) four(k);
    return;
  }
  for (int k = 0; k < whole; ++k) four(k);
  for (int k0 = 4 * whole; k0 < 4 * rounds && i0 + 32 * k0 < L; k0 += 4) {   // one per lane
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = src[32 * (k0 + j) + (lane ^ ((((k0 + j) >> rs) & 1) << 4))];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = i0 + 32 * (k0 + j) + lane;
      if (i < L) {
        if (kResidual && any && ((mk[base + k0 + j] >> lane) & 1)) v[j] = fmaf(om, Elem<T>::ld(xg + i), v[j]);
        if (silu) v[j] = siluf_(v[j]);
        Elem<T>::st(yg + i, v[j]);
      }
    }
  }
}

// exclusive scan of v over the eight row groups of a fragment (lanes with the same t), along time or against it, with
// the powers of one, two and four steps; total: of all eight
template <bool kUp>
__device__ __forceinline__ float scan8(float v, float q1, float q2, float q4, float& total) {
  const int lane = threadIdx.x & 31, g = lane >> 2, at = kUp ? g : 7 - g;
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    const float u = kUp ? __shfl_up_sync(0xffffffffu, v, 4 * o) : __shfl_down_sync(0xffffffffu, v, 4 * o);
    if (at >= o) v = fmaf(o == 1 ? q1 : o == 2 ? q2 : q4, u, v);
  }
  total = __shfl_sync(0xffffffffu, v, (kUp ? 28 : 0) + (lane & 3));
  const float before = kUp ? __shfl_up_sync(0xffffffffu, v, 4) : __shfl_down_sync(0xffffffffu, v, 4);
  return at == 0 ? 0.f : before;
}

// kGroups: groups of 16 segments that a warp holds the states of
template <typename T, bool kBidir, bool kNorm, int kGroups>
__global__ void __launch_bounds__(kMaxThreads, 1) rowres_kernel(RowArgs a) {
  constexpr int kStateTiles = kBidir ? 4 : 2, kStateK = kBidir ? 2 : 1;
  extern __shared__ __align__(16) unsigned char smem[];
  const int L = a.L, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int team = w / a.warps, wr = w % a.warps;   // row of the CTA's, warp of the row's
  const int g = lane >> 2, t = lane & 3;
  const int nseg = (blockDim.x >> 5) * kGroups * 16;
  constexpr int rs = kGroups == 2 ? 2 : kGroups == 4 ? 3 : 4;   // log2 of the segments a lane holds
  using o = RowSmem<kBidir>;
  const int mine = team * a.warps * kGroups * 16;   // the row's first segment in the CTA's buffers
  float* xs = reinterpret_cast<float*>(smem + o::rows) + kSeg * mine;
  const unsigned char* fv = smem + o::frag;
  const unsigned char* ft = fv + 2 * kStateTiles * kBlockBytes;
  const unsigned char* fe = ft + 8 * kBlockBytes;
  const float* qt = reinterpret_cast<const float*>(smem + o::q);
  float* tot = reinterpret_cast<float*>(smem + o::tot) + 32 * team * a.warps;   // [warps][32]
  float* red = reinterpret_cast<float*>(smem + o::red) + 3 * team * a.warps;
  unsigned* masks = reinterpret_cast<unsigned*>(smem + o::mask(nseg)) + mine;   // two sets of nseg words
  const int teams = (blockDim.x >> 5) / a.warps, steps = (a.B + teams - 1) / teams;   // (of a channel)
  const long long units = (long long)a.D * steps;
  const int first = (int)(units * blockIdx.x / gridDim.x), last = (int)(units * (blockIdx.x + 1) / gridDim.x);
  int have = -1;
  unsigned next_any = 0u;
  bool next_live = false;

  for (int u = first - 1; u < last; ++u) {   // sequences of a channel follow each other: its matrices stay
    constexpr int segs = kGroups * 16;
    const int base = wr * segs;
    const unsigned any = next_any;
    const bool live = next_live;   // (states and outputs of nothing but padding come from the other warps alone)
    const int d = max(u, 0) / steps, b = max(u, 0) % steps * teams + team;
    const bool row = b < a.B;       // (else nothing to do but to keep the barriers)
    const T* xg = reinterpret_cast<const T*>(a.x) + b * a.xsb + d * a.xsd;
    T* yg = reinterpret_cast<T*>(a.y) + b * a.ysb + d * a.ysd;
    unsigned* mk = masks + (u & 1) * nseg;   // (the next row's is read while this row arrives)
    if (u >= first) {
      if (!kNorm || d != have) __syncthreads();   // (the row before is done with the tables and the warps' totals)
      if (d != have) prepare_channel<kBidir>(a, d, kGroups, smem);
      __syncwarp();   // (all lanes are done with the warp's segments of the row before)
      // ---- a warp loads, zeroes, normalises and emits the segments it owns
      if (live) load_x_row<T, rs>(xg, L, base, xs);
      if (sizeof(T) == 4) asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (u + 1 < last) {
      const int d1 = (u + 1) / steps, b1 = (u + 1) % steps * teams + team;
      unsigned all = ~0u;
      if (b1 < a.B)
        next_any = load_mask(a.mask ? a.mask + (size_t)b1 * L : nullptr, b1 == 0, L, base, segs, masks + ((u + 1) & 1) * nseg, all);
      next_live = all != ~0u;
      const int n = min(kSeg * segs, L - kSeg * base);
      if (lane == 0 && n > 0 && next_live) {
        const T* xn = reinterpret_cast<const T*>(a.x) + b1 * a.xsb + d1 * a.xsd + (long long)kSeg * base;
        const uintptr_t from = (reinterpret_cast<uintptr_t>(xn) + 15) & ~(uintptr_t)15, to = reinterpret_cast<uintptr_t>(xn + n) & ~(uintptr_t)15;
        if (to > from) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(from), "r"((unsigned)(to - from)) : "memory");
      }
    }
    if (u < first) continue;
    if (sizeof(T) == 4) asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (d != have) {
      __syncthreads();   // (the tables are complete)
      have = d;
    } else {
      __syncwarp();
    }

    float sc = 1.f, sh = 0.f;
    if (kNorm) {
      // one pass: mean and squared deviations of 32 positions at a time, merged
      Run r{0.f, 0.f, 0.f};
      auto moments = [&](auto masked) {
        constexpr bool kMasked = decltype(masked)::value;
        for (int k0 = 0; k0 < 4 * kGroups; k0 += 8) {
          float4 v[8];
          unsigned m[8];
          float n = 32.f, sum = 0.f, m2 = 0.f;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int i = (k0 + k) * 32 + lane;
            v[k] = *reinterpret_cast<const float4*>(xs + 4 * piece(base + (i >> 3), i & 7, rs));
            if (kMasked) {
              m[k] = (mk[base + (i >> 3)] >> (4 * (i & 7))) & 15u;
              v[k] = keep(v[k], m[k]);
              n -= (float)__popc(m[k]);
            }
            sum += (v[k].x + v[k].y) + (v[k].z + v[k].w);
          }
          const float c = n > 0.f ? sum / n : 0.f;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            float4 e = make_float4(v[k].x - c, v[k].y - c, v[k].z - c, v[k].w - c);
            if (kMasked) e = keep(e, m[k]);
            m2 = fmaf(e.x, e.x, m2); m2 = fmaf(e.y, e.y, m2); m2 = fmaf(e.z, e.z, m2); m2 = fmaf(e.w, e.w, m2);
          }
          r = combine(r, Run{n, c, m2});
        }
      };
      if (live && any) moments(std::true_type{});
      else if (live) moments(std::false_type{});
      r = row_run(r, red, wr, a.warps);
      const float cnt = r.n, mean = r.mean, var = cnt > 0.f ? r.m2 / cnt : 0.f;
      const float rstd = rsqrtf(var + a.eps);
      sc = rstd * __ldg(a.ngamma + d);
      sh = fmaf(-mean, sc, __ldg(a.nbeta + d));
      if (wr == 0 && lane == 0 && row) {
        const long long at = (long long)b * a.D + d;
        if (a.mean_out) a.mean_out[at] = mean;
        if (a.rstd_out) a.rstd_out[at] = rstd;
        if (a.count_out && d == 0) a.count_out[b] = (long long)(cnt + 0.5f);
      }
    }

    if (live && any) {   // normalised and zeroed ahead: the products take the values as they find them
      for (int k0 = 0; k0 < 4 * kGroups; k0 += 4) {
        float4 v[4];
        unsigned m[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int i = (k0 + k) * 32 + lane;
          v[k] = *reinterpret_cast<const float4*>(xs + 4 * piece(base + (i >> 3), i & 7, rs));
          m[k] = mk[base + (i >> 3)] >> (4 * (i & 7));
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int i = (k0 + k) * 32 + lane;
          if (kNorm) v[k] = make_float4(fmaf(v[k].x, sc, sh), fmaf(v[k].y, sc, sh), fmaf(v[k].z, sc, sh), fmaf(v[k].w, sc, sh));
          *reinterpret_cast<float4*>(xs + 4 * piece(base + (i >> 3), i & 7, rs)) = keep(v[k], m[k]);
        }
      }
      sc = 1.f;
      sh = 0.f;
      __syncwarp();
    }
    // the segments of a fragment's rows g and g + 8: a lane holds a run of 2 per_warp that follow each other
    auto seg_of = [&](int group, int h) { return base + (g << rs) + 2 * group + h; };
    // A fragments of 16 segments, positions 16 kt + 4 t .. + 3 of each
    auto load_x = [&](int group, int kt, uint32_t (&f)[3][4]) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float4 v = *reinterpret_cast<const float4*>(xs + 4 * piece(seg_of(group, h), 4 * kt + t, rs));
        if (kNorm) {
          v.x = fmaf(v.x, sc, sh); v.y = fmaf(v.y, sc, sh); v.z = fmaf(v.z, sc, sh); v.w = fmaf(v.w, sc, sh);
        }
        split3(v.x, v.y, f[0][h], f[1][h], f[2][h]);
        split3(v.z, v.w, f[0][2 + h], f[1][2 + h], f[2][2 + h]);
      }
    };

    // ---- 16 segments at a time: local states (column tile nt, rows g (st[..][nt][0, 1]) and g + 8 (2, 3), columns
    // 8 nt + 2 t, + 1), and the outputs of the inputs themselves in the inputs' place
    float st[kGroups][kStateTiles][4];
    const float om = __ldg(a.omega + d);
    if (live) {
#pragma unroll
      for (int gr = 0; gr < kGroups; ++gr) {
        __syncwarp();   // (keeps the groups apart: several at once do not fit in registers)
        uint32_t f[2][3][4];
        load_x(gr, 0, f[0]);
        load_x(gr, 1, f[1]);
        auto states = [&] {
#pragma unroll
          for (int nt = 0; nt < kStateTiles; ++nt) products<2, false>(st[gr][nt], f, fv + nt * kBlockBytes, kStateTiles * kBlockBytes);
        };
        // Causal rows: T's zeros do not keep a NaN or an infinity from the positions before it, and the products would make
        // up to 31 earlier outputs NaN.  A segment with one takes its outputs from the finite values alone, NaN from there
        // on; its state is NaN, as are all later ones.
        int bad[2] = {kSeg, kSeg};   // first such position of the lane's two segments
        bool odd = false;
        if constexpr (!kBidir && !kNorm) {
          states();
          unsigned e = 0u;   // bit 15 or 31: a leading part whose exponent is all ones
#pragma unroll
          for (int i = 0; i < 4; ++i) e |= ((f[0][0][i] & 0x7f807f80u) + 0x00800080u) | ((f[1][0][i] & 0x7f807f80u) + 0x00800080u);
          odd = __any_sync(0xffffffffu, (e & 0x80008000u) != 0u);
          if (odd) {
#pragma unroll
            for (int kt = 0; kt < 2; ++kt)
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const float4 v = *reinterpret_cast<const float4*>(xs + 4 * piece(seg_of(gr, h), 4 * kt + t, rs));
                float u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int c = 3; c >= 0; --c)
                  if (!(fabsf(u[c]) < 0x1.FFp127f)) {   // (from there on the leading part is an infinity)
                    bad[h] = min(bad[h], 16 * kt + 4 * t + c);
                    u[c] = 0.f;
                  }
                split3(u[0], u[1], f[kt][0][h], f[kt][1][h], f[kt][2][h]);
                split3(u[2], u[3], f[kt][0][2 + h], f[kt][1][2 + h], f[kt][2][2 + h]);
              }
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int s = 1; s < 4; s <<= 1) bad[h] = min(bad[h], __shfl_xor_sync(0xffffffffu, bad[h], s));
          }
        }
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float y[2][4];
          products<2, true>(y[0], f, ft + 2 * half * kBlockBytes, 4 * kBlockBytes);
          products<2, true>(y[1], f, ft + (2 * half + 1) * kBlockBytes, 4 * kBlockBytes);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float4* at = reinterpret_cast<float4*>(xs + 4 * piece(seg_of(gr, h), 4 * half + t, rs));
            float4 v = *at;
            if (kNorm) v = make_float4(fmaf(v.x, sc, sh), fmaf(v.y, sc, sh), fmaf(v.z, sc, sh), fmaf(v.w, sc, sh));
            float4 r = make_float4(fmaf(om, v.x, y[0][2 * h]), fmaf(om, v.y, y[0][2 * h + 1]), fmaf(om, v.z, y[1][2 * h]),
                                   fmaf(om, v.w, y[1][2 * h + 1]));
            if (!kBidir && !kNorm && odd) {
              const int p = 16 * half + 4 * t;
              const float nan = __int_as_float(0x7fffffff);
              r = make_float4(p < bad[h] ? r.x : nan, p + 1 < bad[h] ? r.y : nan, p + 2 < bad[h] ? r.z : nan, p + 3 < bad[h] ? r.w : nan);
            }
            *at = r;
          }
        }
        if constexpr (kBidir || kNorm) states();
      }
    } else {
#pragma unroll
      for (int gr = 0; gr < kGroups; ++gr)
#pragma unroll
        for (int nt = 0; nt < kStateTiles; ++nt) st[gr][nt][0] = st[gr][nt][1] = st[gr][nt][2] = st[gr][nt][3] = 0.f;
#pragma unroll 4
      for (int k = 0; k < 4 * kGroups; ++k) *reinterpret_cast<float4*>(xs + kSeg * base + 128 * k + 4 * lane) = make_float4(0.f, 0.f, 0.f, 0.f);
    }

    // ---- states that enter each segment: totals of the lanes' runs, scanned over lanes, then over warps, and the runs
    // again from what enters them
    float enter[kStateTiles][2];
#pragma unroll
    for (int nt = 0; nt < kStateTiles; ++nt) {
      float total[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        auto q = [&](int row) { return qt[row * 32 + 8 * nt + 2 * t + c]; };
        const float q1 = q(kQ1);
        float v = 0.f;
#pragma unroll
        for (int k = 0; k < 2 * kGroups; ++k) {
          const int at = nt < 2 ? k : 2 * kGroups - 1 - k;
          v = fmaf(q1, v, st[at >> 1][nt][2 * (at & 1) + c]);
        }
        enter[nt][c] = nt < 2 ? scan8<true>(v, q(kQRun + 1), q(kQRun + 2), q(kQRun + 4), total[c])
                              : scan8<false>(v, q(kQRun + 1), q(kQRun + 2), q(kQRun + 4), total[c]);
      }
      if (g == 0) *reinterpret_cast<float2*>(tot + wr * 32 + 8 * nt + 2 * t) = make_float2(total[0], total[1]);
    }
    __syncthreads();
#pragma unroll
    for (int nt = 0; nt < kStateTiles; ++nt) {
      const bool up = nt < 2;
      auto q2 = [&](int row) { return *reinterpret_cast<const float2*>(qt + row * 32 + 8 * nt + 2 * t); };
      const float2 q1 = q2(kQ1), qw = q2(kQRun + 8), qg = q2(kQRun + (up ? g : 7 - g));
      float2 c = make_float2(0.f, 0.f);
      for (int k = 0; k < (up ? wr : a.warps - 1 - wr); ++k) {
        const float2 v = *reinterpret_cast<const float2*>(tot + (up ? k : a.warps - 1 - k) * 32 + 8 * nt + 2 * t);
        c.x = fmaf(qw.x, c.x, v.x);
        c.y = fmaf(qw.y, c.y, v.y);
      }
      c.x = fmaf(qg.x, c.x, enter[nt][0]);
      c.y = fmaf(qg.y, c.y, enter[nt][1]);
#pragma unroll
      for (int k = 0; k < 2 * kGroups; ++k) {
        const int at = up ? k : 2 * kGroups - 1 - k;
        float &x = st[at >> 1][nt][2 * (at & 1)], &y = st[at >> 1][nt][2 * (at & 1) + 1];
        const float lx = x, ly = y;
        x = c.x;
        y = c.y;
        c.x = fmaf(q1.x, c.x, lx);
        c.y = fmaf(q1.y, c.y, ly);
      }
    }

    // ---- what the entering states add to the outputs; then the rows are stored.  (One form for all: a second one for
    // aligned rows without padding, storing from registers, gained 3 % where all warps took it and lost a third where
    // they did not, the code of both being too much for the instruction cache.)
#pragma unroll
    for (int gr = 0; gr < kGroups; ++gr) {
      __syncwarp();
      uint32_t f[kStateK][3][4];
#pragma unroll
      for (int kt = 0; kt < kStateK; ++kt)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float(&s)[4] = st[gr][2 * kt + h];
          split3(s[0], s[1], f[kt][0][2 * h], f[kt][1][2 * h], f[kt][2][2 * h]);
          split3(s[2], s[3], f[kt][0][2 * h + 1], f[kt][1][2 * h + 1], f[kt][2][2 * h + 1]);
        }
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        float y[2][4];
        products<kStateK, true>(y[0], f, fe + 2 * half * kBlockBytes, 4 * kBlockBytes);
        products<kStateK, true>(y[1], f, fe + (2 * half + 1) * kBlockBytes, 4 * kBlockBytes);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float4* at = reinterpret_cast<float4*>(xs + 4 * piece(seg_of(gr, h), 4 * half + t, rs));
          const float4 v = *at;
          *at = make_float4(v.x + y[0][2 * h], v.y + y[0][2 * h + 1], v.z + y[1][2 * h], v.w + y[1][2 * h + 1]);
        }
      }
    }
    __syncwarp();
    if (row) store_row<T, !kNorm, rs>(xs, mk, any, L, base, om, a.silu, xg, yg);
  }
}

template <typename T, bool kBidir, bool kNorm>
bool launch_rowres(RowArgs a, cudaStream_t s) {
  // warps of two groups of 16 segments (1024 positions) while four of them hold the row, of four groups (causal: up
  // to eight) beyond: more, smaller CTAs keep the SM busy across the load and store of each row
  constexpr int kMost = kBidir ? 4 : 8;
  const int pairs = (a.L + 1023) / 1024;
  int per = 2;
  if (pairs > 4) per = 4;
  if (per < kMost && pairs > 2 * (kMaxThreads / 32)) per = kMost;
  const int warps = (pairs + per / 2 - 1) / (per / 2);
  if (warps > kMaxThreads / 32) return false;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return false;
  // several rows of a channel per CTA, up to eight warps, while that leaves a CTA for every SM: its matrices (microseconds of
  // one warp) are prepared once for all
  int teams = std::max(1, std::min(8 / warps, a.B));
  while (teams > 1 && (long long)a.D * ((a.B + teams - 1) / teams) < sms) teams = (teams + 1) / 2;
  a.warps = warps;
  const int threads = 32 * warps * teams;
  const int smem = RowSmem<kBidir>::total(warps * teams * per * 16);
  if (smem > 220 * 1024) return false;
  const int by_smem = (227 * 1024) / (smem + 1024), by_regs = kMaxThreads / threads;   // (128 registers per thread)
  const int per_sm = std::max(1, std::min(by_smem, by_regs));
  const long long units = (long long)a.D * ((a.B + teams - 1) / teams);
  const unsigned grid = (unsigned)std::min<long long>(units, (long long)sms * per_sm);
  auto run = [&](auto kernel) { launch(kernel, dim3(grid), dim3(threads), (size_t)smem, (void*)s, a); };
  if (per == 2) run(rowres_kernel<T, kBidir, kNorm, 2>);
  else if (per == 4) run(rowres_kernel<T, kBidir, kNorm, 4>);
  else run(rowres_kernel<T, kBidir, kNorm, kMost>);
  g_last_kernel.store("rowres", std::memory_order_relaxed);
  return true;
}

}  // namespace

// Tries the row-resident path: length stride 1 on both tensors, ndim <= 16, no carried state, no
// truncation, the row fits in shared memory, at least 512 positions.
bool rowres_try(int dtype, const RowArgs& a, long long xsl, long long ysl, bool bidir, bool norm, cudaStream_t s) {
  if (g_options[OPT_DISABLE_STREAM].load() != 0) return false;
  if (xsl != 1 || ysl != 1 || a.N > kRowNP || a.L < 512 || a.L > 65535) return false;
  if ((long long)a.B * a.D > 0x7fffffffLL) return false;
  switch (dtype) {
#define MEGA_ROW_CASE(DT, TY)                                                                                       \
  case DT:                                                                                                          \
    return bidir ? (norm ? launch_rowres<TY, true, true>(a, s) : launch_rowres<TY, true, false>(a, s))              \
                 : (norm ? launch_rowres<TY, false, true>(a, s) : launch_rowres<TY, false, false>(a, s));
    MEGA_ROW_CASE(MEGA_F32, float)
    MEGA_ROW_CASE(MEGA_BF16, __nv_bfloat16)
    MEGA_ROW_CASE(MEGA_F16, __half)
#undef MEGA_ROW_CASE
    default: return false;
  }
}

}  // namespace mega

using namespace mega;

extern "C" MEGA_API int mega_sqn_ema_fwd(const void* x, void* y, int dtype, int B, int D, int L, int64_t xsb,
                                         int64_t xsd, int64_t xsl, int64_t ysb, int64_t ysd, int64_t ysl,
                                         const float* norm_gamma, const float* norm_beta, double eps,
                                         int64_t* count_out, float* mean_out, float* rstd_out, const float* p,
                                         const float* q, const float* gamma_hat, const float* omega, int N,
                                         const uint8_t* pad_mask, unsigned flags, mega_stream_t stream) {
  if (!x || !y || !norm_gamma || !norm_beta || !p || !q || !gamma_hat || !omega) return MEGA_ERR_NULL;
  if (!valid_dtype(dtype)) return MEGA_ERR_DTYPE;
  if (B <= 0 || D <= 0 || L <= 0) return MEGA_ERR_SHAPE;
  if (N < 1 || N > MEGA_MAX_NDIM) return MEGA_ERR_NDIM;
  if (!aligned_to(x, elem_size(dtype)) || !aligned_to(y, elem_size(dtype))) return MEGA_ERR_ALIGN;
  RowArgs a{};
  a.x = x; a.y = y; a.B = B; a.D = D; a.L = L; a.N = N;
  a.xsb = xsb; a.xsd = xsd; a.ysb = ysb; a.ysd = ysd;
  a.p = p; a.q = q; a.g = gamma_hat; a.omega = omega; a.mask = pad_mask;
  a.ngamma = norm_gamma; a.nbeta = norm_beta; a.eps = (float)eps;
  a.count_out = (long long*)count_out; a.mean_out = mean_out; a.rstd_out = rstd_out;
  a.shift = (flags & MEGA_EMA_NO_SHIFT) ? 0 : 1;
  a.silu = (flags & MEGA_EMA_SILU) ? 1 : 0;
  if (!rowres_try(dtype, a, xsl, ysl, (flags & MEGA_EMA_BIDIRECTIONAL) != 0, true, (cudaStream_t)stream))
    return MEGA_ERR_UNSUPPORTED;
  return check_launch("sqn_ema_fwd");
}
