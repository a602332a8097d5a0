// How the kernels that are parallel over time (scan_ema.cu, scan_norm.cu) read their inputs: a warp walks one
// segment of 32 adjacent channels, a lane one channel.
#pragma once
#include "common.cuh"
#include "tma.cuh"

namespace mega {

namespace {

constexpr int kWarps = 4;   // warps (segments) per block
constexpr int kU = 8;       // steps of an unrolled group

// ---- the inputs of a walk ----------------------------------------------------------------------------
// A warp fetches its 32 channels in tiles of 2 KB (32 steps of a 16-bit type, 16 of fp32) with 16-byte
// asynchronous copies into a ring of its own, kRing - 1 tiles ahead of their use: loads straight into registers,
// eight steps ahead, kept too few bytes in flight (0.6 TB/s on B = 8, L = 4096, D = 1024 bf16).  No barrier
// beyond the warp's is involved.
constexpr int kTileBytes = 2048;
constexpr int kRing = 4;

template <typename T, int kCh = 32>
__device__ __forceinline__ void fetch_tile(uint32_t dst, const T* row, long long stride, int rows, int d_left, int lane) {
  constexpr int kPer = kCh * (int)sizeof(T) / 16;   // 16-byte pieces of a row
#pragma unroll
  for (int i = 0; i < kTileBytes / 16 / 32; ++i) {
    const int id = lane + 32 * i;
    const int r = id / kPer, c = (id % kPer) * (16 / (int)sizeof(T));
    const bool in = r < rows && c < d_left;
    const T* src = in ? row + (long long)r * stride + c : row;
    const int bytes = in ? min(16, (d_left - c) * (int)sizeof(T)) : 0;   // (nothing behind the last channel is read)
    asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;" ::"r"(dst + id * 16), "l"(src), "r"(bytes) : "memory");
  }
}
__device__ __forceinline__ void tile_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void tile_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Walks the steps [t0, t1) of 32 channels in time order (kDir = 1) or reversed (-1); f(k, v, g, pad) sees step
// k = 0, 1, ... of that order.  x, g: first channel of the warp; ring: the warp's (two of them with kTwo).
template <typename T, int kDir, bool kTwo, bool kMask, typename F>
__device__ __forceinline__ void walk(const T* x, long long xsl, const T* g, long long gsl, const unsigned char* m, int t0,
                                     int t1, int d_left, unsigned char* ring, F&& f) {
  constexpr int kR = kTileBytes / (32 * (int)sizeof(T));
  const int lane = threadIdx.x & 31;
  const int n = t1 - t0;
  const int first = kDir > 0 ? t0 : t1 - 1;
  const T* px = x + (long long)first * xsl;
  const T* pg = kTwo ? g + (long long)first * gsl : nullptr;
  const long long dx = kDir > 0 ? xsl : -xsl, dg = kDir > 0 ? gsl : -gsl;
  const int tiles = (n + kR - 1) / kR;
  const uint32_t rs = smem_u32(ring);
  auto issue = [&](int j) {
    if (j < tiles) {
      const int slot = j % kRing;
      fetch_tile<T>(rs + slot * kTileBytes, px + (long long)(j * kR) * dx, dx, n - j * kR, d_left, lane);
      if (kTwo)
        fetch_tile<T>(rs + (kRing + slot) * kTileBytes, pg + (long long)(j * kR) * dg, dg, n - j * kR, d_left, lane);
    }
    tile_commit();
  };
  auto flags = [&](int j) -> unsigned {   // bit r: step r of tile j is padded
    if (!kMask) return 0u;
    const int k = j * kR + lane;
    const bool pad = lane < kR && k < n && __ldg(m + first + kDir * k) != 0;
    return __ballot_sync(0xffffffffu, pad);
  };
  __syncwarp();   // (the walk before has read the last tiles of the ring)
#pragma unroll
  for (int j = 0; j < kRing - 1; ++j) issue(j);
  unsigned next = flags(0);
  for (int j = 0; j < tiles; ++j) {
    tile_wait<kRing - 2>();
    __syncwarp();
    issue(j + kRing - 1);
    const unsigned bits = next;
    if (j + 1 < tiles) next = flags(j + 1);
    const T* tx = reinterpret_cast<const T*>(ring + (j % kRing) * kTileBytes) + lane;
    const T* tg = reinterpret_cast<const T*>(ring + (kRing + j % kRing) * kTileBytes) + lane;
    const int rows = min(kR, n - j * kR);
    int r0 = 0;
    for (; r0 + kU <= rows; r0 += kU) {
#pragma unroll
      for (int u = 0; u < kU; ++u)
        f(j * kR + r0 + u, Elem<T>::ld_shared(tx + (r0 + u) * 32), kTwo ? Elem<T>::ld_shared(tg + (r0 + u) * 32) : 0.f,
          kMask && ((bits >> (r0 + u)) & 1u) != 0);
    }
    for (; r0 < rows; ++r0)
      f(j * kR + r0, Elem<T>::ld_shared(tx + r0 * 32), kTwo ? Elem<T>::ld_shared(tg + r0 * 32) : 0.f,
        kMask && ((bits >> r0) & 1u) != 0);
  }
  tile_wait<0>();
}

// ---- two adjacent channels per lane, in packed fp32 arithmetic: half the instructions per element ------------
template <typename T>
__device__ __forceinline__ f32x2 pair_ld(const T* p) {   // (shared memory)
  if constexpr (sizeof(T) == 4) {
    return *reinterpret_cast<const f32x2*>(p);
  } else {
    const uint32_t v = *reinterpret_cast<const uint32_t*>(p);
    return pack2(Elem<T>::ld_shared(reinterpret_cast<const T*>(&v)), Elem<T>::ld_shared(reinterpret_cast<const T*>(&v) + 1));
  }
}
template <typename T>
__device__ __forceinline__ void pair_st(T* p, f32x2 v) {
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<f32x2*>(p) = v;
  } else {
    float lo, hi;
    unpack2(v, lo, hi);
    uint32_t w;
    Elem<T>::st(reinterpret_cast<T*>(&w), lo);
    Elem<T>::st(reinterpret_cast<T*>(&w) + 1, hi);
    *reinterpret_cast<uint32_t*>(p) = w;
  }
}

// walk() in time order for 64 channels, rings of kSlots tiles: f(v, g, pad) sees the pairs of every step.
template <typename T, bool kTwo, bool kMask, int kSlots = kRing, typename F>
__device__ __forceinline__ void walk_pairs(const T* x, long long xsl, const T* g, long long gsl, const unsigned char* m, int t0, int t1,
                                           int d_left, unsigned char* ring, F&& f) {
  constexpr int kR = kTileBytes / (64 * (int)sizeof(T));
  const int lane = threadIdx.x & 31, n = t1 - t0, tiles = (n + kR - 1) / kR;
  const T* px = x + (long long)t0 * xsl;
  const T* pg = kTwo ? g + (long long)t0 * gsl : nullptr;
  const uint32_t rs = smem_u32(ring);
  auto issue = [&](int j) {
    if (j < tiles) {
      const int slot = j % kSlots;
      fetch_tile<T, 64>(rs + slot * kTileBytes, px + (long long)(j * kR) * xsl, xsl, n - j * kR, d_left, lane);
      if (kTwo) fetch_tile<T, 64>(rs + (kSlots + slot) * kTileBytes, pg + (long long)(j * kR) * gsl, gsl, n - j * kR, d_left, lane);
    }
    tile_commit();
  };
  auto flags = [&](int j) -> unsigned {   // bit r: step r of tile j is padded
    if (!kMask) return 0u;
    const int k = j * kR + lane;
    return __ballot_sync(0xffffffffu, lane < kR && k < n && __ldg(m + t0 + k) != 0);
  };
#pragma unroll
  for (int j = 0; j < kSlots - 1; ++j) issue(j);
  unsigned next = flags(0);
  for (int j = 0; j < tiles; ++j) {
    tile_wait<kSlots - 2>();
    __syncwarp();
    issue(j + kSlots - 1);
    const unsigned bits = next;
    if (j + 1 < tiles) next = flags(j + 1);
    const T* tx = reinterpret_cast<const T*>(ring + (j % kSlots) * kTileBytes) + 2 * lane;
    const T* tg = reinterpret_cast<const T*>(ring + (kSlots + j % kSlots) * kTileBytes) + 2 * lane;
    const int rows = min(kR, n - j * kR);
    int r0 = 0;
    for (; r0 + kU <= rows; r0 += kU) {
#pragma unroll
      for (int u = 0; u < kU; ++u)
        f(pair_ld(tx + (r0 + u) * 64), kTwo ? pair_ld(tg + (r0 + u) * 64) : 0ull, kMask && ((bits >> (r0 + u)) & 1u) != 0);
    }
    for (; r0 < rows; ++r0) f(pair_ld(tx + r0 * 64), kTwo ? pair_ld(tg + r0 * 64) : 0ull, kMask && ((bits >> r0) & 1u) != 0);
  }
  tile_wait<0>();
}

}  // namespace

// channels contiguous, rows that start at 16-byte boundaries
static inline bool rows_ok(int dtype, const void* p, long long sb, long long sl, long long sd) {
  const long long es = elem_size(dtype);
  return sd == 1 && aligned_to(p, 16) && (sb * es) % 16 == 0 && (sl * es) % 16 == 0;
}
// ... and are whole 16-byte pieces (where a lane takes two channels)
static inline bool pieces_ok(int dtype, int D) { return (D * elem_size(dtype)) % 16 == 0; }

}  // namespace mega
