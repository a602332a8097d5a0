// fp32 contractions on the bf16 tensor pipe: a float is exactly the sum of three bf16 values (rowres.cu, chunk_ema.cu).
#pragma once
#include "common.cuh"
#include "tma.cuh"

namespace mega {

namespace {

constexpr int kBlockBytes = 32 * 24;   // a B fragment (16 x 8) in three bf16 parts: uint4 and uint2 per lane

__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
// two floats as three packed bf16 pairs whose sums they are
__device__ __forceinline__ void split3(float lo, float hi, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
  const f32x2 minus = pack2(-1.f, -1.f);
  f32x2 v = pack2(lo, hi);
  p0 = bf16_pair(lo, hi);
  v = fma2(pack2(__uint_as_float(p0 << 16), __uint_as_float(p0 & 0xffff0000u)), minus, v);
  unpack2(v, lo, hi);
  p1 = bf16_pair(lo, hi);
  v = fma2(pack2(__uint_as_float(p1 << 16), __uint_as_float(p1 & 0xffff0000u)), minus, v);
  unpack2(v, lo, hi);
  p2 = bf16_pair(lo, hi);
}

__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// the same onto zero: the product alone
__device__ __forceinline__ void mma0(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

struct Frag {   // B fragment: parts 0 and 1 in u, part 2 in v
  uint4 u;
  uint2 v;
};
__device__ __forceinline__ Frag load_frag(const unsigned char* block) {
  const int lane = threadIdx.x & 31;
  return {*reinterpret_cast<const uint4*>(block + lane * 16), *reinterpret_cast<const uint2*>(block + 512 + lane * 8)};
}
// a lane's entries of a B fragment: rows 2t, 2t + 1, 2t + 8, 2t + 9 of its column
__device__ __forceinline__ void store_frag(unsigned char* block, const float (&v)[4]) {
  const int lane = threadIdx.x & 31;
  uint32_t lo[3], hi[3];
  split3(v[0], v[1], lo[0], lo[1], lo[2]);
  split3(v[2], v[3], hi[0], hi[1], hi[2]);
  *reinterpret_cast<uint4*>(block + lane * 16) = make_uint4(lo[0], hi[0], lo[1], hi[1]);
  *reinterpret_cast<uint2*>(block + 512 + lane * 8) = make_uint2(lo[2], hi[2]);
}

}  // namespace

}  // namespace mega
