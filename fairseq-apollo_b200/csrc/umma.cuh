// tcgen05 (tensor memory, tensor-core products issued by one thread) for sm_100a: the few forms that are used here.
//
// Operands in shared memory are stored without swizzle: eight rows of 16 bytes are a core matrix of 128 contiguous bytes.  K-major
// (a row's 16 bytes are eight consecutive k): `lead` is the distance of core matrices that follow each other in k, `stride` of
// those that follow in m or n.  MN-major (the 16 bytes are eight consecutive m, a core matrix's rows are eight consecutive k): the
// same two distances, lead in k and stride in m.
#pragma once
#include <stdint.h>

namespace mega {

__device__ __forceinline__ uint64_t umma_desc(uint32_t at, uint32_t lead, uint32_t stride) {
  return (uint64_t)((at >> 4) & 0x3fffu) | ((uint64_t)(lead >> 4) << 16) | ((uint64_t)(stride >> 4) << 32) | (1ull << 46);
}
// bf16 operands, fp32 sums; a_mn: A is MN-major
__host__ __device__ constexpr uint32_t umma_idesc(int m, int n, bool a_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn ? 1u : 0u) << 15) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
// one lane of a warp that is here as a whole (so chosen, its products are issued from uniform registers: four times as fast)
__device__ __forceinline__ bool umma_elect() {
  uint32_t one;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
  return one != 0;
}
// d (+)= a b for k = 16
__device__ __forceinline__ void umma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool onto) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
               "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)onto)
               : "memory");
}
// d = a b, of which rows 16 j to 16 j + 15 alone are written; a from shared memory, or from tensor memory
#define MEGA_UMMA_16_ROWS(A, TY)                                                                                                       \
  const uint32_t off = j & 1 ? 0x0000ffffu : 0xffff0000u; /* (a bit per row: not written) */                                           \
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, 0, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], " A ", %2, %3, {%4, %5, %6, %7}, p;\n\t}" \
               ::"r"(d), TY(a), "l"(b), "r"(idesc), "r"(j >> 1 == 0 ? off : ~0u), "r"(j >> 1 == 1 ? off : ~0u),                        \
               "r"(j >> 1 == 2 ? off : ~0u), "r"(j >> 1 == 3 ? off : ~0u)                                                              \
               : "memory")
__device__ __forceinline__ void umma_16_rows(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, int j) { MEGA_UMMA_16_ROWS("%1", "l"); }
__device__ __forceinline__ void umma_16_rows(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, int j) { MEGA_UMMA_16_ROWS("[%1]", "r"); }
#undef MEGA_UMMA_16_ROWS
// the barrier completes when all products issued so far by this thread have
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tm_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tm_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tm_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tm_alloc(uint32_t to, int columns) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(to), "r"(columns) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tm_free(uint32_t at, int columns) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(at), "r"(columns) : "memory");
}
__device__ __forceinline__ void tm_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tm_st8(uint32_t at, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(at), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
// lane i of a warp: row i of its quarter, consecutive columns
__device__ __forceinline__ void tm_ld2(uint32_t at, float* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "r"(at) : "memory");
}
__device__ __forceinline__ void tm_ld32(uint32_t at, float* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
      "%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]),
        "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]), "=f"(v[16]), "=f"(v[17]), "=f"(v[18]),
        "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]), "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]),
        "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
      : "r"(at)
      : "memory");
}
}  // namespace mega
