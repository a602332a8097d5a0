// Shared device/host helpers for the mega_b200 kernels (sm_100a).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <initializer_list>
#include <utility>

#include "mega_b200.h"

namespace mega {

// ---- launch bookkeeping ---------------------------------------------------
extern std::atomic<uint64_t> g_launches;
extern thread_local char g_cuda_err[256];
extern std::atomic<int> g_options[8];
enum { OPT_DISABLE_STREAM = 0, OPT_DISABLE_MMA = 1, OPT_MMA_TILE = 2, OPT_WAIT_LIMIT = 3, OPT_WITHHOLD_LOAD = 4, OPT_SPLIT = 5, OPT_CHUNK = 6, OPT_CHUNK_STEPS = 7 };
// Name of the kernel family of the most recent launch (test aid): launch() sets "other", the
// launchers of the named families overwrite it right after.
extern std::atomic<const char*> g_last_kernel;
int check_launch(const char* what);

// Single-token step with N / 4 lanes per (sequence, channel) (csrc/fused.cu): TimestepNorm update
// when count is given, then the pole update; false (nothing launched) when N is not 4, 8, 16 or 32
// or a state / coefficient pointer is not 16-byte aligned.  `after`: launched as launch_after does.
bool step_lanes_try(int dtype, const void* x, void* y, void* xn_out, int B, int D, int N, const long long* count,
                    float* mean, float* var, const float* gamma, const float* beta, float eps, const float* p,
                    const float* q, const float* g, const float* omega, const float* h_in, float* h_out, int silu,
                    void* stream, long long* count_next = nullptr, bool after = false);

// Above the default 48 KB the dynamic shared-memory size is an opt-in attribute of the kernel ON THE CURRENT
// DEVICE; it is raised once per kernel and device (abi.cu), as setting it costs a microsecond or two of every launch.
void allow_smem(const void* kernel, size_t bytes);

template <typename... KArgs, typename... Args>
static inline void launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, void* stream,
                          Args... args) {
  if (smem > 48 * 1024) allow_smem(reinterpret_cast<const void*>(kernel), smem);
  kernel<<<grid, block, smem, (cudaStream_t)stream>>>(static_cast<KArgs>(args)...);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  g_last_kernel.store("other", std::memory_order_relaxed);
}

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// A launch that may begin before the one before it on the stream has ended: its kernel waits (pdl_wait) before it reads
// anything that launch, or any earlier one, writes, and lets its own successor begin (pdl_next) when that is safe.
template <typename... KArgs, typename... Args>
static inline void launch_after(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, void* stream, Args... args) {
  if (smem > 48 * 1024) allow_smem(reinterpret_cast<const void*>(kernel), smem);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  g_last_kernel.store("other", std::memory_order_relaxed);
}

// Zeroes `n` consecutive arrays of floats on the stream, as one piece where they lie side by side.
static inline bool zero_arrays(cudaStream_t s, std::initializer_list<std::pair<float*, size_t>> arrays) {
  float* at = nullptr;
  size_t len = 0;
  for (const auto& a : arrays) {
    if (at && at + len == a.first) {
      len += a.second;
      continue;
    }
    if (at && cudaMemsetAsync(at, 0, len * sizeof(float), s) != cudaSuccess) return false;
    at = a.first;
    len = a.second;
  }
  return !at || cudaMemsetAsync(at, 0, len * sizeof(float), s) == cudaSuccess;
}

// ---- element I/O ------------------------------------------------------------
template <typename T>
struct Elem;

// `ldv`: the same read-only load as `ld`, issued through a volatile asm statement so that the
// compiler keeps a batch of independent loads together at the top of an unrolled block instead
// of sinking each one to its use (kernels with few resident warps hide latency per thread).
template <>
struct Elem<float> {
  static __device__ __forceinline__ float ld(const float* p) { return __ldg(p); }
  static __device__ __forceinline__ float ldv(const float* p) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
  }
  static __device__ __forceinline__ float ld_shared(const float* p) { return *p; }
  static __device__ __forceinline__ void st(float* p, float v) { *p = v; }
};
template <>
struct Elem<__nv_bfloat16> {
  static __device__ __forceinline__ float ld(const __nv_bfloat16* p) {
    return __bfloat162float(__ldg(p));
  }
  static __device__ __forceinline__ float ldv(const __nv_bfloat16* p) {
    unsigned short v;
    asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return __uint_as_float((unsigned)v << 16);
  }
  static __device__ __forceinline__ float ld_shared(const __nv_bfloat16* p) { return __bfloat162float(*p); }
  static __device__ __forceinline__ void st(__nv_bfloat16* p, float v) {
    *p = __float2bfloat16_rn(v);
  }
};
template <>
struct Elem<__half> {
  static __device__ __forceinline__ float ld(const __half* p) { return __half2float(__ldg(p)); }
  static __device__ __forceinline__ float ldv(const __half* p) {
    unsigned short v;
    asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return __half2float(__ushort_as_half(v));
  }
  static __device__ __forceinline__ float ld_shared(const __half* p) { return __half2float(*p); }
  static __device__ __forceinline__ void st(__half* p, float v) { *p = __float2half_rn(v); }
};

// v, 0 where rounding took it below; NaN stays NaN (fmaxf would drop it)
__device__ __forceinline__ float not_negative(float v) { return v < 0.f ? 0.f : v; }
// MUFU approximations (about 1 ulp): no slow path, no subroutine call in a serial loop
__device__ __forceinline__ float rcp_approx(float v) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float rsqrt_approx(float v) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float sigmoidf_(float v) { return 1.0f / (1.0f + __expf(-v)); }
__device__ __forceinline__ float siluf_(float v) { return v / (1.0f + __expf(-v)); }
// sigmoid(v) to a few units of its last place, however nearly closed the gate: 0.5 + 0.5 tanh.approx(v / 2) is good to 2^-12
// of 1, which at v = -8 is most of the value.  fp32 activations take the full-range exponential and division, 16-bit ones
// two MUFU operations.
template <typename T>
__device__ __forceinline__ float exp_of(float v) {
  return sizeof(T) == 4 ? expf(v) : __expf(v);
}
template <typename T>
__device__ __forceinline__ float sigmoid_of(float v) {
  const float e = 1.f + exp_of<T>(-v);
  return sizeof(T) == 4 ? 1.f / e : rcp_approx(e);
}
// sigmoid(v) and sigmoid(-v)
struct Gate {
  float s, c;
};
template <typename T>
__device__ __forceinline__ Gate gate_of(float v) {
  const float e = exp_of<T>(-fabsf(v)), r = sizeof(T) == 4 ? 1.f / (1.f + e) : rcp_approx(1.f + e), l = e * r;
  return v >= 0.f ? Gate{r, l} : Gate{l, r};
}
// silu(v) = v * sigmoid(v) = h + h * tanh(h), h = v / 2: one MUFU op (tanh.approx, relative error
// about 2^-11) and two FP32 ops.  For kernels whose output is rounded to bf16 / fp16 anyway.
__device__ __forceinline__ float silu_tanh(float v) {
  const float h = 0.5f * v;
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(h));
  return fmaf(h, t, h);
}

static inline int elem_size(int dtype) { return dtype == MEGA_F32 ? 4 : 2; }

static inline bool valid_dtype(int dtype) {
  return dtype == MEGA_F32 || dtype == MEGA_BF16 || dtype == MEGA_F16;
}

static inline bool aligned_to(const void* p, size_t a) {
  return (reinterpret_cast<uintptr_t>(p) % a) == 0;
}

// Whether two arrays of n floats share memory (running statistics may be updated in place).
static inline bool overlap(const float* a, const float* b, size_t n) {
  const uintptr_t x = reinterpret_cast<uintptr_t>(a), y = reinterpret_cast<uintptr_t>(b), bytes = n * sizeof(float);
  return a != nullptr && b != nullptr && x < y + bytes && y < x + bytes;
}

static inline int next_pow2_ndim(int n) {
  int v = 2;
  while (v < n) v <<= 1;
  return v;
}

// Dispatch helpers: call f.template operator()<T>() for the activation dtype.
#define MEGA_DISPATCH_DTYPE(dtype, ...)                 \
  switch (dtype) {                                      \
    case MEGA_F32: { using T = float; __VA_ARGS__; } break;           \
    case MEGA_BF16: { using T = __nv_bfloat16; __VA_ARGS__; } break;  \
    case MEGA_F16: { using T = __half; __VA_ARGS__; } break;          \
    default: return MEGA_ERR_DTYPE;                     \
  }

#define MEGA_DISPATCH_NP(np, ...)                       \
  switch (np) {                                         \
    case 2: { constexpr int NP = 2; __VA_ARGS__; } break;   \
    case 4: { constexpr int NP = 4; __VA_ARGS__; } break;   \
    case 8: { constexpr int NP = 8; __VA_ARGS__; } break;   \
    case 16: { constexpr int NP = 16; __VA_ARGS__; } break; \
    case 32: { constexpr int NP = 32; __VA_ARGS__; } break; \
    default: return MEGA_ERR_NDIM;                      \
  }

}  // namespace mega
