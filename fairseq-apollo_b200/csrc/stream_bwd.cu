// Streamed backward of the per-feature TimestepNorm from statistics saved by its forward, for channel-contiguous
// activations ((B, L, D) memory).  Same data movement as the streamed forward kernels: a CTA owns kW adjacent channels of
// one sequence, tiles of kR timesteps arrive through a TMA ring (cp.async.bulk.tensor + mbarrier) and the input gradient
// leaves through TMA stores, so HBM sees whole row segments while every thread keeps its channel's recurrences in
// registers.  Time is walked backwards once.
#include <mutex>

#include "common.cuh"
#include "stream_bwd.cuh"
#include "tma.cuh"

namespace mega {

namespace {

constexpr int kW = 64;   // channels per CTA (= threads)
constexpr int kR = 32;   // timesteps per tile
constexpr int kS = 3;    // ring depth
constexpr int kHead = 512;

// ---------------------------------------------------------------------------------------------
// TimestepNorm
// ---------------------------------------------------------------------------------------------
template <typename T>
struct TsnCfg {
  static constexpr int kTileT = kR * kW * (int)sizeof(T);   // x, dy, dx
  static constexpr int kTileF = kR * kW * 4;                // cumrstd
  static constexpr int kTileM = (kR + 1) * kW * 4;          // cummean, with the row before the tile
  static constexpr int kStage = 2 * kTileT + kTileF + kTileM;
  static constexpr int kSmem = kHead + kS * kStage + 2 * kTileT + 128;
};

template <typename T, bool kMask>
__global__ void __launch_bounds__(kW) tsn_bwd_stream_kernel(const __grid_constant__ CUtensorMap tmx,
                                                            const __grid_constant__ CUtensorMap tmg,
                                                            const __grid_constant__ CUtensorMap tmd,
                                                            const __grid_constant__ CUtensorMap tmm,
                                                            const __grid_constant__ CUtensorMap tmr,
                                                            TsnBwdStreamArgs a) {
  using C = TsnCfg<T>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  float* cbuf = reinterpret_cast<float*>(base);                      // [2][kR] 1/count per row, < 0: padded
  uint64_t* full = reinterpret_cast<uint64_t*>(base + 2 * kR * 4);   // [kS]
  unsigned char* stages = base + kHead;
  T* outs = reinterpret_cast<T*>(base + kHead + kS * C::kStage);     // [2][kR][kW]

  const int tid = threadIdx.x;
  const int d0 = blockIdx.x * kW;
  const int b = blockIdx.y;
  const int d = d0 + tid;
  const bool valid = d < a.D;
  const int dc = valid ? d : a.D - 1;
  const int L = a.L;
  const int nt = (L + kR - 1) / kR;

  auto issue = [&](int k) {  // k-th tile in processing order = tile nt-1-k of the sequence
    const int s = k % kS, i = nt - 1 - k;
    unsigned char* st = stages + (size_t)s * C::kStage;
    mbar_expect_tx(&full[s], C::kStage);
    tma_load_3d(st, &tmx, d0, i * kR, b, &full[s]);
    tma_load_3d(st + C::kTileT, &tmg, d0, i * kR, b, &full[s]);
    tma_load_3d(st + 2 * C::kTileT, &tmr, d0, i * kR, b, &full[s]);
    tma_load_3d(st + 2 * C::kTileT + C::kTileF, &tmm, d0, i * kR - 1, b, &full[s]);
  };
  if (tid == 0) {
    prefetch_tensormap(&tmx);
    prefetch_tensormap(&tmg);
    prefetch_tensormap(&tmd);
    prefetch_tensormap(&tmm);
    prefetch_tensormap(&tmr);
#pragma unroll
    for (int s = 0; s < kS; ++s) mbar_init(&full[s], 1);
    mbar_fence_init();
  }
  __syncthreads();
  if (tid == 0)
    for (int k = 0; k < kS && k < nt; ++k) issue(k);

  const float w = __ldg(a.gamma + dc);
  const float pm = a.prev_mean[(size_t)b * a.D + dc];
  float ug = a.dmean ? a.dmean[(size_t)b * a.D + dc] : 0.f;
  float vg = a.dvar ? a.dvar[(size_t)b * a.D + dc] : 0.f;
  float wg = 0.f, bg = 0.f;

  // warp 0 walks the count backwards and publishes 1/count per row of the next tile
  long long cnt_run = a.count[b];
  const unsigned char* mrow = kMask ? a.mask + (size_t)b * L : nullptr;
  auto publish = [&](int k, unsigned char mk_byte) {
    const int i = nt - 1 - k;
    const int t = i * kR + tid;
    const bool masked = (t >= L) || (kMask && mk_byte != 0);
    const unsigned vmask = __ballot_sync(0xffffffffu, !masked);
    const unsigned later = tid == 31 ? 0u : (vmask & (0xffffffffu << (tid + 1)));
    const float cf = rcp_approx((float)(cnt_run - __popc(later)));
    cbuf[(k & 1) * kR + tid] = masked ? -1.0f : cf;
    cnt_run -= __popc(vmask);
  };
  if (tid < 32) {
    const int t = (nt - 1) * kR + tid;
    publish(0, (kMask && t < L) ? mrow[t] : 0);
  }
  __syncthreads();

  for (int k = 0; k < nt; ++k) {
    const int s = k % kS;
    const uint32_t ph = (uint32_t)((k / kS) & 1);
    const int i = nt - 1 - k;
    const int o = k & 1;
    unsigned char mb_next = 0;
    if (kMask && tid < 32 && k + 1 < nt) {
      const int t = (i - 1) * kR + tid;
      if (t < L) mb_next = mrow[t];
    }
    const bool ok = mbar_wait(&full[s], ph);
    const unsigned char* st = stages + (size_t)s * C::kStage;
    const T* xt = reinterpret_cast<const T*>(st) + tid;
    const T* gt = reinterpret_cast<const T*>(st + C::kTileT) + tid;
    const float* rt = reinterpret_cast<const float*>(st + 2 * C::kTileT) + tid;
    const float* mt = reinterpret_cast<const float*>(st + 2 * C::kTileT + C::kTileF) + tid;  // row r+1 = step r
    T* ot = outs + (size_t)o * kR * kW + tid;
    const float* cf = cbuf + o * kR;
    const int rows = min(kR, L - i * kR);
#pragma unroll 8
    for (int rr = 0; rr < kR; ++rr) {
      const int r = kR - 1 - rr;
      if (r < rows) {
        const float coef = cf[r];
        const bool mk = coef < 0.f;
        const float x = Elem<T>::ld_shared(xt + r * kW), dy = Elem<T>::ld_shared(gt + r * kW);
        const float u = mt[(r + 1) * kW], rs = rt[r * kW];
        const float pu = (i == 0 && r == 0) ? pm : mt[r * kW];
        const float dyr = dy * rs, delta = x - u, xp = x - pu;
        const float dv = vg - 0.5f * dy * w * delta * (rs * rs * rs);
        const float du = ug - (w * dyr + coef * dv * xp);
        const float dx = w * dyr + dv * coef * (delta + xp) + coef * du;
        Elem<T>::st(ot + r * kW, mk ? 0.f : dx);
        ug = mk ? ug : (1.f - coef) * du - coef * delta * dv;
        vg = mk ? vg : (1.f - coef) * dv;
        wg = mk ? wg : fmaf(dyr, delta, wg);
        bg = mk ? bg : bg + dy;
      }
    }
    if (tid < 32 && k + 1 < nt) publish(k + 1, mb_next);
    fence_proxy_async();
    if (tid == 0) bulk_wait_read<0>();
    if (__syncthreads_or(!ok)) break;
    if (tid == 0) {
      tma_store_3d(&tmd, d0, i * kR, b, outs + (size_t)o * kR * kW);
      bulk_commit();
      if (k + kS < nt) issue(k + kS);
    }
  }
  if (tid == 0) bulk_wait<0>();
  if (valid) {
    a.dprev_mean[(size_t)b * a.D + d] = ug;
    a.dprev_var[(size_t)b * a.D + d] = vg;
    atomicAdd(a.dgamma + d, wg);
    atomicAdd(a.dbeta + d, bg);
  }
}

template <typename K>
static bool set_smem(K kern, int bytes) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
}

}  // namespace

bool tsn_bwd_stream_try(int dtype, const void* dy, const void* x, void* dx, long long gsb, long long gsl,
                        long long gsd, long long xsb, long long xsl, long long xsd, long long dsb, long long dsl,
                        long long dsd, const float* cummean, const float* cumrstd, const TsnBwdStreamArgs& a,
                        cudaStream_t s) {
  if (g_options[OPT_DISABLE_STREAM].load() != 0) return false;
  if (gsd != 1 || xsd != 1 || dsd != 1 || a.B > 65535 || a.D < 8) return false;
  CUtensorMap tx, tg, td, tm, tr;
  if (!make_tensor_map_3d(&tx, dtype, x, a.D, a.L, a.B, xsl, xsb, kW, kR, 1, CU_TENSOR_MAP_SWIZZLE_NONE)) return false;
  if (!make_tensor_map_3d(&tg, dtype, dy, a.D, a.L, a.B, gsl, gsb, kW, kR, 1, CU_TENSOR_MAP_SWIZZLE_NONE)) return false;
  if (!make_tensor_map_3d(&td, dtype, dx, a.D, a.L, a.B, dsl, dsb, kW, kR, 1, CU_TENSOR_MAP_SWIZZLE_NONE)) return false;
  if (!make_tensor_map_3d(&tm, MEGA_F32, cummean, a.D, a.L, a.B, a.D, (long long)a.L * a.D, kW, kR + 1, 1,
                          CU_TENSOR_MAP_SWIZZLE_NONE))
    return false;
  if (!make_tensor_map_3d(&tr, MEGA_F32, cumrstd, a.D, a.L, a.B, a.D, (long long)a.L * a.D, kW, kR, 1,
                          CU_TENSOR_MAP_SWIZZLE_NONE))
    return false;
  dim3 grid((a.D + kW - 1) / kW, a.B);
  bool ok = true;
  switch (dtype) {
#define MEGA_TSN_BWD_CASE(DT, TY)                                                                  \
  case DT: {                                                                                       \
    static std::once_flag once;                                                                    \
    static bool attr_ok = true;                                                                    \
    std::call_once(once, [&] {                                                                     \
      attr_ok = set_smem(tsn_bwd_stream_kernel<TY, true>, TsnCfg<TY>::kSmem) &&                    \
                set_smem(tsn_bwd_stream_kernel<TY, false>, TsnCfg<TY>::kSmem);                     \
    });                                                                                            \
    if (!attr_ok) { cudaGetLastError(); return false; }                                            \
    if (a.mask) launch(tsn_bwd_stream_kernel<TY, true>, grid, dim3(kW), (size_t)TsnCfg<TY>::kSmem, (void*)s, tx, \
                       tg, td, tm, tr, a);                                                         \
    else launch(tsn_bwd_stream_kernel<TY, false>, grid, dim3(kW), (size_t)TsnCfg<TY>::kSmem, (void*)s, tx, tg, \
                td, tm, tr, a);                                                                    \
  } break;
    MEGA_TSN_BWD_CASE(MEGA_F32, float)
    MEGA_TSN_BWD_CASE(MEGA_BF16, __nv_bfloat16)
    MEGA_TSN_BWD_CASE(MEGA_F16, __half)
#undef MEGA_TSN_BWD_CASE
    default: ok = false;
  }
  return ok;
}

cudaError_t stream_bwd_read_device_error(int* v, bool reset) { return read_device_error(v, reset); }

}  // namespace mega
