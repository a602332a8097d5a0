// The library's scratch pool (scratch.cuh).
#include <mutex>

#include "scratch.cuh"

namespace mega {

static cudaMemPool_t scratch_pool() {
  constexpr int kDevs = 16;
  static std::mutex mutex;
  static cudaMemPool_t pools[kDevs] = {};
  static bool tried[kDevs] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevs) return nullptr;
  std::lock_guard<std::mutex> lock(mutex);
  if (!tried[dev]) {
    tried[dev] = true;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;   // (the only kind: device memory that stays in place)
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t p = nullptr;
    if (cudaMemPoolCreate(&p, &props) == cudaSuccess) {
      unsigned long long keep = kScratchKept;
      cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
      pools[dev] = p;
    }
    cudaGetLastError();
  }
  return pools[dev];
}

void* scratch_alloc(size_t bytes, cudaStream_t s) {
  cudaMemPool_t pool = scratch_pool();
  void* p = nullptr;
  if (pool == nullptr || cudaMallocFromPoolAsync(&p, bytes ? bytes : 1, pool, s) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return p;
}

void scratch_free(void* p, cudaStream_t s) {
  if (cudaFreeAsync(p, s) != cudaSuccess) cudaGetLastError();
}

}  // namespace mega
