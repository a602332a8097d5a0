// Interface of the fused TimestepNorm -> EMA kernel with accumulators in tensor memory (tmem_ema.cu).
#pragma once
#include <cuda_runtime.h>

#include "stream_cl.cuh"

namespace mega {

// bf16, channel stride 1 (whole 16-byte pieces), real poles, ndim <= 16, L a multiple of 16 where a state is exported.  Without norm the
// EMA by itself, no mask.  False, nothing launched, outside of that.  asked: 4 or 9, 10, 12, 16: blocks of four sequences, or of eight in 1, 2, 4, 8 runs along time that different blocks take one after the other (0: as
// estimated).
bool tmem_ema_try(int dtype, const void* x, void* y, void* xn, long long xsb, long long xsl, long long ysb, long long ysl, bool norm,
                  const StreamArgs& a, cudaStream_t s, int asked = 0);
// Its estimated time.
double tmem_ema_us(const StreamArgs& a, bool norm, bool xn);
// TimestepNorm by itself in the same way (bf16, x and y distinct), and its estimated time.
bool tmem_norm_try(int dtype, const void* x, void* y, long long xsb, long long xsl, long long ysb, long long ysl, const StreamArgs& a,
                   cudaStream_t s);
double tmem_norm_us(const StreamArgs& a);
cudaError_t tmem_ema_read_device_error(int* v, bool reset);

}  // namespace mega
