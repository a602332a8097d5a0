// TimestepNorm -> causal EMA in forms that are parallel over time (norm_ema_split.cu).
#pragma once
#include <cuda_runtime.h>

#include "stream_cl.cuh"

namespace mega {

// Runs the call in one of those forms when that is estimated to be faster than the fused kernels, which walk every
// sequence as one chain.  False (nothing launched) otherwise or outside the operators' envelopes.
bool norm_ema_split_try(int dtype, const void* x, void* y, void* xn, long long xsb, long long xsl, long long xsd,
                        long long ysb, long long ysl, long long ysd, const StreamArgs& a, cudaStream_t s);

}  // namespace mega
