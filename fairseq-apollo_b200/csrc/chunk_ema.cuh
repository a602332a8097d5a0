// Interface of the causal EMA as matrix products of chunks, parallel over time (chunk_ema.cu).
#pragma once
#include <cuda_runtime.h>

#include "scan_ema.cuh"

namespace mega {

// Each returns false, having launched nothing, outside its envelope (causal, no norm in front, ndim <= 16, channels
// contiguous in whole 16-byte pieces on every tensor), when another form is predicted to be faster, or without scratch memory.
// Forward: x of type dtype, y of type out_dtype (the same, or, without a mask, x in fp32 and y of 16 bits); x may be y where the types are the
// same.  Backward: a.y is dx, which is neither x nor dy.
// asked: whatever the prediction says.
bool chunk_ema_fwd_try(int dtype, int out_dtype, const ScanArgs& a, long long xsd, long long ysd, cudaStream_t s, bool asked = false);
double chunk_ema_fwd_us(int dtype, const ScanArgs& a);   // predicted time, 1e30 outside the envelope
bool chunk_ema_bwd_try(int dtype, const ScanArgs& a, long long xsd, long long ysd, long long gsd, cudaStream_t s);

}  // namespace mega
