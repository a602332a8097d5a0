// Interface of the EMA layer in one launch (scan_cluster.cu): channel-contiguous activations, sequences that fit the
// shared memory of a cluster.
#pragma once
#include <cuda_runtime.h>

#include "scan_ema.cuh"

namespace mega {

// Predicted time, 1e30 where the three launches of scan_ema.cu do as well or the sequence does not fit.
double scan_cluster_us(int dtype, const ScanArgs& a);
// For calls inside the envelope of scan_ema_fwd_ok.  Returns false, having launched nothing, when not predicted to pay.
bool scan_cluster_try(int dtype, const ScanArgs& a, cudaStream_t s);

// The layer by itself, bf16, causal: whether one launch of this kernel is predicted to beat the tensor-core kernel, which
// walks a sequence as one chain of steps.
bool scan_cluster_first(int dtype, const ScanArgs& a, long long xsd, long long ysd);

}  // namespace mega
