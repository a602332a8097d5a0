// Interface of the EMA kernels that are parallel over time (scan_ema.cu): channel-contiguous activations.
#pragma once
#include <cuda_runtime.h>

namespace mega {

struct ScanArgs {
  const void* x;
  void* y;          // forward: output
  const void* dy;   // backward: output gradient; y is then the input gradient
  int B, D, L, N;
  long long xsb, xsl, ysb, ysl, gsb, gsl;
  const float *p, *q, *g, *omega;    // (K, N) rows, K = D or 2D; complex: q, g interleaved (re, im)
  const unsigned char* mask;         // (B, L) or null
  const float* h_in;                 // (B, D, N[, 2]) or null, causal only
  float* h_out;
  int cplx, bidir, shift, silu;
  float *dp, *dq, *dg, *domega;      // backward: zeroed accumulators
  // TimestepNorm in front of a causal forward (prev_count not null); xn: its output, strided like y, or null
  const long long* prev_count;
  const float *prev_mean, *prev_var, *gamma, *beta;
  float eps;
  long long* count_out;
  float *mean_out, *var_out;
  void* xn;
};

// Each returns false, having launched nothing, outside its envelope (channel stride other than 1, inputs whose rows
// do not start at 16-byte boundaries (behind a norm: are not whole 16-byte pieces), ndim > 16, too many sequences for the grid) or when there is no scratch memory.
// The forward may run in place (x == y, same strides): a warp reads its rows ahead of where it writes them.
bool scan_ema_fwd_ok(int dtype, const ScanArgs& a, long long xsd, long long ysd);   // the envelope alone
bool scan_ema_fwd_try(int dtype, const ScanArgs& a, long long xsd, long long ysd, cudaStream_t s);
double scan_ema_fwd_us(const ScanArgs& a);   // predicted time of the scan's launches, causal, no norm in front
bool scan_ema_bwd_try(int dtype, const ScanArgs& a, long long xsd, long long ysd, long long gsd, cudaStream_t s);

}  // namespace mega
