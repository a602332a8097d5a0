// Interface of the per-feature norms that are parallel over time (scan_norm.cu).
#pragma once
#include <cuda_runtime.h>

namespace mega {

struct ScanNormArgs {
  const void* x;
  void* y;          // forward: output; backward: input gradient
  float* wide;      // forward: the output in fp32 too, dense (B, L, D), or null; y may then be null
  const void* dy;
  int B, D, L;
  long long xsb, xsl, ysb, ysl, gsb, gsl;
  const long long* prev_count;
  const float *prev_mean, *prev_var;   // (B, D)
  const float *gamma, *beta;
  const unsigned char* mask;           // (B, L) or null
  float eps;
  long long* count_out;                // forward
  float *mean_out, *var_out;
  const float *dmean, *dvar;           // backward: gradients of the returned statistics, or null
  float *dprev_mean, *dprev_var, *dgamma, *dbeta;
};

// Each returns false, having launched nothing, outside its envelope (channels not contiguous, rows that are not
// whole 16-byte pieces, too many sequences for the grid, statistics updated in place) or when there is no scratch memory.
bool scan_norm_fwd_try(int dtype, const ScanNormArgs& a, long long xsd, long long ysd, cudaStream_t s);
double scan_norm_us(const ScanNormArgs& a);   // of the forward
bool stats_in_place(const ScanNormArgs& a);   // whether the new statistics go where the incoming ones are
bool scan_norm_bwd_try(int dtype, const ScanNormArgs& a, long long xsd, long long ysd, long long gsd, cudaStream_t s);

// Per-channel SequenceNorm: var_out receives rstd; the backward takes the forward's count, mean and rstd as
// prev_count, prev_mean and prev_var.
bool scan_sqn_fwd_try(int dtype, const ScanNormArgs& a, long long xsd, long long ysd, cudaStream_t s);
bool scan_sqn_bwd_try(int dtype, const ScanNormArgs& a, long long xsd, long long ysd, long long gsd, cudaStream_t s);

}  // namespace mega
