// Single-token step of TimestepNorm -> complex EMA as block_step.cu launches it (cema.cu); false (nothing launched)
// for pole counts other than 2, 4, 8, 16, 32 or unaligned states.
#pragma once
namespace mega {
bool cema_step_lanes_try(int dtype, const void* x, void* y, void* xn_out, int B, int D, int N, const long long* count,
                         float* mean, float* var, const float* gamma, const float* beta, float eps, const float* p,
                         const float* q, const float* g, const float* omega, const float* h_in, float* h_out, int silu,
                         void* stream, long long* count_next, bool after = false);
}  // namespace mega
