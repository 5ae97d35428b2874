// Passes that only the whole-call drivers launch.
#pragma once
#include <cuda_runtime.h>

namespace i8m {
// final fold of per-chunk partials (i8m_stats layout) into norm[b] and amax[b]; either may be null
int fold_stats(const float* partials, int batch, long long count, float* norm, float* amax, cudaStream_t stream);
// r[b][i][i] += shift for i < logical, r (batch, m, m) in a 16-bit compute type
int add_diagonal(void* r, int compute, int batch, int m, int logical, float shift, cudaStream_t stream);
// norm[b] <- max(norm[b], eps) / gain
int clamp_divide(float* norm, int batch, float eps, float gain, cudaStream_t stream);
// i8m_apply that can also copy the status word to pinned host memory (both pointers null: it does not)
int apply_updates(void* const* params, int count, const void* update, long long numel, int param_dtype,
                  int update_dtype, int decay_mode, float decay, float neg_lr, const unsigned* status,
                  unsigned* status_host, cudaStream_t stream);
}  // namespace i8m
