// What the whole-call drivers launch beyond the C ABI's own entry points.
#pragma once
#include <cuda_runtime.h>

namespace i8m {
// out = left * right^T with the epilogues of i8m_float_gemm; an operand with its _mn flag set is stored with its
// rows along K, (batch, k, m) or (batch, k, n), instead of (batch, m, k) or (batch, n, k).
struct FloatGemm {
  const void *left, *left_lo, *right, *right_lo;
  void *out, *out_t, *out_lo, *out_t_lo;
  int compute, mode, batch, m, n, k, lm, ln;
  int symmetric, final, transpose, out_dtype;
  int left_mn, right_mn;
  float ca, cb, cc;
  float* amax;     // final products, optional: [batch] maximum magnitude of the stored values (zeroed by the caller)
  unsigned* status;
  cudaStream_t stream;
};
int float_gemm(const FloatGemm& g);
int float_gemm_to_bq(const void* left, const void* right, int right_mn, void* q, void* q_t, float* scale, int compute,
                     int user_dtype, int batch, int m, int n, int k, int lm, int ln, int lp, int hp, unsigned* status,
                     cudaStream_t stream);
// i8m_i8_gemm whose right operand may be stored with its rows along K, (batch, k, n) (b_mn set)
int i8_gemm(int mode, const signed char* a, const signed char* b, int b_mn, const signed char* row_b, void* out, void* maximum,
            const float* a_scale, const float* b_scale, const float* diag, int batch, int m, int n, int k, int lm, int ln,
            float alpha, float beta, int final, int transpose, int out_dtype, unsigned* status, cudaStream_t stream);
// i8m_input_quant and i8m_output_quant without the transposed copy
int input_quant(const void* x, int in_dtype, const float* amax, const float* norm, signed char* a8, float* a_scale, int batch,
                int rows, int cols, int lp, int hp, int transpose, float eps, cudaStream_t stream);
int output_quant(const float* input, const float* maximum, signed char* out, float* scale, int batch, int m, int n,
                 cudaStream_t stream);
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
