// C ABI: global-scale INT8 products.
#include "launch_gemm.cuh"
#include "drivers.cuh"
#include "epi_int8.cuh"

using namespace i8m;

int i8m::i8_gemm(int mode, const int8_t* a, const int8_t* b, int b_mn, const int8_t* row_b, void* out, void* maximum,
                 const float* a_scale, const float* b_scale, const float* diag, int batch, int m, int n, int k, int lm, int ln,
                 float alpha, float beta, int final, int transpose, int out_dtype, unsigned* status, cudaStream_t stream) {
  if (!out) return fail(I8M_E_ARGUMENT, "i8_gemm: null output");
  I8Args g;
  g.out = out; g.maximum = maximum; g.a_scale = a_scale; g.b_scale = b_scale; g.diag = diag;
  g.row_b = row_b; g.alpha = alpha; g.beta = beta; g.out_dtype = out_dtype; g.transpose = transpose;
  g.gain = alpha; g.use_gain = mode == 4;
  GemmCall c;
  c.a = a; c.b = b; c.b_mn = b_mn; c.batch = batch; c.m = m; c.n = n; c.k = k; c.lm = lm; c.ln = ln;
  c.sym = mode < 2; c.status = status; c.stream = stream;
  if (mode == 4) mode = 2;   // update whose right-hand scale is multiplied by alpha
  if (mode == 0) {
    if (!maximum) return fail(I8M_E_ARGUMENT, "i8_gemm: gram needs a maximum slot");
    return launch_gemm<EpiI8<I8_GRAM>>(c, g, "i8_gemm(gram)");
  }
  if (mode == 1) {
    if (!maximum || !a_scale || !diag) return fail(I8M_E_ARGUMENT, "i8_gemm: square needs scale, diag, maximum");
    return launch_gemm<EpiI8<I8_SQUARE>>(c, g, "i8_gemm(square)");
  }
  if (mode == 2) {
    if (!a_scale || !b_scale || !diag || !row_b) return fail(I8M_E_ARGUMENT, "i8_gemm: update needs scales, diag, row_b");
    if (final) {
      if (!float_dtype_ok(out_dtype)) return fail(I8M_E_ARGUMENT, "i8_gemm: bad out_dtype");
      return launch_gemm<EpiI8<I8_UPDATE_FINAL>>(c, g, "i8_gemm(final update)");
    }
    if (!maximum) return fail(I8M_E_ARGUMENT, "i8_gemm: update needs a maximum slot");
    return launch_gemm<EpiI8<I8_UPDATE>>(c, g, "i8_gemm(update)");
  }
  return fail(I8M_E_ARGUMENT, "i8_gemm: bad mode %d", mode);
}
extern "C" int i8m_i8_gemm(int mode, const int8_t* a, const int8_t* b_t, const int8_t* row_b,
                           void* out, void* maximum, const float* a_scale, const float* b_scale,
                           const float* diag, int batch, int m, int n, int k, int lm, int ln,
                           float alpha, float beta, int final, int transpose, int out_dtype,
                           uint32_t* status, i8m_stream_t stream) {
  return i8_gemm(mode, a, b_t, 0, row_b, out, maximum, a_scale, b_scale, diag, batch, m, n, k, lm, ln, alpha, beta, final,
                 transpose, out_dtype, status, S(stream));
}
