// C ABI: block-quantised products.
#include "launch_gemm.cuh"
#include "epi_bq.cuh"

using namespace i8m;

template <bool FP8>
static int bq_gemm_typed(int mode, const void* a, const float* sa, const float* da, const void* b_t,
                         const float* sb, const void* row_b, void* out, void* out_t, float* so,
                         float* dout, int batch, int m, int n, int k, int lm, int ln, float ca,
                         float cb, float cc, int final, int transpose, int out_dtype,
                         unsigned* status, cudaStream_t stream) {
  BqArgs g;
  g.sa = sa; g.sb = sb; g.da = da; g.row_b = static_cast<const uint8_t*>(row_b);
  g.out = out; g.out_t = out_t; g.so = so; g.dout = dout;
  g.ca = ca; g.cb = cb; g.cc = cc; g.out_dtype = out_dtype; g.transpose = transpose;
  if (mode == 0) {
    if (!so || !dout) return fail(I8M_E_ARGUMENT, "bq_gemm: gram needs scale and diagonal outputs");
    return launch_bq<EpiBq<FP8, BQ_GRAM>>(a, b_t, batch, m, n, k, lm, ln, 1, status, g, stream, "bq_gemm(gram)");
  }
  if (mode == 1) {
    if (!so || !dout || !da) return fail(I8M_E_ARGUMENT, "bq_gemm: poly needs scale, diagonal in and out");
    return launch_bq<EpiBq<FP8, BQ_POLY>>(a, b_t, batch, m, n, k, lm, ln, 1, status, g, stream, "bq_gemm(poly)");
  }
  if (mode == 2) {
    if (!da || !row_b) return fail(I8M_E_ARGUMENT, "bq_gemm: update needs the diagonal and row_b");
    if (final) {
      if (!float_dtype_ok(out_dtype)) return fail(I8M_E_ARGUMENT, "bq_gemm: bad out_dtype");
      return launch_bq<EpiBq<FP8, BQ_UPDATE_FINAL>>(a, b_t, batch, m, n, k, lm, ln, 0, status, g, stream,
                                                   "bq_gemm(final update)");
    }
    if (!so || !out_t) return fail(I8M_E_ARGUMENT, "bq_gemm: update needs scale and transposed outputs");
    return launch_bq<EpiBq<FP8, BQ_UPDATE>>(a, b_t, batch, m, n, k, lm, ln, 0, status, g, stream, "bq_gemm(update)");
  }
  return fail(I8M_E_ARGUMENT, "bq_gemm: bad mode %d", mode);
}

extern "C" int i8m_bq_gemm(int fp8, int mode, const void* a, const float* sa, const float* da,
                           const void* b_t, const float* sb, const void* row_b, void* out,
                           void* out_t, float* so, float* dout, int batch, int m, int n, int k,
                           int lm, int ln, float ca, float cb, float cc, int final, int transpose,
                           int out_dtype, uint32_t* status, i8m_stream_t stream) {
  if (!out || !sa || !sb) return fail(I8M_E_ARGUMENT, "bq_gemm: null pointer");
  if (m % 128 || n % 128 || k % 128) return fail(I8M_E_ARGUMENT, "bq_gemm: extents must be multiples of 128");
  if (fp8)
    return bq_gemm_typed<true>(mode, a, sa, da, b_t, sb, row_b, out, out_t, so, dout, batch, m, n, k,
                               lm, ln, ca, cb, cc, final, transpose, out_dtype, status, S(stream));
  return bq_gemm_typed<false>(mode, a, sa, da, b_t, sb, row_b, out, out_t, so, dout, batch, m, n, k,
                              lm, ln, ca, cb, cc, final, transpose, out_dtype, status, S(stream));
}
