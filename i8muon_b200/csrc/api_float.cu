// C ABI: floating-point products.
#include "launch_gemm.cuh"
#include "drivers.cuh"
#include "epi_float.cuh"
#include "epi_float_bq.cuh"

using namespace i8m;

namespace {

template <typename E>
int float_gemm_typed(const FloatGemm& f) {
  FloatArgs a;
  a.out = f.out; a.out_t = f.out_t; a.out_lo = f.out_lo; a.out_t_lo = f.out_t_lo;
  a.src = f.left; a.src_lo = f.left_lo;
  a.out_dtype = f.out_dtype; a.transpose = f.transpose;
  a.ca = f.ca; a.cb = f.cb; a.cc = f.cc;
  a.amax = f.final ? f.amax : nullptr;
  GemmCall g;
  g.a = f.left; g.a_lo = f.left_lo; g.b = f.right; g.b_lo = f.right_lo; g.a_mn = f.left_mn; g.b_mn = f.right_mn;
  g.batch = f.batch; g.m = f.m; g.n = f.n; g.k = f.k; g.lm = f.lm; g.ln = f.ln;
  g.sym = f.final ? 0 : f.symmetric; g.status = f.status; g.stream = f.stream;
  if (f.mode == 1) {
    if (f.final) return fail(I8M_E_ARGUMENT, "float_gemm: the polynomial mode has no final variant");
    if (f.k != f.n) return fail(I8M_E_ARGUMENT, "float_gemm: polynomial mode needs a square left operand");
    return launch_gemm<EpiFloat<E, MODE_QUAD>>(g, a, "float_gemm(poly)");
  }
  if (f.final) {
    if (!float_dtype_ok(f.out_dtype)) return fail(I8M_E_ARGUMENT, "float_gemm: bad out_dtype %d", f.out_dtype);
    return launch_gemm<EpiFloat<E, MODE_FINAL>>(g, a, "float_gemm(final)");
  }
  return launch_gemm<EpiFloat<E, MODE_PLAIN>>(g, a, "float_gemm");
}
}  // namespace

int i8m::float_gemm(const FloatGemm& f) {
  if (!f.out || (f.mode != 0 && f.mode != 1)) return fail(I8M_E_ARGUMENT, "float_gemm: bad argument");
  if (f.compute == I8M_F32) return float_gemm_typed<float>(f);
  if (f.compute == I8M_F16) return float_gemm_typed<__half>(f);
  if (f.compute == I8M_BF16) return float_gemm_typed<__nv_bfloat16>(f);
  return fail(I8M_E_ARGUMENT, "float_gemm: bad compute dtype %d", f.compute);
}
extern "C" int i8m_float_gemm(const void* left, const void* left_lo, const void* right_t,
                              const void* right_t_lo, void* out, void* out_t, void* out_lo,
                              void* out_t_lo, int compute, int mode, int batch, int m, int n, int k,
                              int lm, int ln, int symmetric, int final, int transpose,
                              int out_dtype, float ca, float cb, float cc, uint32_t* status,
                              i8m_stream_t stream) {
  return float_gemm(FloatGemm{left, left_lo, right_t, right_t_lo, out, out_t, out_lo, out_t_lo, compute, mode, batch, m, n, k,
                              lm, ln, symmetric, final, transpose, out_dtype, 0, 0, ca, cb, cc, nullptr, status, S(stream)});
}

// FP16 / BF16 product whose result leaves as block-quantised INT8 operands (the end of the FP16 first
// iteration of an fp16-first INT8-BQ call): persistent kernel only.
template <typename E>
static int float_gemm_to_bq_typed(const void* left, const void* right, int right_mn, const FloatToBqArgs& args, int batch,
                                  int m, int n, int k, int lm, int ln, unsigned* status, cudaStream_t stream) {
  using Epi = EpiFloatToBq<E>;
  GemmGeom g{};
  g.batch = batch; g.m = m; g.n = n; g.k = k; g.lm = lm; g.ln = ln;
  g.tiles_m = cdiv(m, TILE); g.tiles_n = cdiv(n, TILE);
  g.sym = 0;
  g.tiles_per_batch = g.tiles_m * g.tiles_n;
  g.num_kb = cdiv((long long)k * 2, 128);
  g.b_mn = right_mn;
  g.group = wide_group(2LL * k);
  g.a_raw = left; g.b_raw = right; g.status = status;
  const long long blocks = (long long)g.tiles_per_batch * batch;
  if (blocks > 0x7fffffffLL) return fail(I8M_E_LIMIT, "float_gemm_to_bq: too many tiles");
  CUtensorMap ma, mb;
  if (int rc = make_operand_map(&ma, left, 2, k, m, batch)) return rc;
  if (int rc = make_operand_map(&mb, right, 2, k, n, batch, right_mn)) return rc;
  if (g_wholek_variant == 0) {
    constexpr size_t WSMEM = wholek_wide_smem_bytes<Epi>();
    auto wk = wholek_wide_kernel<Epi>;
    static SmemAllowed allowed;
    if (int rc = allow_smem(allowed, wk, WSMEM)) return rc;
    const long long pairs = (long long)wide_units_per_batch(g.tiles_m, g.tiles_n, 0) * batch;
    g.narrow = narrow_units(blocks, pairs, g.num_kb, sm_count());
    const long long units = g.narrow ? blocks : pairs;
    launch(wk, unsigned(std::min<long long>(units, sm_count())), WKW_THREADS, WSMEM, stream, ma, mb, g, args);
    LAUNCH_CHECK("float_gemm_to_bq");
    return 0;
  }
  constexpr size_t SMEM = size_t(WKP_STAGES) * 2 * TILE_BYTES + sizeof(Ctrl) + Epi::TSM_BYTES + 1024;
  auto kernel = wholek_persistent_kernel<Epi>;
  static SmemAllowed allowed;
  if (int rc = allow_smem(allowed, kernel, SMEM)) return rc;
  const unsigned grid = unsigned(std::min<long long>(blocks, sm_count()));
  launch(kernel, grid, WKP_THREADS, SMEM, stream, ma, mb, g, args);
  LAUNCH_CHECK("float_gemm_to_bq");
  return 0;
}

int i8m::float_gemm_to_bq(const void* left, const void* right, int right_mn, void* q, void* q_t, float* scale, int compute,
                          int user_dtype, int batch, int m, int n, int k, int lm, int ln, int lp, int hp, unsigned* status,
                          cudaStream_t stream) {
  if (!left || !right || !q || !q_t || !scale || !status) return fail(I8M_E_ARGUMENT, "float_gemm_to_bq: null pointer");
  if (batch < 1 || m < 1 || n < 1 || k < 1 || lm < 1 || ln < 1 || lm > m || ln > n)
    return fail(I8M_E_ARGUMENT, "float_gemm_to_bq: bad extents");
  if (lp % 128 || hp % 128 || lp < m || hp < n || cdiv(lp, 128) != cdiv(m, 128) || cdiv(hp, 128) != cdiv(n, 128))
    return fail(I8M_E_ARGUMENT, "float_gemm_to_bq: lp, hp must be m, n rounded up to multiples of 128");
  if (!float_dtype_ok(user_dtype)) return fail(I8M_E_ARGUMENT, "float_gemm_to_bq: bad user dtype");
  FloatToBqArgs a;
  a.q = static_cast<uint8_t*>(q); a.qt = static_cast<uint8_t*>(q_t); a.scale = scale;
  a.lp = lp; a.hp = hp; a.user_dtype = user_dtype;
  if (compute == I8M_F16)
    return float_gemm_to_bq_typed<__half>(left, right, right_mn, a, batch, m, n, k, lm, ln, status, stream);
  if (compute == I8M_BF16)
    return float_gemm_to_bq_typed<__nv_bfloat16>(left, right, right_mn, a, batch, m, n, k, lm, ln, status, stream);
  return fail(I8M_E_ARGUMENT, "float_gemm_to_bq: compute must be a 16-bit type");
}
extern "C" int i8m_float_gemm_to_bq(const void* left, const void* right_t, void* q, void* q_t, float* scale,
                                    int compute, int user_dtype, int batch, int m, int n, int k, int lm, int ln,
                                    int lp, int hp, uint32_t* status, i8m_stream_t stream) {
  return float_gemm_to_bq(left, right_t, 0, q, q_t, scale, compute, user_dtype, batch, m, n, k, lm, ln, lp, hp, status,
                          S(stream));
}
