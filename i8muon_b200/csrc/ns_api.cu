// Host side of the C ABI: library state and the C++ drivers that sequence one whole Newton-Schulz call out
// of the stage kernels.  No device memory is allocated here; the caller's
// workspace is carved up by a bump allocator.
#include "host.cuh"
#include "drivers.cuh"

#include <cstring>
#include <mutex>
#include <string>

using namespace i8m;

namespace i8m {

thread_local char g_error[512] = "";
thread_local int g_debug_simt = 0;
thread_local int g_starve_producers = 0;
thread_local int g_wholek_variant = 0;
thread_local int g_cta_limit = 0;
thread_local int g_bq_variant = 0;
std::atomic<unsigned long long> g_launches{0};

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_error, sizeof(g_error), fmt, ap);
  va_end(ap);
  return code;
}
int sm_count() {
  static int counts[64] = {};
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return 148;
  if (counts[device] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || n <= 0) n = 148;
    counts[device] = n;
  }
  return g_cta_limit > 0 ? std::min(counts[device], g_cta_limit) : counts[device];
}


namespace {
// ------------------------------------------------------- tensor map encode
using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                              CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                              CUtensorMapFloatOOBfill);
EncodeFn g_encode = nullptr;
std::once_flag g_encode_once;

int load_encode() {
  std::call_once(g_encode_once, [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) ==
            cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      g_encode = reinterpret_cast<EncodeFn>(fn);
  });
  return g_encode ? 0 : fail(I8M_E_CUDA, "cuTensorMapEncodeTiled is not available in this driver");
}
}  // namespace

int make_operand_map(CUtensorMap* map, const void* ptr, int esize, int k, int extent, int batch, int mn) {
  const int inner = mn ? extent : k, rows = mn ? k : extent;
  if (int rc = load_encode()) return rc;
  if ((reinterpret_cast<uintptr_t>(ptr) & 15u) != 0)
    return fail(I8M_E_ARGUMENT, "GEMM operand is not 16-byte aligned");
  if ((size_t(inner) * esize) % 16 != 0)
    return fail(I8M_E_ARGUMENT, "GEMM operand row pitch (%d x %d bytes) is not a multiple of 16", inner, esize);
  CUtensorMapDataType dt = esize == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                         : esize == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16
                                      : CU_TENSOR_MAP_DATA_TYPE_UINT32;
  cuuint64_t dims[3] = {cuuint64_t(inner), cuuint64_t(rows), cuuint64_t(batch)};
  cuuint64_t strides[2] = {cuuint64_t(inner) * esize, cuuint64_t(inner) * esize * rows};
  cuuint32_t box[3] = {cuuint32_t(128 / esize), cuuint32_t(mn ? 128 / esize : 128), 1u};
  cuuint32_t estr[3] = {1u, 1u, 1u};
  CUresult r = g_encode(map, dt, 3, const_cast<void*>(ptr), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(I8M_E_CUDA, "cuTensorMapEncodeTiled failed with code %d", int(r));
  return 0;
}

}  // namespace i8m

// =========================================================== library state
extern "C" int i8m_version(void) { return 100; }
extern "C" const char* i8m_build_info(void) {
  static char info[256];
  snprintf(info, sizeof(info),
           "i8muon_b200 arch=sm_100a cudart=%d tile=128x128x128B threads=%d mma=tcgen05 copy=tma "
           "fmad=off",
           CUDART_VERSION, GEMM_THREADS);
  return info;
}
extern "C" const char* i8m_last_error(void) { return g_error; }
extern "C" unsigned long long i8m_launch_count(void) { return g_launches.load(); }
extern "C" int i8m_set_debug_core(int simt) {
  g_debug_simt = simt == 1 ? 1 : 0;
  g_starve_producers = simt == 2 ? 1 : 0;
  return 0;
}
extern "C" int i8m_set_cta_limit(int max_ctas) {
  if (max_ctas < 0) return fail(I8M_E_ARGUMENT, "set_cta_limit: negative limit");
  g_cta_limit = max_ctas;
  return 0;
}
extern "C" int i8m_variant_count(const char* operation) {
  if (operation && std::strcmp(operation, "bq_gemm") == 0) return BQ_VARIANTS;
  if (operation && std::strcmp(operation, "wholek_gemm") == 0) return WHOLEK_VARIANTS;
  return 0;
}
extern "C" int i8m_set_variant(const char* operation, int variant) {
  if (!operation || (std::strcmp(operation, "bq_gemm") != 0 && std::strcmp(operation, "wholek_gemm") != 0))
    return fail(I8M_E_ARGUMENT, "set_variant: unknown operation");
  if (variant < 0 || variant >= i8m_variant_count(operation))
    return fail(I8M_E_ARGUMENT, "set_variant: %s has variants 0 to %d", operation, i8m_variant_count(operation) - 1);
  if (operation[0] == 'b') g_bq_variant = variant;
  else g_wholek_variant = variant;
  return 0;
}

// ============================================== whole Newton-Schulz drivers
namespace {

struct Bump {
  char* base;
  size_t used = 0, cap;
  bool dry;
  Bump(void* p, size_t c, bool d) : base(static_cast<char*>(p)), cap(c), dry(d) {}
  void* take(size_t bytes) {
    size_t off = align256(used);
    used = off + bytes;
    return dry ? nullptr : base + off;
  }
  template <typename T>
  T* take_n(size_t n) { return static_cast<T*>(take(n * sizeof(T))); }
};

struct NsCall {
  int route, dtype, batch, rows, cols, compute, steps, fp16_first;
  int factored = 0;   // coefficient rows are (c, p, q) of c * ((G + p I)^2 + q I)
  int deterministic = 1;   // 0: one-pass statistics with atomics (summation order not reproducible)
  const float* stats_partials = nullptr;   // partials of the statistics over x, computed by the caller (i8m_momentum)
  int fuse_first_row = 1;   // fp16-first INT8-BQ: the first row's update quantises its own result
  int wholek[3] = {-1, -1, -1};   // global INT8: kernel variant of the Gram / square / update product (-1: thread's)
  const void* x;
  void* out;
  const double* coeffs;
  float eps;
  const char* gram_order;
  unsigned* status;
  cudaStream_t stream;
};

int call_stats(const NsCall& c, const void* x, int B, long long count, void* scratch, size_t sbytes, float* norm,
               float* amax) {
  if (c.stats_partials && x == c.x) {
    // the producer of x left the per-chunk partials: only the final fold remains
    return fold_stats(c.stats_partials, B, count, norm, amax, c.stream);
  }
  if (c.deterministic) return i8m_stats(x, c.dtype, B, count, scratch, sbytes, norm, amax, c.stream);
  return i8m_stats_onepass(x, c.dtype, B, count, scratch, sbytes, norm, amax, c.stream);
}
size_t stats_bytes(int B, long long count) {
  size_t sbytes = 0;
  i8m_stats_scratch_bytes(B, count, &sbytes);
  return std::max(sbytes, size_t(3) * B * sizeof(float));   // either flavour fits
}

// A matrix in the floating compute dtype: one plane, or (hi, lo) for FP32.
struct FMat {
  void* p = nullptr;
  void* lo = nullptr;
};
FMat take_fmat(Bump& ws, size_t elems, int compute) {
  FMat m;
  m.p = ws.take(elems * dtype_size(compute));
  if (compute == I8M_F32) m.lo = ws.take(elems * 4);
  return m;
}

// Restart string of a Gram-space call, padded to the number of iterations.
int restart_order(const NsCall& c, int steps, std::string& order) {
  order = c.gram_order ? c.gram_order : "00100";
  if (order.empty() || order[0] != '0' || order.find_first_not_of("01") != std::string::npos)
    return fail(I8M_E_ARGUMENT, "gram_order must be a binary string starting with 0");
  if (int(order.size()) < steps) order.append(size_t(steps) - order.size(), '0');
  return 0;
}

struct BqOperands {   // where a floating first row leaves its result for the block-quantised rows
  uint8_t* a = nullptr;
  uint8_t* at = nullptr;
  float* sa = nullptr;
  int lp = 0, hp = 0;
};

// Floating NS (regular and Gram) in a 16-bit compute type; with plan == true only the workspace is sized.
// The matrix X stays in the caller's orientation, padded to multiples of 16, and is stored once: the products that
// run along its rows read it K-major, those that run across them MN-major.
//   wide (l x h)   Gram X X^T: both K-major;           update Q X: X is the right operand, MN-major
//   tall (h x l)   Gram X^T X: both operands MN-major; update X Q: X is the left operand, K-major (Q is symmetric)
int run_float16(const NsCall& c, Bump& ws, bool plan, bool gram, const void* x, void* out, int out_dtype, int steps,
                const double* coeffs, int compute, bool normalize_input, bool factored, const BqOperands* to_bq,
                float* final_amax) {
  const int B = c.batch, rows = c.rows, cols = c.cols;
  const int l = std::min(rows, cols), h = std::max(rows, cols);
  const int lp = pad_to(l, 16), hp = pad_to(h, 16), rp = pad_to(rows, 16), cp = pad_to(cols, 16);
  const int tall = rows > cols;
  const size_t es = 2, full = size_t(B) * rp * cp * es, sq = size_t(B) * lp * lp * es;
  void *a = ws.take(full), *y = ws.take(full);
  void *r = ws.take(sq), *q0 = ws.take(sq), *z = nullptr, *q1 = nullptr;
  if (gram) { z = ws.take(sq); q1 = ws.take(sq); }
  float* norm = ws.take_n<float>(B);
  const size_t sbytes = stats_bytes(B, (long long)rows * cols);
  void* scratch = ws.take(sbytes);
  if (plan) return 0;

  if (normalize_input)
    if (int rc = call_stats(c, x, B, (long long)rows * cols, scratch, sbytes, norm, nullptr)) return rc;
  if (int rc = i8m_normalize(x, c.dtype, normalize_input ? norm : nullptr, a, nullptr, nullptr, nullptr, compute, B, rows,
                             cols, rp, cp, 0, c.eps, c.stream))
    return rc;
  FloatGemm base{};
  base.compute = compute; base.batch = B; base.status = c.status; base.stream = c.stream; base.out_dtype = out_dtype;
  auto square = [&](const void* left, const void* right, void* o, int mode, double ca, double cb, double cc) {
    FloatGemm g = base;   // symmetric l x l product of two l x l matrices
    g.left = left; g.right = right; g.out = o; g.mode = mode;
    g.m = g.n = g.k = lp; g.lm = g.ln = l; g.symmetric = 1;
    g.ca = float(ca); g.cb = float(cb); g.cc = float(cc);
    return float_gemm(g);
  };
  auto outer = [&](void* o) {
    FloatGemm g = base;   // R = X X^T or X^T X
    g.left = g.right = a; g.left_mn = g.right_mn = tall; g.out = o;
    g.m = g.n = lp; g.k = hp; g.lm = g.ln = l; g.symmetric = 1;
    return float_gemm(g);
  };
  auto update = [&](const void* q, void* o, int final) {
    FloatGemm g = base;
    g.left = tall ? a : q; g.right = tall ? q : a; g.right_mn = !tall;
    g.out = o; g.final = final; g.amax = final ? final_amax : nullptr;
    g.m = rp; g.n = cp; g.k = lp; g.lm = rows; g.ln = cols;
    return float_gemm(g);
  };
  if (!gram) {
    for (int it = 0; it < steps; ++it) {
      double ca = coeffs[3 * it], cb = coeffs[3 * it + 1], cc = coeffs[3 * it + 2];
      if (int rc = outer(r)) return rc;
      if (factored) {
        // completed-square row (c, p, q): shift the Gram diagonal by p, then c*q I + c R'^2
        // (src/i8muon/_cutlass_prec.py:97-100)
        const double fc = ca, fp = cb, fq = cc;
        if (int rc = add_diagonal(r, compute, B, lp, l, float(fp), c.stream)) return rc;
        ca = fc * fq; cb = 0.0; cc = fc;
      }
      if (int rc = square(r, r, q0, 1, ca, cb, cc)) return rc;
      const bool final = it == steps - 1;
      if (final && to_bq)   // the result leaves as INT8 blocks of the wide orientation
        return float_gemm_to_bq(q0, a, !tall, to_bq->a, to_bq->at, to_bq->sa, compute, out_dtype, B, lp, hp, lp, l, h,
                                to_bq->lp, to_bq->hp, c.status, c.stream);
      if (int rc = update(q0, final ? out : y, final)) return rc;
      std::swap(a, y);
    }
    return 0;
  }
  // Gram-space iteration with restarts (src/i8muon/_cutlass_prec.py:107-130).
  std::string order;
  if (int rc = restart_order(c, steps, order)) return rc;
  for (int it = 0; it < steps; ++it) {
    const double ca = coeffs[3 * it], cb = coeffs[3 * it + 1], cc = coeffs[3 * it + 2];
    const char kind = order[size_t(it)];
    const bool refresh = it + 1 < steps && order[size_t(it) + 1] == '0';
    if (kind == '1') {
      if (int rc = update(q0, y, 0)) return rc;
      std::swap(a, y);
    }
    if (kind == '1' || it == 0) {
      if (int rc = outer(r)) return rc;
      if (int rc = square(r, r, q0, 1, ca, cb, cc)) return rc;
      if (refresh) {
        if (int rc = square(r, q0, q1, 0, 0, 0, 0)) return rc;
        if (int rc = square(q0, q1, r, 0, 0, 0, 0)) return rc;
      }
    } else {
      if (int rc = square(r, r, z, 1, ca, cb, cc)) return rc;
      if (int rc = square(z, q0, q1, 0, 0, 0, 0)) return rc;
      std::swap(q0, q1);
      if (refresh) {
        if (int rc = square(r, z, q1, 0, 0, 0, 0)) return rc;
        if (int rc = square(z, q1, r, 0, 0, 0, 0)) return rc;
      }
    }
  }
  return update(q0, out, 1);
}

// FP32 compute: every matrix as two planes, X and its transpose both stored (TF32 operands are read K-major only).
int run_float32(const NsCall& c, Bump& ws, bool plan, bool gram, const void* x, void* out, int out_dtype, int steps,
                const double* coeffs) {
  const int compute = I8M_F32;
  const int B = c.batch, rows = c.rows, cols = c.cols;
  const int l = std::min(rows, cols), h = std::max(rows, cols);
  const int lp = pad_to(l, 16), hp = pad_to(h, 16);
  const int transpose = rows > cols;
  const size_t wide = size_t(B) * lp * hp, sq = size_t(B) * lp * lp;
  FMat a = take_fmat(ws, wide, compute), at = take_fmat(ws, wide, compute);
  FMat y = take_fmat(ws, wide, compute), yt = take_fmat(ws, wide, compute);
  FMat r = take_fmat(ws, sq, compute), q0 = take_fmat(ws, sq, compute);
  FMat z, q1;
  if (gram) { z = take_fmat(ws, sq, compute); q1 = take_fmat(ws, sq, compute); }
  float* norm = ws.take_n<float>(B);
  const size_t sbytes = stats_bytes(B, (long long)rows * cols);
  void* scratch = ws.take(sbytes);
  if (plan) return 0;

  if (int rc = call_stats(c, x, B, (long long)rows * cols, scratch, sbytes, norm, nullptr)) return rc;
  if (int rc = i8m_normalize(x, c.dtype, norm, a.p, at.p, a.lo, at.lo,
                             compute, B, rows, cols, lp, hp, transpose, c.eps, c.stream))
    return rc;
  auto gemm = [&](const FMat& left, const FMat& right, const FMat& o, const FMat& ot, int mode, int n,
                  int k, int ln, int sym, int final, int tr, void* user, double ca, double cb,
                  double cc) -> int {
    return i8m_float_gemm(left.p, left.lo, right.p, right.lo, final ? user : o.p, ot.p, o.lo, ot.lo,
                          compute, mode, B, lp, n, k, l, ln, sym, final, tr, out_dtype, float(ca),
                          float(cb), float(cc), c.status, c.stream);
  };
  const FMat none;
  if (!gram) {
    for (int it = 0; it < steps; ++it) {
      const double ca = coeffs[3 * it], cb = coeffs[3 * it + 1], cc = coeffs[3 * it + 2];
      if (int rc = gemm(a, a, r, none, 0, lp, hp, l, 1, 0, 0, nullptr, 0, 0, 0)) return rc;
      if (int rc = gemm(r, r, q0, none, 1, lp, lp, l, 1, 0, 0, nullptr, ca, cb, cc)) return rc;
      const bool final = it == steps - 1;
      if (int rc = gemm(q0, at, y, yt, 0, hp, lp, h, 0, final, final && transpose, out, 0, 0, 0)) return rc;
      if (!final) { std::swap(a, y); std::swap(at, yt); }
    }
    return 0;
  }
  // Gram-space iteration with restarts (src/i8muon/_cutlass_prec.py:107-130).
  std::string order;
  if (int rc = restart_order(c, steps, order)) return rc;
  for (int it = 0; it < steps; ++it) {
    const double ca = coeffs[3 * it], cb = coeffs[3 * it + 1], cc = coeffs[3 * it + 2];
    const char kind = order[size_t(it)];
    const bool refresh = it + 1 < steps && order[size_t(it) + 1] == '0';
    if (kind == '1') {
      if (int rc = gemm(q0, at, y, yt, 0, hp, lp, h, 0, 0, 0, nullptr, 0, 0, 0)) return rc;
      std::swap(a, y); std::swap(at, yt);
    }
    if (kind == '1' || it == 0) {
      if (int rc = gemm(a, a, r, none, 0, lp, hp, l, 1, 0, 0, nullptr, 0, 0, 0)) return rc;
      if (int rc = gemm(r, r, q0, none, 1, lp, lp, l, 1, 0, 0, nullptr, ca, cb, cc)) return rc;
      if (refresh) {
        if (int rc = gemm(r, q0, q1, none, 0, lp, lp, l, 1, 0, 0, nullptr, 0, 0, 0)) return rc;
        if (int rc = gemm(q0, q1, r, none, 0, lp, lp, l, 1, 0, 0, nullptr, 0, 0, 0)) return rc;
      }
    } else {
      if (int rc = gemm(r, r, z, none, 1, lp, lp, l, 1, 0, 0, nullptr, ca, cb, cc)) return rc;
      if (int rc = gemm(z, q0, q1, none, 0, lp, lp, l, 1, 0, 0, nullptr, 0, 0, 0)) return rc;
      std::swap(q0, q1);
      if (refresh) {
        if (int rc = gemm(r, z, q1, none, 0, lp, lp, l, 1, 0, 0, nullptr, 0, 0, 0)) return rc;
        if (int rc = gemm(z, q1, r, none, 0, lp, lp, l, 1, 0, 0, nullptr, 0, 0, 0)) return rc;
      }
    }
  }
  return gemm(q0, at, y, yt, 0, hp, lp, h, 0, 1, transpose, out, 0, 0, 0);
}

int run_float(const NsCall& c, Bump& ws, bool plan, bool gram, const void* x, void* out, int out_dtype, int steps,
              const double* coeffs, int compute, bool normalize_input, bool factored = false,
              const BqOperands* to_bq = nullptr, float* final_amax = nullptr) {
  if (compute == I8M_F32) return run_float32(c, ws, plan, gram, x, out, out_dtype, steps, coeffs);
  return run_float16(c, ws, plan, gram, x, out, out_dtype, steps, coeffs, compute, normalize_input, factored, to_bq, final_amax);
}

// global-scale INT8 NS (src/i8muon/_cutlass.py:162-251)
int run_int8(const NsCall& c, Bump& ws, bool plan, const void* x, int steps, const double* coeffs,
             bool normalize_input, bool factored = false, const float* given_amax = nullptr) {
  const int B = c.batch, rows = c.rows, cols = c.cols;
  const int l = std::min(rows, cols), h = std::max(rows, cols);
  const int lp = pad_to(l, 16), hp = pad_to(h, 16);
  const int transpose = rows > cols;
  const size_t wide = size_t(B) * lp * hp, sq = size_t(B) * lp * lp;
  int8_t* a8 = ws.take_n<int8_t>(wide);
  float* work = ws.take_n<float>(wide);      // int32 Gram / fp32 polynomial / fp32 update
  int8_t* s8 = ws.take_n<int8_t>(sq);         // quantised Gram, then quantised polynomial
  float* a_scale = ws.take_n<float>(B);
  float* g_scale = ws.take_n<float>(B);
  float* p_scale = ws.take_n<float>(B);
  float* g_diag = ws.take_n<float>(size_t(B) * lp);
  float* p_diag = ws.take_n<float>(size_t(B) * lp);
  float* maxima = ws.take_n<float>(size_t(3) * steps * B);
  float* norm = ws.take_n<float>(B);
  float* amax = ws.take_n<float>(B);
  const size_t sbytes = stats_bytes(B, (long long)rows * cols);
  void* scratch = ws.take(sbytes);
  if (plan) return 0;
  if ((long long)hp * 127 * 127 > 0x7fffffffLL)
    return fail(I8M_E_LIMIT, "inner dimension can overflow the int32 accumulator");

  CUDA_TRY(cudaMemsetAsync(maxima, 0, size_t(3) * steps * B * sizeof(float), c.stream));
  if (given_amax == nullptr) {
    if (int rc = call_stats(c, x, B, (long long)rows * cols, scratch, sbytes, normalize_input ? norm : nullptr, amax))
      return rc;
  }
  if (int rc = input_quant(x, c.dtype, given_amax ? given_amax : amax, normalize_input ? norm : nullptr, a8, a_scale, B, rows,
                           cols, lp, hp, transpose, c.eps, c.stream))
    return rc;
  for (int it = 0; it < steps; ++it) {
    // A completed-square row (c, p, q) is the same five stages with the Gram diagonal shifted
    // by p, the polynomial G'^2 + q I (b = 0, c = 1, a = q: bit-identical expressions to the
    // reference's unscaled modes) and c folded into the update's right-hand scale
    // (src/i8muon/_cutlass.py:196-246).
    float ca = float(coeffs[3 * it]), cb = float(coeffs[3 * it + 1]), cc = float(coeffs[3 * it + 2]);
    float shift = 0.f, gain = 0.f;
    if (factored) { gain = ca; shift = cb; ca = cc; cb = 0.f; cc = 1.f; }
    float* gmax = maxima + size_t(3 * it) * B;
    float* pmax = gmax + B;
    float* ymax = pmax + B;
    const int thread_wholek = g_wholek_variant;
    auto pick = [&](int op) { g_wholek_variant = c.wholek[op] < 0 ? thread_wholek : c.wholek[op]; };
    struct Restore { int v; ~Restore() { g_wholek_variant = v; } } restore{thread_wholek};
    pick(0);
    if (int rc = i8m_i8_gemm(0, a8, a8, nullptr, work, gmax, nullptr, nullptr, nullptr, B, lp, lp, hp, l,
                             l, 0, 0, 0, 0, 0, c.status, c.stream))
      return rc;
    if (int rc = i8m_symmetric_quant(work, gmax, a_scale, nullptr, s8, g_scale, g_diag, B, lp, 0, shift, 0, 0, c.stream))
      return rc;
    pick(1);
    if (int rc = i8m_i8_gemm(1, s8, s8, nullptr, work, pmax, g_scale, nullptr, g_diag, B, lp, lp, lp, l, l,
                             cb, cc, 0, 0, 0, c.status, c.stream))
      return rc;
    if (int rc = i8m_symmetric_quant(work, pmax, g_scale, g_diag, s8, p_scale, p_diag, B, lp, 1, ca, cb, cc, c.stream))
      return rc;
    const bool final = it == steps - 1;
    pick(2);
    // X is stored once: the update reads it across K
    if (int rc = i8_gemm(factored ? 4 : 2, s8, a8, 1, a8, final ? c.out : static_cast<void*>(work), ymax, p_scale,
                             a_scale, p_diag, B, lp, hp, lp, l, h, gain, 0, final, transpose, c.dtype,
                             c.status, c.stream))
      return rc;
    if (!final)
      if (int rc = output_quant(work, ymax, a8, a_scale, B, lp, hp, c.stream)) return rc;
  }
  return 0;
}

// grouped cubics with a terminal quintic, all INT8 (src/i8muon/_cutlass_cubic.py:8-71): per cubic the
// Gram product, its quantisation with the shifted FP32 diagonal, the update with -gain folded into
// the right-hand scale, and the output quantisation; then the regular five stages of the last row.
int run_int8_cubic(const NsCall& c, Bump& ws, bool plan) {
  const int B = c.batch, rows = c.rows, cols = c.cols;
  const int l = std::min(rows, cols), h = std::max(rows, cols);
  const int lp = pad_to(l, 16), hp = pad_to(h, 16);
  const int transpose = rows > cols;
  const int cubics = c.steps - 2;
  const size_t wide = size_t(B) * lp * hp, sq = size_t(B) * lp * lp;
  int8_t* a8 = ws.take_n<int8_t>(wide);
  float* work = ws.take_n<float>(wide);
  int8_t* s8 = ws.take_n<int8_t>(sq);
  float* a_scale = ws.take_n<float>(B);
  float* g_scale = ws.take_n<float>(B);
  float* p_scale = ws.take_n<float>(B);
  float* g_diag = ws.take_n<float>(size_t(B) * lp);
  float* p_diag = ws.take_n<float>(size_t(B) * lp);
  const size_t slots = size_t(2) * std::max(cubics, 0) + 3;
  float* maxima = ws.take_n<float>(slots * B);
  float* norm = ws.take_n<float>(B);
  float* amax = ws.take_n<float>(B);
  const size_t sbytes = stats_bytes(B, (long long)rows * cols);
  void* scratch = ws.take(sbytes);
  if (plan) return 0;
  if (cubics < 1) return fail(I8M_E_ARGUMENT, "the cubic route needs an input-gain row, cubic rows and a terminal row");
  if ((long long)hp * 127 * 127 > 0x7fffffffLL)
    return fail(I8M_E_LIMIT, "inner dimension can overflow the int32 accumulator");
  const float input_gain = float(c.coeffs[0]);
  if (!(input_gain > 0.f) || !(c.eps > 0.f)) return fail(I8M_E_ARGUMENT, "the cubic route needs positive input_gain and eps");
  CUDA_TRY(cudaMemsetAsync(maxima, 0, slots * B * sizeof(float), c.stream));
  if (int rc = call_stats(c, c.x, B, (long long)rows * cols, scratch, sbytes, norm, amax)) return rc;
  if (int rc = clamp_divide(norm, B, c.eps, input_gain, c.stream)) return rc;
  if (int rc = input_quant(c.x, c.dtype, amax, norm, a8, a_scale, B, rows, cols, lp, hp, transpose, 0.f, c.stream))
    return rc;
  for (int i = 0; i < cubics; ++i) {
    const float gain = float(c.coeffs[3 * (i + 1)]), shift = float(c.coeffs[3 * (i + 1) + 1]);
    float* gmax = maxima + size_t(2 * i) * B;
    float* ymax = gmax + B;
    if (int rc = i8m_i8_gemm(0, a8, a8, nullptr, work, gmax, nullptr, nullptr, nullptr, B, lp, lp, hp, l, l, 0, 0, 0, 0, 0,
                             c.status, c.stream))
      return rc;
    if (int rc = i8m_symmetric_quant(work, gmax, a_scale, nullptr, s8, g_scale, g_diag, B, lp, 0, shift, 0, 0, c.stream))
      return rc;
    if (int rc = i8_gemm(4, s8, a8, 1, a8, work, ymax, g_scale, a_scale, g_diag, B, lp, hp, lp, l, h, -gain, 0, 0, 0, 0,
                             c.status, c.stream))
      return rc;
    if (int rc = output_quant(work, ymax, a8, a_scale, B, lp, hp, c.stream)) return rc;
  }
  const double* abc = c.coeffs + 3 * (c.steps - 1);
  float* gmax = maxima + size_t(2 * cubics) * B;
  float* pmax = gmax + B;
  if (int rc = i8m_i8_gemm(0, a8, a8, nullptr, work, gmax, nullptr, nullptr, nullptr, B, lp, lp, hp, l, l, 0, 0, 0, 0, 0,
                           c.status, c.stream))
    return rc;
  if (int rc = i8m_symmetric_quant(work, gmax, a_scale, nullptr, s8, g_scale, g_diag, B, lp, 0, 0, 0, 0, c.stream)) return rc;
  if (int rc = i8m_i8_gemm(1, s8, s8, nullptr, work, pmax, g_scale, nullptr, g_diag, B, lp, lp, lp, l, l, float(abc[1]),
                           float(abc[2]), 0, 0, 0, c.status, c.stream))
    return rc;
  if (int rc = i8m_symmetric_quant(work, pmax, g_scale, g_diag, s8, p_scale, p_diag, B, lp, 1, float(abc[0]), float(abc[1]),
                                   float(abc[2]), c.stream))
    return rc;
  return i8_gemm(2, s8, a8, 1, a8, c.out, nullptr, p_scale, a_scale, p_diag, B, lp, hp, lp, l, h, 0, 0, 1, transpose,
                     c.dtype, c.status, c.stream);
}

// block-quantised NS (src/i8muon/_cutlass_bq.py:15-70)
int run_bq(const NsCall& c, Bump& ws, bool plan, bool fp8, const void* x, int steps,
           const double* coeffs, bool normalize_input, const BqOperands* given = nullptr) {
  const int B = c.batch, rows = c.rows, cols = c.cols;
  const int l = std::min(rows, cols), h = std::max(rows, cols);
  const int lp = pad_to(l, 128), hp = pad_to(h, 128);
  const int transpose = rows > cols;
  const size_t wide = size_t(B) * lp * hp, sq = size_t(B) * lp * lp;
  const int lq = lp / 128, hq = hp / 128;
  // `given`: the operands were quantised already (by the floating first row's epilogue)
  uint8_t* a = given ? given->a : ws.take_n<uint8_t>(wide);
  uint8_t* at = given ? given->at : ws.take_n<uint8_t>(wide);
  uint8_t* y = ws.take_n<uint8_t>(wide);
  uint8_t* yt = ws.take_n<uint8_t>(wide);
  uint8_t* gq = ws.take_n<uint8_t>(sq);
  uint8_t* pq = ws.take_n<uint8_t>(sq);
  float* sa = given ? given->sa : ws.take_n<float>(size_t(B) * lq * hq);
  float* sy = ws.take_n<float>(size_t(B) * lq * hq);
  float* sg = ws.take_n<float>(size_t(B) * lq * lq);
  float* sp = ws.take_n<float>(size_t(B) * lq * lq);
  float* dg = ws.take_n<float>(size_t(B) * lp);
  float* dp = ws.take_n<float>(size_t(B) * lp);
  float* norm = ws.take_n<float>(B);
  const size_t sbytes = stats_bytes(B, (long long)rows * cols);
  void* scratch = ws.take(sbytes);
  if (plan) return 0;

  if (!given) {
    if (normalize_input)
      if (int rc = call_stats(c, x, B, (long long)rows * cols, scratch, sbytes, norm, nullptr)) return rc;
    if (int rc = i8m_bq_quant(x, c.dtype, normalize_input ? norm : nullptr, a, at, sa, fp8, B, rows, cols,
                              lp, hp, transpose, c.eps, c.stream))
      return rc;
  }
  for (int it = 0; it < steps; ++it) {
    const float ca = float(coeffs[3 * it]), cb = float(coeffs[3 * it + 1]), cc = float(coeffs[3 * it + 2]);
    if (int rc = i8m_bq_gemm(fp8, 0, a, sa, nullptr, a, sa, nullptr, gq, nullptr, sg, dg, B, lp, lp, hp, l,
                             l, 0, 0, 0, 0, 0, 0, c.status, c.stream))
      return rc;
    if (int rc = i8m_bq_gemm(fp8, 1, gq, sg, dg, gq, sg, nullptr, pq, nullptr, sp, dp, B, lp, lp, lp, l, l,
                             ca, cb, cc, 0, 0, 0, c.status, c.stream))
      return rc;
    const bool final = it == steps - 1;
    if (int rc = i8m_bq_gemm(fp8, 2, pq, sp, dp, at, sa, a, final ? c.out : static_cast<void*>(y),
                             final ? nullptr : yt, final ? nullptr : sy, nullptr, B, lp, hp, lp, l, h, 0,
                             0, 0, final, transpose, c.dtype, c.status, c.stream))
      return rc;
    if (!final) { std::swap(a, y); std::swap(at, yt); std::swap(sa, sy); }
  }
  return 0;
}

int ns_dispatch(const NsCall& c, Bump& ws, bool plan) {
  if (c.batch < 1 || c.batch > 65535) return fail(I8M_E_ARGUMENT, "batch size must be between 1 and 65535");
  if (c.rows < 1 || c.cols < 1) return fail(I8M_E_ARGUMENT, "matrix dimensions must be positive");
  if (!float_dtype_ok(c.dtype)) return fail(I8M_E_ARGUMENT, "input must be float32, float16 or bfloat16");
  if (c.steps < 1) return fail(I8M_E_ARGUMENT, "at least one coefficient row is required");
  switch (c.route) {
    case I8M_ROUTE_FLOAT:
    case I8M_ROUTE_GRAM:
      if (!float_dtype_ok(c.compute)) return fail(I8M_E_ARGUMENT, "bad compute dtype %d", c.compute);
      return run_float(c, ws, plan, c.route == I8M_ROUTE_GRAM, c.x, c.out, c.dtype, c.steps, c.coeffs,
                       c.compute, true);
    case I8M_ROUTE_INT8_FACTORED: {
      // completed-square rows (c, p, q), src/i8muon/_cutlass.py:93-128
      if (!c.fp16_first) return run_int8(c, ws, plan, c.x, c.steps, c.coeffs, true, true);
      if (c.steps == 1)
        return run_float(c, ws, plan, false, c.x, c.out, c.dtype, 1, c.coeffs, I8M_F16, true, true);
      void* first = ws.take(size_t(c.batch) * c.rows * c.cols * dtype_size(c.dtype));
      size_t mark = ws.used;
      if (int rc = run_float(c, ws, plan, false, c.x, first, c.dtype, 1, c.coeffs, I8M_F16, true, true)) return rc;
      size_t after_float = ws.used;
      ws.used = mark;
      int rc = run_int8(c, ws, plan, first, c.steps - 1, plan ? nullptr : c.coeffs + 3, false, true);
      ws.used = std::max(ws.used, after_float);
      return rc;
    }
    case I8M_ROUTE_INT8:
    case I8M_ROUTE_BQ_INT8: {
      const bool bq = c.route == I8M_ROUTE_BQ_INT8;
      if (!c.fp16_first)
        return bq ? run_bq(c, ws, plan, false, c.x, c.steps, c.coeffs, true)
                  : run_int8(c, ws, plan, c.x, c.steps, c.coeffs, true);
      // First row in FP16 with its result rounded to the input dtype, then the
      // quantised rows without re-normalising (src/i8muon/_cutlass.py:137-142).
      if (c.steps == 1)
        return run_float(c, ws, plan, false, c.x, c.out, c.dtype, 1, c.coeffs, I8M_F16, true);
      if (bq && c.fuse_first_row) {
        // The first row's update product quantises its own result (the CTA tile is the quantisation
        // block): no 16-bit intermediate in HBM, no standalone quantisation pass.
        const int l = std::min(c.rows, c.cols), h = std::max(c.rows, c.cols);
        BqOperands ops;
        ops.lp = pad_to(l, 128); ops.hp = pad_to(h, 128);
        const size_t wide = size_t(c.batch) * ops.lp * ops.hp;
        ops.a = ws.take_n<uint8_t>(wide);
        ops.at = ws.take_n<uint8_t>(wide);
        ops.sa = ws.take_n<float>(size_t(c.batch) * (ops.lp / 128) * (ops.hp / 128));
        const size_t mark = ws.used;
        if (int rc = run_float(c, ws, plan, false, c.x, nullptr, c.dtype, 1, c.coeffs, I8M_F16, true, false, &ops)) return rc;
        const size_t after_float = ws.used;
        ws.used = mark;  // the quantised rows reuse the floating stage's scratch
        const int rc = run_bq(c, ws, plan, false, nullptr, c.steps - 1, plan ? nullptr : c.coeffs + 3, false, &ops);
        ws.used = std::max(ws.used, after_float);
        return rc;
      }
      void* first = ws.take(size_t(c.batch) * c.rows * c.cols * dtype_size(c.dtype));
      // global INT8: the first row's final store also leaves max |X1| per matrix, the scale of the rows
      // that follow (deterministic: a maximum does not depend on the order of its operands)
      float* first_amax = bq ? nullptr : ws.take_n<float>(c.batch);
      size_t mark = ws.used;
      if (!plan && first_amax) CUDA_TRY(cudaMemsetAsync(first_amax, 0, size_t(c.batch) * sizeof(float), c.stream));
      if (int rc = run_float(c, ws, plan, false, c.x, first, c.dtype, 1, c.coeffs, I8M_F16, true, false, nullptr,
                             first_amax))
        return rc;
      size_t after_float = ws.used;
      ws.used = mark;  // the quantised stage reuses the floating stage's scratch
      int rc = bq ? run_bq(c, ws, plan, false, first, c.steps - 1, plan ? nullptr : c.coeffs + 3, false)
                  : run_int8(c, ws, plan, first, c.steps - 1, plan ? nullptr : c.coeffs + 3, false, false, first_amax);
      ws.used = std::max(ws.used, after_float);
      return rc;
    }
    case I8M_ROUTE_BQ_FP8:
      return run_bq(c, ws, plan, true, c.x, c.steps, c.coeffs, true);
    case I8M_ROUTE_INT8_CUBIC:
      return run_int8_cubic(c, ws, plan);
    default:
      return fail(I8M_E_ARGUMENT, "unknown route %d", c.route);
  }
}

}  // namespace

extern "C" int i8m_ns_workspace_bytes(int route, int batch, int rows, int cols, int dtype,
                                      int compute, int steps, int fp16_first, size_t* bytes) {
  if (!bytes) return fail(I8M_E_ARGUMENT, "ns_workspace_bytes: null result pointer");
  NsCall c{};
  c.route = route; c.dtype = dtype; c.batch = batch; c.rows = rows; c.cols = cols;
  c.compute = compute; c.steps = steps; c.fp16_first = fp16_first;
  Bump ws(nullptr, ~size_t(0), true);
  if (int rc = ns_dispatch(c, ws, true)) return rc;
  *bytes = align256(ws.used);
  return 0;
}

extern "C" int i8m_ns_run(int route, const void* x, void* out, int dtype, int batch, int rows,
                          int cols, int compute, const double* coeffs, int steps, float eps,
                          int fp16_first, int deterministic, int variants, const char* gram_order,
                          const float* stats_partials, void* workspace, size_t workspace_bytes, uint32_t* status,
                          i8m_stream_t stream) {
  if (!x || !out || !coeffs || !workspace || !status) return fail(I8M_E_ARGUMENT, "ns_run: null pointer");
  if (x == out) return fail(I8M_E_ARGUMENT, "ns_run: out may not alias x");
  if ((reinterpret_cast<uintptr_t>(workspace) & 255u) != 0)
    return fail(I8M_E_ARGUMENT, "ns_run: workspace must be 256-byte aligned");
  size_t need = 0;
  if (int rc = i8m_ns_workspace_bytes(route, batch, rows, cols, dtype, compute, steps, fp16_first, &need)) return rc;
  if (workspace_bytes < need)
    return fail(I8M_E_WORKSPACE, "ns_run: workspace %zu < %zu bytes", workspace_bytes, need);
  NsCall c{};
  c.route = route; c.dtype = dtype; c.batch = batch; c.rows = rows; c.cols = cols;
  c.compute = compute; c.steps = steps; c.fp16_first = fp16_first;
  c.x = x; c.out = out; c.coeffs = coeffs; c.eps = eps; c.gram_order = gram_order;
  c.status = status; c.stream = S(stream);
  c.deterministic = deterministic ? 1 : 0;
  c.stats_partials = stats_partials;
  Bump ws(workspace, workspace_bytes, false);
  if (variants < 0) return ns_dispatch(c, ws, false);
  // this call's own kernel selection; the thread's setting comes back whatever happens
  const int bq = variants & 0xff, wholek = (variants >> 8) & 0xff;
  const int wk_square = (variants >> 16) & 0xff, wk_update = (variants >> 24) & 0x7f;
  if (bq >= BQ_VARIANTS || wholek >= WHOLEK_VARIANTS || wk_square >= WHOLEK_VARIANTS || wk_update >= WHOLEK_VARIANTS)
    return fail(I8M_E_ARGUMENT, "ns_run: unknown kernel variant 0x%x", variants);
  const int saved_bq = g_bq_variant, saved_wholek = g_wholek_variant;
  g_bq_variant = bq;
  g_wholek_variant = wholek;
  c.wholek[0] = wholek; c.wholek[1] = wk_square; c.wholek[2] = wk_update;
  const int rc = ns_dispatch(c, ws, false);
  g_bq_variant = saved_bq;
  g_wholek_variant = saved_wholek;
  return rc;
}

// ================================================= one shape group of a step
namespace {
struct GroupLayout { size_t update, ortho, stats, workspace, workspace_bytes, total; long long numel; int batch; };
int group_layout(const i8m_group_plan* p, GroupLayout& l) {
  if (!p || p->count < 1 || p->leading < 1 || p->rows < 1 || p->cols < 1 || !float_dtype_ok(p->grad_dtype))
    return fail(I8M_E_ARGUMENT, "group: bad plan");
  const long long batch = (long long)p->count * p->leading;
  if (batch > 65535) return fail(I8M_E_ARGUMENT, "batch size must be between 1 and 65535");
  l.batch = int(batch);
  l.numel = (long long)p->leading * p->rows * p->cols;
  const size_t stacked = align256(size_t(p->count) * size_t(l.numel) * dtype_size(p->grad_dtype));
  size_t stats = 0;
  if (p->use_stats)
    if (int rc = i8m_stats_scratch_bytes(p->count, l.numel, &stats)) return rc;
  if (int rc = i8m_ns_workspace_bytes(p->route, l.batch, p->rows, p->cols, p->grad_dtype, p->compute, p->steps,
                                      p->fp16_first, &l.workspace_bytes))
    return rc;
  l.update = 0; l.ortho = stacked; l.stats = 2 * stacked; l.workspace = l.stats + align256(stats);
  l.total = l.workspace + l.workspace_bytes;
  return 0;
}
}  // namespace

extern "C" int i8m_group_bytes(const i8m_group_plan* plan, size_t* bytes) {
  if (!bytes) return fail(I8M_E_ARGUMENT, "group_bytes: null result pointer");
  GroupLayout l;
  if (int rc = group_layout(plan, l)) return rc;
  *bytes = l.total;
  return 0;
}

extern "C" int i8m_group_step(const i8m_group_plan* plan, const void* const* grads, void* const* bufs,
                              void* const* params, void* block, size_t block_bytes, float buf_weight, float mu,
                              float decay, float neg_lr, i8m_stream_t stream) {
  GroupLayout l;
  if (int rc = group_layout(plan, l)) return rc;
  if (!block || (reinterpret_cast<uintptr_t>(block) & 255u) != 0)
    return fail(I8M_E_ARGUMENT, "group_step: the block must be 256-byte aligned");
  if (block_bytes < l.total) return fail(I8M_E_WORKSPACE, "group_step: block %zu < %zu bytes", block_bytes, l.total);
  char* base = static_cast<char*>(block);
  float* stats = plan->use_stats ? reinterpret_cast<float*>(base + l.stats) : nullptr;
  if (int rc = i8m_momentum(grads, bufs, plan->count, base + l.update, l.numel, plan->grad_dtype, buf_weight, mu,
                            plan->nesterov, stats, stream))
    return rc;
  if (int rc = i8m_ns_run(plan->route, base + l.update, base + l.ortho, plan->grad_dtype, l.batch, plan->rows, plan->cols,
                          plan->compute, plan->coeffs, plan->steps, plan->eps, plan->fp16_first, plan->deterministic,
                          plan->variants, plan->gram_order, stats, base + l.workspace, l.workspace_bytes,
                          plan->status_device, stream))
    return rc;
  return apply_updates(params, plan->count, base + l.ortho, l.numel, plan->param_dtype, plan->grad_dtype,
                       plan->decay_mode, decay, neg_lr, plan->status_host ? plan->status_device : nullptr,
                       plan->status_host, S(stream));
}
