// C ABI: statistics, prologues, re-quantisers and the optimizer kernels (the memory-bound passes).
#include "host.cuh"
#include "passes.cuh"
#include "drivers.cuh"

#include <mutex>

using namespace i8m;

// ================================================================== stats
extern "C" int i8m_stats_scratch_bytes(int batch, long long count, size_t* bytes) {
  if (batch < 1 || count < 1 || !bytes) return fail(I8M_E_ARGUMENT, "stats_scratch_bytes: bad argument");
  if (count / STATS_CHUNK >= 0x7fffffffLL) return fail(I8M_E_LIMIT, "stats_scratch_bytes: count %lld is too large", count);
  *bytes = size_t(2) * batch * size_t(count / STATS_CHUNK + (count % STATS_CHUNK != 0)) * sizeof(float);
  return 0;
}
extern "C" int i8m_stats(const void* x, int dtype, int batch, long long count, void* scratch,
                         size_t scratch_bytes, float* norm, float* amax, i8m_stream_t stream) {
  if (!x || !scratch || batch < 1 || batch > 65535 || count < 1 || !float_dtype_ok(dtype))
    return fail(I8M_E_ARGUMENT, "stats: bad argument");
  if (count / STATS_CHUNK >= 0x7fffffffLL) return fail(I8M_E_LIMIT, "stats: count %lld is too large", count);
  const int chunks = int(count / STATS_CHUNK + (count % STATS_CHUNK != 0));
  size_t need = size_t(2) * batch * chunks * sizeof(float);
  if (scratch_bytes < need) return fail(I8M_E_WORKSPACE, "stats: scratch %zu < %zu bytes", scratch_bytes, need);
  float* psum = static_cast<float*>(scratch);
  float* pmax = psum + size_t(batch) * chunks;
  DISPATCH_IN(dtype, In, (launch(stats_partial_kernel<In>, dim3(chunks, batch), STATS_THREADS, 0, S(stream),
                             static_cast<const In*>(x), psum, pmax, count, chunks)));
  LAUNCH_CHECK("stats_partial");
  launch(stats_final_kernel, batch, STATS_THREADS, 0, S(stream), psum, pmax, norm, amax, chunks);
  LAUNCH_CHECK("stats_final");
  return 0;
}

// One launch, atomics, summation order not reproducible (the reference's deterministic=False path).
extern "C" int i8m_stats_onepass(const void* x, int dtype, int batch, long long count, void* scratch,
                                 size_t scratch_bytes, float* norm, float* amax, i8m_stream_t stream) {
  if (!x || !scratch || batch < 1 || batch > 65535 || count < 1 || !float_dtype_ok(dtype))
    return fail(I8M_E_ARGUMENT, "stats_onepass: bad argument");
  if (count / STATS_CHUNK >= 0x7fffffffLL) return fail(I8M_E_LIMIT, "stats_onepass: count %lld is too large", count);
  const int chunks = int(count / STATS_CHUNK + (count % STATS_CHUNK != 0));
  const size_t need = size_t(3) * batch * sizeof(float);
  if (scratch_bytes < need) return fail(I8M_E_WORKSPACE, "stats_onepass: scratch %zu < %zu bytes", scratch_bytes, need);
  CUDA_TRY(cudaMemsetAsync(scratch, 0, need, S(stream)));
  float* sumsq = static_cast<float*>(scratch);
  unsigned* bits = reinterpret_cast<unsigned*>(sumsq + batch);
  unsigned* arrived = bits + batch;
  DISPATCH_IN(dtype, In, (launch(stats_onepass_kernel<In>, dim3(chunks, batch), STATS_THREADS, 0, S(stream),
                             static_cast<const In*>(x), sumsq, bits, arrived, norm, amax, count, chunks)));
  LAUNCH_CHECK("stats_onepass");
  return 0;
}

// ------------------------------------------------------ stats without allocation
// Scratch for i8m_stats_static lives in the library image: 2^20 floats (4 MiB) per GPU
// that loads the library, held until the process exits.
constexpr size_t STATIC_SCRATCH_FLOATS = size_t(1) << 20;
static __device__ __align__(256) float g_static_stats_scratch[STATIC_SCRATCH_FLOATS];
namespace {
constexpr int MAX_DEVICES = 64;
float* g_static_scratch_ptr[MAX_DEVICES] = {};
std::mutex g_static_scratch_mutex;
}  // namespace

extern "C" int i8m_stats_static(const void* x, int dtype, int batch, long long count, float* norm,
                                float* amax, i8m_stream_t stream) {
  if (!x || batch < 1 || batch > 65535 || count < 1 || !float_dtype_ok(dtype))
    return fail(I8M_E_ARGUMENT, "stats_static: bad argument");
  // no sum or product here can wrap: chunks is compared with the limit before it is multiplied
  const long long chunks = count / STATS_CHUNK + (count % STATS_CHUNK != 0);
  if (chunks > (long long)(STATIC_SCRATCH_FLOATS / 2) / batch)
    return fail(I8M_E_LIMIT,
                "stats_static: batch * ceil(count / 8192) = %lld exceeds the built-in scratch of %zu "
                "partials; use i8m_stats with caller scratch",
                (long long)batch * chunks, STATIC_SCRATCH_FLOATS / 2);
  int device = -1;
  CUDA_TRY(cudaGetDevice(&device));
  if (device < 0 || device >= MAX_DEVICES) return fail(I8M_E_LIMIT, "stats_static: device index %d", device);
  float* scratch = nullptr;
  {
    // First call on this device: resolve the device address of the array.  In host
    // code the array's name is only a handle, never a pointer a kernel may use.
    std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
    if (!g_static_scratch_ptr[device]) {
      void* address = nullptr;
      CUDA_TRY(cudaGetSymbolAddress(&address, g_static_stats_scratch));
      g_static_scratch_ptr[device] = static_cast<float*>(address);
    }
    scratch = g_static_scratch_ptr[device];
  }
  // Every partial that the second pass reads is written by the first pass of the
  // same call, so nothing left over from an earlier call needs clearing.
  float* psum = scratch;
  float* pmax = scratch + size_t(batch) * chunks;
  DISPATCH_IN(dtype, In, (launch(stats_partial_kernel<In>, dim3(unsigned(chunks), batch), STATS_THREADS, 0, S(stream),
                             static_cast<const In*>(x), psum, pmax, count, int(chunks))));
  LAUNCH_CHECK("stats_partial(static)");
  launch(stats_final_kernel, batch, STATS_THREADS, 0, S(stream), psum, pmax, norm, amax, int(chunks));
  LAUNCH_CHECK("stats_final(static)");
  return 0;
}

extern "C" int i8m_normalize(const void* x, int in_dtype, const float* norm, void* a, void* a_t,
                             void* a_lo, void* a_t_lo, int compute, int batch, int rows, int cols,
                             int lp, int hp, int transpose, float eps, i8m_stream_t stream) {
  if (!x || !a || !float_dtype_ok(in_dtype) || !float_dtype_ok(compute) || batch < 1 || batch > 65535)
    return fail(I8M_E_ARGUMENT, "normalize: bad argument");
  if (compute == I8M_F32 && (!a_lo || (a_t && !a_t_lo)))
    return fail(I8M_E_ARGUMENT, "normalize: FP32 compute needs the low planes");
  // grid in the input's orientation, covering the padded extent
  const int prow = transpose ? hp : lp, pcol = transpose ? lp : hp;
  dim3 grid(cdiv(pcol, 32), cdiv(prow, 32), batch);
#define NORM_LAUNCH(E)                                                                         \
  DISPATCH_IN(in_dtype, In, (launch(normalize_kernel<In, E>, grid, 256, 0, S(stream),              \
                                static_cast<const In*>(x), norm, static_cast<E*>(a),           \
                                static_cast<E*>(a_t), static_cast<float*>(a_lo),               \
                                static_cast<float*>(a_t_lo), rows, cols, lp, hp, transpose, eps)))
  if (a_t == nullptr && !transpose && compute != I8M_F32 && hp % 8 == 0 && (reinterpret_cast<uintptr_t>(a) & 15u) == 0) {
    // no transposed copy: a plain element-wise pass
    const bool vectors = (size_t(cols) * dtype_size(in_dtype)) % 16 == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
    const long long groups = (long long)lp * (hp / 8);
    const dim3 rgrid(unsigned(std::min<long long>(cdiv(groups, 256), std::max(1, 148 * 32 / batch))), batch);
#define NORM_ROWS(In, E)                                                                                              \
  do {                                                                                                                \
    if (vectors)                                                                                                      \
      launch(normalize_rows_kernel<In, E, true>, rgrid, 256, 0, S(stream), static_cast<const In*>(x), norm,           \
             static_cast<E*>(a), rows, cols, lp, hp, eps);                                                            \
    else                                                                                                              \
      launch(normalize_rows_kernel<In, E, false>, rgrid, 256, 0, S(stream), static_cast<const In*>(x), norm,          \
             static_cast<E*>(a), rows, cols, lp, hp, eps);                                                            \
  } while (0)
    if (compute == I8M_F16) DISPATCH_IN(in_dtype, In, NORM_ROWS(In, __half));
    else DISPATCH_IN(in_dtype, In, NORM_ROWS(In, __nv_bfloat16));
#undef NORM_ROWS
    LAUNCH_CHECK("normalize");
    return 0;
  }
  // 16-bit out, rows of whole 16-byte vectors: the vectorised kernel
  const bool vec = compute != I8M_F32 && cols % 8 == 0 && lp % 8 == 0 && hp % 8 == 0 &&
                   ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(a) |
                     reinterpret_cast<uintptr_t>(a_t)) & 15u) == 0;
  if (vec) {
    dim3 vgrid(cdiv(pcol, 64), cdiv(prow, 64), batch);
#define NORM_VEC(In, E)                                                                              \
  launch(normalize_vec_kernel<In, E>, vgrid, 256, 0, S(stream), static_cast<const In*>(x), norm,         \
                                                            static_cast<E*>(a), static_cast<E*>(a_t), \
                                                            rows, cols, lp, hp, transpose, eps)
    if (in_dtype == I8M_F32 && compute == I8M_F16) NORM_VEC(float, __half);
    else if (in_dtype == I8M_F32) NORM_VEC(float, __nv_bfloat16);
    else if (in_dtype == I8M_F16 && compute == I8M_F16) NORM_VEC(__half, __half);
    else if (in_dtype == I8M_F16) NORM_VEC(__half, __nv_bfloat16);
    else if (compute == I8M_F16) NORM_VEC(__nv_bfloat16, __half);
    else NORM_VEC(__nv_bfloat16, __nv_bfloat16);
#undef NORM_VEC
  } else if (compute == I8M_F32) NORM_LAUNCH(float);
  else if (compute == I8M_F16) NORM_LAUNCH(__half);
  else NORM_LAUNCH(__nv_bfloat16);
#undef NORM_LAUNCH
  LAUNCH_CHECK("normalize");
  return 0;
}

namespace {
// One CTA-sized piece of an elementwise pass: grid-stride, about eight waves at most.
unsigned flat_blocks(long long quads) { return unsigned(std::min<long long>(cdiv(quads, 1024), 8LL * 148)); }

// a8 or a8_t may be null: only the other one is written then
int input_quant_any(const void* x, int in_dtype, const float* amax, const float* norm, int8_t* a8, int8_t* a8_t, float* a_scale,
                    int batch, int rows, int cols, int lp, int hp, int transpose, float eps, cudaStream_t stream) {
  const int prow = transpose ? hp : lp, pcol = transpose ? lp : hp;
  int8_t* same = transpose ? a8_t : a8;
  int8_t* other = transpose ? a8 : a8_t;
  const bool aligned = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(a8) | reinterpret_cast<uintptr_t>(a8_t)) & 15u) == 0;
  const bool unpadded = rows == prow && cols == pcol && aligned;
  const float e = norm ? eps : 0.f;
  if (unpadded && other == nullptr) {
    const long long quads = (long long)rows * cols / 4;
    DISPATCH_IN(in_dtype, In, (launch(input_quant_flat_kernel<In>, dim3(flat_blocks(quads), batch), 256, 0, stream,
                                  static_cast<const In*>(x), amax, norm, reinterpret_cast<uint32_t*>(same), a_scale, quads, e, 0)));
  } else if (unpadded && rows % 128 == 0 && cols % 128 == 0) {
    // whole 128 x 128 tiles: vector loads, packed stores, transposes in registers
    DISPATCH_IN(in_dtype, In, (launch(input_quant128_kernel<In>, dim3(cols / 128, rows / 128, batch), 256, 0, stream,
                                  static_cast<const In*>(x), amax, norm, same, other, a_scale, rows, cols, e)));
  } else {
    dim3 grid(cdiv(pcol, 32), cdiv(prow, 32), batch);
    DISPATCH_IN(in_dtype, In, (launch(input_quant_kernel<In>, grid, 256, 0, stream, static_cast<const In*>(x), amax, norm,
                                  a8, a8_t, a_scale, rows, cols, lp, hp, transpose, e)));
  }
  LAUNCH_CHECK("input_quant");
  return 0;
}
}  // namespace
int i8m::input_quant(const void* x, int in_dtype, const float* amax, const float* norm, int8_t* a8, float* a_scale, int batch,
                     int rows, int cols, int lp, int hp, int transpose, float eps, cudaStream_t stream) {
  return input_quant_any(x, in_dtype, amax, norm, a8, nullptr, a_scale, batch, rows, cols, lp, hp, transpose, eps, stream);
}
int i8m::output_quant(const float* input, const float* maximum, int8_t* out, float* scale, int batch, int m, int n,
                      cudaStream_t stream) {
  const long long quads = (long long)m * n / 4;   // m and n are padded to multiples of 16
  launch(input_quant_flat_kernel<float>, dim3(flat_blocks(quads), batch), 256, 0, stream, input, maximum,
         static_cast<const float*>(nullptr), reinterpret_cast<uint32_t*>(out), scale, quads, 0.f, 1);
  LAUNCH_CHECK("output_quant");
  return 0;
}
extern "C" int i8m_input_quant(const void* x, int in_dtype, const float* amax, const float* norm,
                               int8_t* a8, int8_t* a8_t, float* a_scale, int batch, int rows,
                               int cols, int lp, int hp, int transpose, float eps,
                               i8m_stream_t stream) {
  if (!x || !amax || !a8 || !a8_t || !a_scale || !float_dtype_ok(in_dtype) || batch < 1 || batch > 65535)
    return fail(I8M_E_ARGUMENT, "input_quant: bad argument");
  return input_quant_any(x, in_dtype, amax, norm, a8, a8_t, a_scale, batch, rows, cols, lp, hp, transpose, eps, S(stream));
}

extern "C" int i8m_symmetric_quant(const void* input, const void* maximum, const float* orig_scale,
                                   const float* orig_diag, int8_t* output, float* scale, float* diag,
                                   int batch, int m, int quad, float c0, float c1, float c2,
                                   i8m_stream_t stream) {
  if (!input || !maximum || !orig_scale || !output || !scale || !diag || batch < 1 || batch > 65535 || m < 1)
    return fail(I8M_E_ARGUMENT, "symmetric_quant: bad argument");
  if (quad && !orig_diag) return fail(I8M_E_ARGUMENT, "symmetric_quant: quad needs the previous diagonal");
  if (m % 128 == 0 && ((reinterpret_cast<uintptr_t>(input) | reinterpret_cast<uintptr_t>(output)) & 15u) == 0) {
    const int t128 = m / 128;
    dim3 grid128(t128 * (t128 + 1) / 2, batch);
    if (quad)
      launch(symmetric_quant128_kernel<float, true>, grid128, 256, 0, S(stream),
          static_cast<const float*>(input), maximum, orig_scale, orig_diag, output, scale, diag, m, c0, c1, c2);
    else
      launch(symmetric_quant128_kernel<int, false>, grid128, 256, 0, S(stream),
          static_cast<const int*>(input), maximum, orig_scale, orig_diag, output, scale, diag, m, c0, c1, c2);
    LAUNCH_CHECK("symmetric_quant");
    return 0;
  }
  const int t = cdiv(m, 32);
  dim3 grid(t * (t + 1) / 2, batch);
  if (quad)
    launch(symmetric_quant_kernel<float, true>, grid, 256, 0, S(stream),
        static_cast<const float*>(input), maximum, orig_scale, orig_diag, output, scale, diag, m, c0, c1, c2);
  else
    launch(symmetric_quant_kernel<int, false>, grid, 256, 0, S(stream),
        static_cast<const int*>(input), maximum, orig_scale, orig_diag, output, scale, diag, m, c0, c1, c2);
  LAUNCH_CHECK("symmetric_quant");
  return 0;
}

extern "C" int i8m_output_quant(const float* input, const float* maximum, int8_t* out, int8_t* out_t,
                                float* scale, int batch, int m, int n, i8m_stream_t stream) {
  if (!input || !maximum || !out || !out_t || !scale || batch < 1 || batch > 65535)
    return fail(I8M_E_ARGUMENT, "output_quant: bad argument");
  if (m % 128 == 0 && n % 128 == 0 &&
      ((reinterpret_cast<uintptr_t>(input) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(out_t)) & 15u) == 0) {
    launch(output_quant128_kernel, dim3(n / 128, m / 128, batch), 256, 0, S(stream), input, maximum, out, out_t, scale, m, n);
    LAUNCH_CHECK("output_quant");
    return 0;
  }
  dim3 grid(cdiv(n, 32), cdiv(m, 32), batch);
  launch(output_quant_kernel, grid, 256, 0, S(stream), input, maximum, out, out_t, scale, m, n);
  LAUNCH_CHECK("output_quant");
  return 0;
}

extern "C" int i8m_bq_quant(const void* x, int in_dtype, const float* norm, void* a, void* a_t,
                            float* scale, int fp8, int batch, int rows, int cols, int lp, int hp,
                            int transpose, float eps, i8m_stream_t stream) {
  if (!x || !a || !a_t || !scale || !float_dtype_ok(in_dtype) || batch < 1 || batch > 65535 ||
      lp % 128 || hp % 128)
    return fail(I8M_E_ARGUMENT, "bq_quant: bad argument");
  dim3 grid(lp / 128, hp / 128, batch);
  if (grid.y > 65535) return fail(I8M_E_LIMIT, "bq_quant: matrix too wide");
  const float e = norm ? eps : 0.f;
  const bool vec = in_dtype != I8M_F32 && cols % 8 == 0 &&
                   ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(a) |
                     reinterpret_cast<uintptr_t>(a_t)) & 15u) == 0;
  if (vec) {
#define BQ_VEC(In, F8)                                                                                  \
  launch(bq_quant_vec_kernel<In, F8>, grid, 256, 0, S(stream), static_cast<const In*>(x), norm,             \
                                                           static_cast<uint8_t*>(a),                    \
                                                           static_cast<uint8_t*>(a_t), scale, rows, cols, \
                                                           lp, hp, transpose, e)
    if (in_dtype == I8M_F16) { if (fp8) BQ_VEC(__half, true); else BQ_VEC(__half, false); }
    else { if (fp8) BQ_VEC(__nv_bfloat16, true); else BQ_VEC(__nv_bfloat16, false); }
#undef BQ_VEC
  } else if (fp8)
    DISPATCH_IN(in_dtype, In, (launch(bq_quant_kernel<In, true>, grid, 256, 0, S(stream),
                                  static_cast<const In*>(x), norm, static_cast<uint8_t*>(a),
                                  static_cast<uint8_t*>(a_t), scale, rows, cols, lp, hp, transpose, e)));
  else
    DISPATCH_IN(in_dtype, In, (launch(bq_quant_kernel<In, false>, grid, 256, 0, S(stream),
                                  static_cast<const In*>(x), norm, static_cast<uint8_t*>(a),
                                  static_cast<uint8_t*>(a_t), scale, rows, cols, lp, hp, transpose, e)));
  LAUNCH_CHECK("bq_quant");
  return 0;
}

// ====================================================== optimizer kernels
extern "C" int i8m_momentum(const void* const* grads, void* const* bufs, int count, void* update,
                            long long numel, int dtype, float buf_weight, float mu, int nesterov,
                            float* stats_partials, i8m_stream_t stream) {
  if (!grads || !bufs || !update || count < 1 || numel < 1 || !float_dtype_ok(dtype))
    return fail(I8M_E_ARGUMENT, "momentum: bad argument");
  if (numel / STATS_CHUNK >= 0x7fffffffLL) return fail(I8M_E_LIMIT, "momentum: tensor too large");
  const size_t es = dtype_size(dtype);
  const int chunks = int(numel / STATS_CHUNK + (numel % STATS_CHUNK != 0));
  const int blocks_x = std::min(chunks, 148 * 16);
  // stats_partials (optional): the scratch layout of i8m_stats over the stacked update,
  // [count][chunks] sums of squares followed by [count][chunks] maxima
  float* psum = stats_partials;
  float* pmax = stats_partials ? stats_partials + size_t(count) * chunks : nullptr;
  for (int first = 0; first < count; first += MT_MAX) {
    const int c = std::min(MT_MAX, count - first);
    MomentumTable tab;
    for (int i = 0; i < c; ++i) {
      if (!grads[first + i] || !bufs[first + i]) return fail(I8M_E_ARGUMENT, "momentum: null tensor");
      tab.grad[i] = grads[first + i];
      tab.buf[i] = bufs[first + i];
    }
    char* u = static_cast<char*>(update) + size_t(first) * numel * es;
    dim3 grid(blocks_x, c);
    DISPATCH_IN(dtype, T, (launch(momentum_kernel<T>, grid, 256, 0, S(stream),
                              tab, reinterpret_cast<T*>(u), numel, buf_weight, mu, nesterov, psum, pmax, chunks, first)));
    LAUNCH_CHECK("momentum");
  }
  return 0;
}

extern "C" int i8m_apply(void* const* params, int count, const void* update, long long numel,
                         int param_dtype, int update_dtype, int decay_mode, float decay,
                         float neg_lr, i8m_stream_t stream) {
  return apply_updates(params, count, update, numel, param_dtype, update_dtype, decay_mode, decay, neg_lr, nullptr,
                       nullptr, S(stream));
}
int i8m::apply_updates(void* const* params, int count, const void* update, long long numel, int param_dtype,
                       int update_dtype, int decay_mode, float decay, float neg_lr, const unsigned* status,
                       unsigned* status_host, cudaStream_t stream) {
  if (!params || !update || count < 1 || numel < 1 || !float_dtype_ok(param_dtype) ||
      !float_dtype_ok(update_dtype) || decay_mode < 0 || decay_mode > 2)
    return fail(I8M_E_ARGUMENT, "apply: bad argument");
  const size_t es = dtype_size(update_dtype);
  const int blocks_x = int(std::min<long long>(cdiv(numel, 256 * 8), 148 * 16));
  for (int first = 0; first < count; first += MT_MAX) {
    const int c = std::min(MT_MAX, count - first);
    ApplyTable tab;
    for (int i = 0; i < c; ++i) {
      if (!params[first + i]) return fail(I8M_E_ARGUMENT, "apply: null tensor");
      tab.param[i] = params[first + i];
    }
    const char* u = static_cast<const char*>(update) + size_t(first) * numel * es;
    dim3 grid(blocks_x, c);
#define APPLY_LAUNCH(P)                                                                        \
  DISPATCH_IN(update_dtype, U, (launch(apply_kernel<P, U>, grid, 256, 0, stream,                \
                                   tab, reinterpret_cast<const U*>(u), numel, decay_mode, decay, neg_lr, status, status_host)))
    if (param_dtype == I8M_F32) APPLY_LAUNCH(float);
    else if (param_dtype == I8M_F16) APPLY_LAUNCH(__half);
    else APPLY_LAUNCH(__nv_bfloat16);
#undef APPLY_LAUNCH
    LAUNCH_CHECK("apply");
  }
  return 0;
}

// AdamW companion for the parameters outside Muon; FP32 moments, parameters and gradients in
// any of the three floating types.  bias corrections are passed by the host (1 - beta^step).
extern "C" int i8m_adamw(void* const* params, const void* const* grads, float* const* exp_avg,
                         float* const* exp_avg_sq, const long long* numel, int count, int param_dtype,
                         int grad_dtype, float lr, float beta1, float beta2, float eps,
                         float weight_decay, float bias_correction1, float bias_correction2,
                         i8m_stream_t stream) {
  if (!params || !grads || !exp_avg || !exp_avg_sq || !numel || count < 1 || !float_dtype_ok(param_dtype) ||
      !float_dtype_ok(grad_dtype) || !(bias_correction1 > 0.f) || !(bias_correction2 > 0.f))
    return fail(I8M_E_ARGUMENT, "adamw: bad argument");
  const float decay = 1.f - lr * weight_decay;
  const float step_size = lr / bias_correction1;
  const float inv_bc2_sqrt = 1.f / sqrtf(bias_correction2);
  for (int first = 0; first < count; first += ADAM_MAX) {
    const int c = std::min(ADAM_MAX, count - first);
    AdamTable tab;
    long long longest = 0;
    for (int i = 0; i < c; ++i) {
      const int k = first + i;
      if (!params[k] || !grads[k] || !exp_avg[k] || !exp_avg_sq[k] || numel[k] < 1)
        return fail(I8M_E_ARGUMENT, "adamw: null tensor or empty tensor");
      tab.param[i] = params[k]; tab.grad[i] = grads[k];
      tab.exp_avg[i] = exp_avg[k]; tab.exp_avg_sq[i] = exp_avg_sq[k];
      tab.numel[i] = numel[k];
      longest = std::max(longest, numel[k]);
    }
    dim3 grid(unsigned(std::min<long long>(cdiv(longest, 256 * 4), 148 * 16)), c);
#define ADAM_LAUNCH(P)                                                                              \
  DISPATCH_IN(grad_dtype, G, (launch(adamw_kernel<P, G>, grid, 256, 0, S(stream), tab, decay, beta1, beta2, eps, \
                                                                              step_size, inv_bc2_sqrt)))
    if (param_dtype == I8M_F32) ADAM_LAUNCH(float);
    else if (param_dtype == I8M_F16) ADAM_LAUNCH(__half);
    else ADAM_LAUNCH(__nv_bfloat16);
#undef ADAM_LAUNCH
    LAUNCH_CHECK("adamw");
  }
  return 0;
}

// ------------------------------------------------------ small passes of the drivers
int i8m::fold_stats(const float* partials, int batch, long long count, float* norm, float* amax, cudaStream_t stream) {
  const int chunks = int(count / STATS_CHUNK + (count % STATS_CHUNK != 0));
  launch(stats_final_kernel, batch, STATS_THREADS, 0, stream, partials, partials + size_t(batch) * chunks, norm, amax, chunks);
  LAUNCH_CHECK("stats_final");
  return 0;
}
int i8m::add_diagonal(void* r, int compute, int batch, int m, int logical, float shift, cudaStream_t stream) {
  const unsigned blocks = unsigned(cdiv((long long)batch * logical, 256));
  if (compute == I8M_F16) launch(diag_add_kernel<__half>, blocks, 256, 0, stream, static_cast<__half*>(r), batch, m, logical, shift);
  else launch(diag_add_kernel<__nv_bfloat16>, blocks, 256, 0, stream, static_cast<__nv_bfloat16*>(r), batch, m, logical, shift);
  LAUNCH_CHECK("diag_add");
  return 0;
}
int i8m::clamp_divide(float* norm, int batch, float eps, float gain, cudaStream_t stream) {
  launch(clamp_divide_kernel, cdiv(batch, 256), 256, 0, stream, norm, batch, eps, gain);
  LAUNCH_CHECK("clamp_divide");
  return 0;
}
