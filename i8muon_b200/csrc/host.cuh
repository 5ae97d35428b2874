// Host-side helpers shared by the translation units of the C ABI: error reporting, launches, tensor-map
// encoding and the per-thread kernel selection.  No device memory is allocated anywhere in the library.
#pragma once
#include "../../include/i8muon_b200.h"
#include "gemm_core.cuh"

#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <utility>

namespace i8m {

// Kernel selection is per calling thread: two engines on two threads (or two devices driven
// from two threads) never see each other's choice.  i8m_ns_run additionally takes the
// selection as an argument and restores the thread's own setting when it returns.
extern thread_local char g_error[512];
extern thread_local int g_debug_simt;
extern thread_local int g_starve_producers;   // test hook: see bq_produce
extern thread_local int g_wholek_variant;     // "wholek_gemm": 0 units of 128 x 256, 1 two streams of 128 x 128 tiles, 2 one CTA per tile
extern thread_local int g_cta_limit;          // persistent GEMM kernels launch at most this many CTAs (0: one per SM)
// block-quantised GEMMs: 0 = split kernel (tail on its own warps, four-stage ring), 1 = fused tail with a
// six-stage ring, 2 = fused tail with a four-stage ring; the host-side tuner chooses per shape
extern thread_local int g_bq_variant;
extern std::atomic<unsigned long long> g_launches;
constexpr int WHOLEK_VARIANTS = 3;
constexpr int BQ_VARIANTS = 3;

int fail(int code, const char* fmt, ...);   // records the message of i8m_last_error and returns the code
#define CUDA_TRY(expr)                                                              \
  do {                                                                              \
    cudaError_t e_ = (expr);                                                        \
    if (e_ != cudaSuccess)                                                          \
      return fail(I8M_E_CUDA, "%s failed: %s", #expr, cudaGetErrorString(e_));      \
  } while (0)
#define LAUNCH_CHECK(name)                                                          \
  do {                                                                              \
    cudaError_t e_ = cudaGetLastError();                                            \
    if (e_ != cudaSuccess)                                                          \
      return fail(I8M_E_CUDA, "launch of %s failed: %s", name, cudaGetErrorString(e_)); \
    g_launches.fetch_add(1, std::memory_order_relaxed);                             \
  } while (0)

// Every kernel is launched with programmatic stream serialisation: it may become resident while its
// predecessor in the stream still runs and waits on the device (pdl_wait) before it touches global memory, so
// launch latency and the prologue lie under the predecessor's tail.  The caller's LAUNCH_CHECK reads the error.
template <typename... P, typename... A>
inline void launch_clusters(void (*kernel)(P...), unsigned cluster, dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                            A&&... args) {
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[0].val.programmaticStreamSerializationAllowed = 1;
  attributes[1].id = cudaLaunchAttributeClusterDimension;
  attributes[1].val.clusterDim.x = cluster; attributes[1].val.clusterDim.y = 1; attributes[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = grid; config.blockDim = block; config.dynamicSmemBytes = smem; config.stream = stream;
  config.attrs = attributes; config.numAttrs = cluster > 1 ? 2 : 1;
  cudaLaunchKernelEx(&config, kernel, P(args)...);
}
template <typename... P, typename... A>
inline void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  launch_clusters(kernel, 1, grid, block, smem, stream, std::forward<A>(args)...);
}
// Dynamic shared memory above 48 KB is allowed once per kernel and device, not once per launch.
struct SmemAllowed { std::atomic<unsigned long long> devices{0}; };
template <typename K>
int allow_smem(SmemAllowed& done, K* kernel, size_t bytes) {
  int device = 0;
  CUDA_TRY(cudaGetDevice(&device));
  const unsigned long long bit = device < 64 ? 1ull << device : 0ull;
  if (done.devices.load(std::memory_order_acquire) & bit) return 0;
  CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)));
  done.devices.fetch_or(bit, std::memory_order_release);
  return 0;
}

inline cudaStream_t S(i8m_stream_t s) { return static_cast<cudaStream_t>(s); }
inline int cdiv(long long a, long long b) { return int((a + b - 1) / b); }
inline int pad_to(int v, int a) { return (v + a - 1) / a * a; }
inline size_t align256(size_t v) { return (v + 255) & ~size_t(255); }

// 3-D map over a row-major operand.  K-major: (batch, extent, k), box {128 bytes of K, 128 rows, 1}; MN-major:
// (batch, k, extent), box {128 bytes along the extent, one K block of rows, 1}.  What lies beyond the tensor reads as zero.
int make_operand_map(CUtensorMap* map, const void* ptr, int esize, int k, int extent, int batch, int mn = 0);
int sm_count();   // of the current device, capped by i8m_set_cta_limit

inline bool float_dtype_ok(int d) { return d == I8M_F32 || d == I8M_F16 || d == I8M_BF16; }
inline size_t dtype_size(int d) { return d == I8M_F32 ? 4 : 2; }

// dtype dispatch helpers for the memory-bound passes
#define DISPATCH_IN(dtype, In, ...)                                  \
  do {                                                               \
    if ((dtype) == I8M_F32) { using In = float; __VA_ARGS__; }       \
    else if ((dtype) == I8M_F16) { using In = __half; __VA_ARGS__; } \
    else { using In = __nv_bfloat16; __VA_ARGS__; }                  \
  } while (0)

}  // namespace i8m
