// Launch templates of the GEMM kernels: one place that fills the geometry, encodes the operand maps and picks the
// kernel for an epilogue.
#pragma once
#include <climits>

#include "host.cuh"
#include "gemm_bq_persistent.cuh"
#include "gemm_bq_split.cuh"
#include "gemm_fp32_cluster.cuh"
#include "gemm_wholek_persistent.cuh"
#include "gemm_wholek_wide.cuh"

namespace i8m {

// Row blocks per group of the wide-unit order: as many as keep the group's left row blocks
// (128 rows x k bytes each) within 32 MB of L2; even, 8 to 64.
inline int wide_group(long long k_bytes) {
  const long long fit = (32LL << 20) / std::max<long long>(1, 128 * k_bytes);
  return int(std::min<long long>(64, std::max<long long>(8, fit))) & ~1;
}

// Whether the persistent whole-K kernel takes units of one tile (128 x 128) instead of two (128 x 256).  A K block costs
// about 540 cycles in a pair and 390 alone (both bound by what the SM takes in from L2: 48 and 32 KB at 89 bytes per
// cycle, the measured rate of such copies), a tile's epilogue about 2000 (an estimate), of which only the last one per CTA
// is not under another unit's K loop.  Pairs win when there are many; with few tiles the number of waves decides.
inline bool narrow_units(long long tiles, long long pairs, int k_blocks, int ctas) {
  const long long one = (tiles + ctas - 1) / ctas * k_blocks * 390 + 2000;
  const long long two = (pairs + ctas - 1) / ctas * k_blocks * 540 + 4000;
  return one < two;
}

// How many clusters of an FP32 kernel are resident at one time (asked once per device); 0 if none fits.
template <class K>
int resident_clusters(std::atomic<int> (&cache)[64], K* kernel, int cluster) {
  int device = 0, n = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) device = 0;
  if ((n = cache[device].load(std::memory_order_relaxed)) > 0) return n;
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeClusterDimension;
  attribute.val.clusterDim.x = unsigned(cluster); attribute.val.clusterDim.y = 1; attribute.val.clusterDim.z = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(unsigned(cluster)); config.blockDim = dim3(F32C_THREADS); config.dynamicSmemBytes = F32C_SMEM;
  config.attrs = &attribute; config.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &config) != cudaSuccess || n < 1) {
    cudaGetLastError();
    return 0;
  }
  cache[device].store(n, std::memory_order_relaxed);
  return n;
}

// FP32 products: K segments whose sums are added in order, and the CTAs that share a tile.
//
// One estimate serves both choices, in nanoseconds: waves of clusters, each the K blocks of one CTA (0.75 us, measured)
// and the end of a tile (about 5 us: prologue, sum, stores).  Measured for 1, 2, 4, 8 CTAs a tile, in us: 10 tiles x 64 K
// blocks 53.5, 30.3, 18.5, 13.9; 36 x 128 (Gram of 1024 x 4096) 100, 54, 59, 55; 144 x 128 107, 112, 147, 184; 156 x 192
// 339, 245, 222, 273: with few tiles a split fills the GPU, with a nearly empty last wave it evens the waves out,
// otherwise it only adds ends of tiles.
inline long long f32_estimate(long long tiles, int resident, int num_kb, int ctas) {
  return (tiles + resident - 1) / resident * ((num_kb + ctas - 1) / ctas * 750LL + 5000);
}
// How many segments the K blocks form: the split that one matrix alone would take.  A function of its extents only - not
// of the batch, and not of the device, whose clusters (74, 33 and 15 on the B200s measured: GPC sizes leave some SMs out)
// are constants here - because it decides the order of the sums and with it the bits of the result.
inline int f32_segments(long long tiles_per_matrix, int num_kb) {
  constexpr int RESIDENT[4] = {148, 74, 33, 15};
  int best = 1;
  long long cost = f32_estimate(tiles_per_matrix, RESIDENT[0], num_kb, 1);
  for (int i = 1; i < 4 && (1 << i) <= num_kb; ++i) {
    const long long c = f32_estimate(tiles_per_matrix, RESIDENT[i], num_kb, 1 << i);
    if (c < cost) { cost = c; best = 1 << i; }
  }
  return best;
}
struct F32Call {
  const CUtensorMap *a, *b, *a2, *b2;
  const GemmGeom* g;
  const FloatArgs* args;
  long long tiles;      // of the whole batch
  cudaStream_t stream;
};
// The best of SPLIT, SPLIT / 2 ... 1 CTAs per tile: `best` and `cost` come with those of the larger splits.  A cluster that
// the device does not offer is left out; one CTA per tile needs none.
template <int MODE, int SPLIT, int SEGMENTS>
int f32_best_split(const F32Call& c, int& best, long long& cost) {
  auto kernel = fp32_cluster_kernel<MODE, SPLIT, SEGMENTS>;
  static SmemAllowed allowed;
  static std::atomic<int> resident[64];
  if (int rc = allow_smem(allowed, kernel, F32C_SMEM)) return rc;
  const int n = resident_clusters(resident, kernel, SPLIT);
  if (n >= 1 && c.tiles * SPLIT <= 0x7fffffffLL) {
    const long long v = f32_estimate(c.tiles, n, c.g->num_kb, SPLIT);
    if (v <= cost) { cost = v; best = SPLIT; }
  }
  if constexpr (SPLIT > 1) return f32_best_split<MODE, SPLIT / 2, SEGMENTS>(c, best, cost);
  return 0;
}
template <int MODE, int SPLIT, int SEGMENTS>
int launch_f32_split(const F32Call& c, int split, const char* name) {
  if constexpr (SPLIT > 1)
    if (split != SPLIT) return launch_f32_split<MODE, SPLIT / 2, SEGMENTS>(c, split, name);
  launch_clusters(fp32_cluster_kernel<MODE, SPLIT, SEGMENTS>, SPLIT, dim3(unsigned(c.tiles * SPLIT)), F32C_THREADS, F32C_SMEM,
                  c.stream, *c.a, *c.b, *c.a2, *c.b2, *c.g, *c.args);
  LAUNCH_CHECK(name);
  return 0;
}
template <int MODE, int SEGMENTS>
int launch_f32_segments(const F32Call& c, const char* name) {
  int split = 1;
  long long cost = LLONG_MAX;
  if (int rc = f32_best_split<MODE, SEGMENTS, SEGMENTS>(c, split, cost)) return rc;
  return launch_f32_split<MODE, SEGMENTS, SEGMENTS>(c, split, name);
}
template <int MODE>
int launch_f32(const F32Call& c, const char* name) {
  switch (f32_segments(c.g->tiles_per_batch, c.g->num_kb)) {
    case 8: return launch_f32_segments<MODE, 8>(c, name);
    case 4: return launch_f32_segments<MODE, 4>(c, name);
    case 2: return launch_f32_segments<MODE, 2>(c, name);
    default: return launch_f32_segments<MODE, 1>(c, name);
  }
}

// One product: operands, extents and what the kernels need besides the epilogue's own arguments.
struct GemmCall {
  const void *a = nullptr, *a_lo = nullptr, *b = nullptr, *b_lo = nullptr;   // low planes: FP32 as two TF32 planes
  int a_mn = 0, b_mn = 0;       // operand stored with its rows along K (GemmGeom)
  int batch = 0, m = 0, n = 0, k = 0, lm = 0, ln = 0, sym = 0;
  unsigned* status = nullptr;
  cudaStream_t stream = nullptr;
};

template <class Epi>
int launch_gemm(const GemmCall& c, const typename Epi::Args& args, const char* name) {
  const int batch = c.batch, m = c.m, n = c.n, k = c.k, sym = c.sym;
  const cudaStream_t stream = c.stream;
  if (batch < 1 || m < 1 || n < 1 || k < 1) return fail(I8M_E_ARGUMENT, "%s: empty problem", name);
  if (!c.a || !c.b || !c.status) return fail(I8M_E_ARGUMENT, "%s: null operand or status pointer", name);
  if (sym && m != n) return fail(I8M_E_ARGUMENT, "%s: symmetric product needs m == n", name);
  if (c.a_mn && !c.b_mn) return fail(I8M_E_ARGUMENT, "%s: no kernel reads only the left operand across K", name);
  constexpr int ES = int(sizeof(typename Epi::Elem));
  constexpr int STAGE_BYTES = 2 * Epi::PARTS * TILE_BYTES;
  constexpr size_t SMEM = size_t(Epi::STAGES) * STAGE_BYTES + sizeof(Ctrl) + 1024;
  GemmGeom g{};
  g.batch = batch; g.m = m; g.n = n; g.k = k; g.lm = c.lm; g.ln = c.ln;
  g.tiles_m = cdiv(m, TILE); g.tiles_n = cdiv(n, TILE);
  g.sym = sym;
  g.a_mn = c.a_mn; g.b_mn = c.b_mn;
  g.tiles_per_batch = sym ? g.tiles_m * (g.tiles_m + 1) / 2 : g.tiles_m * g.tiles_n;
  g.num_kb = cdiv((long long)k * ES, 128);
  g.debug_simt = g_debug_simt | (g_starve_producers ? 0x100 : 0);
  g.group = wide_group((long long)k * ES);
  g.a_raw = c.a; g.b_raw = c.b; g.status = c.status;
  long long blocks = (long long)g.tiles_per_batch * batch;
  if (blocks > 0x7fffffffLL) return fail(I8M_E_LIMIT, "%s: too many tiles", name);
  CUtensorMap ma, mb, ma2, mb2;
  if (int rc = make_operand_map(&ma, c.a, ES, k, m, batch, c.a_mn)) return rc;
  if (int rc = make_operand_map(&mb, c.b, ES, k, n, batch, c.b_mn)) return rc;
  if (Epi::PARTS == 2) {
    if (!c.a_lo || !c.b_lo) return fail(I8M_E_ARGUMENT, "%s: missing low planes", name);
    if (c.a_mn || c.b_mn) return fail(I8M_E_ARGUMENT, "%s: two-plane operands are read along K only", name);
    if (int rc = make_operand_map(&ma2, c.a_lo, ES, k, m, batch)) return rc;
    if (int rc = make_operand_map(&mb2, c.b_lo, ES, k, n, batch)) return rc;
  } else {
    ma2 = ma; mb2 = mb;
  }
  // products that accumulate their whole K extent in tensor memory: persistent kernel
  if constexpr (!Epi::BLOCKQ && Epi::PARTS == 1 && Epi::PROMOTE_KB == 0) {
    if (!g_debug_simt && g_wholek_variant == 0) {
      constexpr size_t WSMEM = wholek_wide_smem_bytes<Epi>();
      auto wk = wholek_wide_kernel<Epi>;
      static SmemAllowed allowed;
      if (int rc = allow_smem(allowed, wk, WSMEM)) return rc;
      const long long pairs = (long long)wide_units_per_batch(g.tiles_m, g.tiles_n, sym) * batch;
      g.narrow = narrow_units(blocks, pairs, g.num_kb, sm_count());
      const long long units = g.narrow ? blocks : pairs;
      launch(wk, unsigned(std::min<long long>(units, sm_count())), WKW_THREADS, WSMEM, stream, ma, mb, g, args);
      LAUNCH_CHECK(name);
      return 0;
    }
    if (!g_debug_simt && g_wholek_variant == 1) {
      constexpr size_t PSMEM = size_t(WKP_STAGES) * 2 * TILE_BYTES + sizeof(Ctrl) + 1024;
      auto pk = wholek_persistent_kernel<Epi>;
      static SmemAllowed allowed;
      if (int rc = allow_smem(allowed, pk, PSMEM)) return rc;
      const unsigned grid = unsigned(std::min<long long>(blocks, sm_count()));
      launch(pk, grid, WKP_THREADS, PSMEM, stream, ma, mb, g, args);
      LAUNCH_CHECK(name);
      return 0;
    }
  }
  if constexpr (Epi::PARTS == 2) {
    if (!g_debug_simt) return launch_f32<Epi::STORE>(F32Call{&ma, &mb, &ma2, &mb2, &g, &args, blocks, stream}, name);
  }
  auto kernel = ns_gemm_kernel<Epi, true>;
  if constexpr (!Epi::BLOCKQ && Epi::PARTS == 1) {
    if (!g_debug_simt) kernel = ns_gemm_kernel<Epi, false>;
  }
  static SmemAllowed allowed[2];
  if (int rc = allow_smem(allowed[g_debug_simt != 0], kernel, SMEM)) return rc;
  launch(kernel, dim3(unsigned(blocks)), WarpLayout<Epi>::THREADS, SMEM, stream, ma, mb, ma2, mb2, g, args);
  LAUNCH_CHECK(name);
  return 0;
}

// Block-quantised GEMMs: persistent kernel, one CTA per SM (the debug core keeps the
// one-tile-per-CTA skeleton).
template <class Epi>
int launch_bq(const void* a, const void* bt, int batch, int m, int n, int k, int lm, int ln, int sym,
              unsigned* status, const typename Epi::Args& args, cudaStream_t stream, const char* name) {
  if (g_debug_simt) {
    GemmCall c;
    c.a = a; c.b = bt; c.batch = batch; c.m = m; c.n = n; c.k = k; c.lm = lm; c.ln = ln; c.sym = sym;
    c.status = status; c.stream = stream;
    return launch_gemm<Epi>(c, args, name);
  }
  if (batch < 1 || m < 1 || n < 1 || k < 1) return fail(I8M_E_ARGUMENT, "%s: empty problem", name);
  if (!a || !bt || !status) return fail(I8M_E_ARGUMENT, "%s: null operand or status pointer", name);
  if (sym && m != n) return fail(I8M_E_ARGUMENT, "%s: symmetric product needs m == n", name);
  GemmGeom g{};
  g.batch = batch; g.m = m; g.n = n; g.k = k; g.lm = lm; g.ln = ln;
  g.tiles_m = cdiv(m, TILE); g.tiles_n = cdiv(n, TILE);
  g.sym = sym;
  g.tiles_per_batch = sym ? g.tiles_m * (g.tiles_m + 1) / 2 : g.tiles_m * g.tiles_n;
  g.num_kb = cdiv(k, 128);
  g.debug_simt = g_starve_producers ? 0x100 : 0;
  g.group = wide_group(k);
  g.a_raw = a; g.b_raw = bt; g.status = status;
  const long long tiles = (long long)g.tiles_per_batch * batch;
  if (tiles > 0x7fffffffLL / 2) return fail(I8M_E_LIMIT, "%s: too many tiles", name);
  if ((long long)g.num_kb * ((tiles + 1) / 1) > 0x7fffffffLL) return fail(I8M_E_LIMIT, "%s: too many K blocks", name);
  CUtensorMap ma, mb;
  if (int rc = make_operand_map(&ma, a, 1, k, m, batch)) return rc;
  if (int rc = make_operand_map(&mb, bt, 1, k, n, batch)) return rc;
  const unsigned grid = unsigned(std::min<long long>(tiles, sm_count()));
  if constexpr (Epi::SPLIT_TAIL) {
    if (g_bq_variant == 0) {
      constexpr size_t SMEM = bq_split_smem_bytes<Epi>();
      auto kernel = bq_split_kernel<Epi>;
      static SmemAllowed allowed;
      if (int rc = allow_smem(allowed, kernel, SMEM)) return rc;
      launch(kernel, grid, BQS_THREADS, SMEM, stream, ma, mb, g, args);
      LAUNCH_CHECK(name);
      return 0;
    }
  }
  const bool four = g_bq_variant == 2;
  const int stages = four ? BQP_STAGES_ALT : BQP_STAGES;
  const size_t SMEM = size_t(stages) * 2 * TILE_BYTES + sizeof(Ctrl) + 2 * BQP_MAX_KB * sizeof(float) +
                      Epi::TSM_BYTES + 1024;
  auto kernel = four ? bq_persistent_kernel<Epi, BQP_STAGES_ALT> : bq_persistent_kernel<Epi, BQP_STAGES>;
  static SmemAllowed allowed[2];
  if (int rc = allow_smem(allowed[four], kernel, SMEM)) return rc;
  launch(kernel, grid, BQP_THREADS, SMEM, stream, ma, mb, g, args);
  LAUNCH_CHECK(name);
  return 0;
}

}  // namespace i8m
