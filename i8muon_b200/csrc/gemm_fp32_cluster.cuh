// FP32 products (three TF32 products of two-plane operands) split along K over a cluster of CTAs.
//
// The K blocks of a 128 x 128 output tile form SEGMENTS = 1, 2, 4 or 8 segments, each summed on its own.  The sums of two
// consecutive segments are added, then these pairs one after the other.  How many segments there are depends on one
// matrix's extents alone (f32_segments), so a result depends neither on the batch it was computed in nor on the device.
// How many CTAs share a tile (SPLIT, up to one per segment) is the launcher's choice and changes no bit: a CTA takes a run
// of segments, holds sums that wait for their partner in tensor memory, and parks what it has in shared memory.  After
// a cluster barrier CTA r finishes the r-th band of 128 / SPLIT rows: it adds up the parked sums of all CTAs in the order
// above (read over distributed shared memory) and stores the band.
//
//   warp 0       TMA producer: 64 KB stages {A hi, A lo, B hi, B lo} of one 32-element K block, three deep
//   warp 1       tcgen05.mma issuer: twelve instructions per K block into one of four 128-column accumulators (three or
//                two where the CTA holds sums of earlier segments: they take 128 columns each)
//   warps 4..11  fold: every K block's accumulator is added into FP32 registers with round-to-nearest (the tensor
//                core accumulates with truncation), two warps per TMEM lane quarter, 64 columns per thread
//   all warps    sum of the partials, fused epilogue, coalesced stores of every plane and orientation
//
// What bounds it: a K block is 768 tensor cycles (12 x 64) and takes 0.75 us, about 1430.  Its twelve instructions read
// 8 KB each and the copies write 64 KB, 160 KB in all, which would be 1280 cycles at 128 bytes per cycle; but the counters put
// the shared-memory banks at a third of their peak (tensor pipe 44 % active), so the rest is not explained.  One CTA
// per tile with four fold warps took 1900 (the fold's TMEM round trips are a serial chain and two accumulators left the
// issuer waiting for it), left three quarters of the GPU idle when a product has few tiles, and stored rows with 32
// sectors per request.  One 1024 x 4096 call 1745 -> 720 us, six of 1537 x 700 1814 -> 867 us.
// What the fixed order of the sums costs, against adding up whatever share each CTA had: nothing for one matrix, 1 to 3 %
// in batches (six of 1537 x 700 858 -> 867 us, 24 of 512 x 2048 1964 -> 2010), 12 % where a segment is a single K block
// (24 of 256 x 256 205 -> 229).  Parking a segment apart wherever its partner is in another CTA's half made the tail read
// twice the sums (two of 512 x 2048 258 -> 285); pairs need that in one place only.
#pragma once
#include "epi_float.cuh"

namespace i8m {

constexpr int F32C_STAGES = 3;
constexpr int F32C_STAGE_BYTES = 4 * TILE_BYTES;
constexpr int F32C_THREADS = 384;
constexpr int F32C_TMEM_TILES = 4;     // of 128 columns: accumulators, and sums of earlier segments
// What a CTA does with the segments it takes.
template <int SPLIT, int SEGMENTS>
struct F32Share {
  static_assert(SPLIT >= 1 && SPLIT <= SEGMENTS && SEGMENTS % SPLIT == 0 && SEGMENTS <= 8, "at most one CTA per segment");
  static constexpr int TAKEN = SEGMENTS / SPLIT;                       // segments per CTA
  static constexpr int HELD = TAKEN == 1 ? 0 : TAKEN == 2 ? 1 : 2;     // sums in tensor memory: half a pair, earlier pairs
  static constexpr int NBUF = F32C_TMEM_TILES - HELD;                  // accumulators
  // Two CTAs with two pairs each: the second one's pairs follow the first one's sum one by one, so it parks them apart.
  static constexpr bool APART = SPLIT > 1 && TAKEN > 2;
  static_assert(!APART || (SPLIT == 2 && TAKEN == 4), "no other CTA has pairs that wait for those before them");
  static constexpr int PARKED = APART ? 2 : 1;                         // parked tiles in a CTA's shared memory
  static constexpr int SUMS = APART ? 3 : SPLIT;                       // parked sums of the cluster
};
constexpr int F32C_FOLD_WARP0 = 4, F32C_FOLD_WARPS = 8;
// The parked tiles: rows of 132 floats (16-byte aligned; a warp's 32 own-row vector stores cover all banks
// evenly).  They and the band of summed rows lie over the operand ring, which is idle by then.
constexpr int F32C_PARK_PITCH = 132;
constexpr int F32C_PARK_BYTES = TILE * F32C_PARK_PITCH * 4;
static_assert(F32C_PARK_BYTES + TILE * TILE * 4 <= F32C_STAGES * F32C_STAGE_BYTES &&
                  2 * F32C_PARK_BYTES + TILE / 2 * TILE * 4 <= F32C_STAGES * F32C_STAGE_BYTES,
              "the parked sums (two tiles with two CTAs per output tile, else one) and the band overlay the ring");
constexpr size_t F32C_SMEM = size_t(F32C_STAGES) * F32C_STAGE_BYTES + sizeof(Ctrl) + 1024;

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The address of this CTA's shared-memory location `addr` in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_map(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float4 ldc128(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void sts32(uint32_t addr, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

// The summed band: rows of 128 floats whose 16-byte quads are XOR-ed with (row / 4) % 8, so that a warp reads and
// writes whole rows, and 4 x 4 blocks down eight row blocks, without bank conflicts.
__device__ __forceinline__ uint32_t band_quad(uint32_t band, int row, int quad) {
  return band + uint32_t(row * TILE + ((quad ^ ((row >> 2) & 7)) << 2)) * 4u;
}

// The end of a product for rows [rank R, rank R + R) of the tile.  Three sweeps: a diagonal tile first gathers its
// band; then along the rows the sum, the polynomial and the row-major stores; then the transposed stores, as 4 x 4
// blocks out of the band.  Shared-memory and global accesses are 16-byte vectors without bank conflicts where the
// matrix allows it (with one scalar read per element the tail of a tile took 10 us).
template <int MODE, int SPLIT, int SEGMENTS>
__device__ __forceinline__ void f32c_tail(const GemmGeom& g, const FloatArgs& a, int b, int tm, int tn, uint32_t park, uint32_t band,
                                          int rank) {
  constexpr int R = TILE / SPLIT, WARPS = F32C_THREADS / 32;
  const int tid = int(threadIdx.x), warp = tid >> 5, lane = tid & 31;
  const int row0 = tm * TILE + rank * R, col0 = tn * TILE;
  const bool diag_tile = g.sym && tm == tn, mirror = g.sym && tm != tn;
  auto aligned16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  // row-major 16-byte accesses: four columns of a row are inside the matrix together or not at all
  bool vectors = (MODE == MODE_FINAL ? g.ln : g.n) % 4 == 0 && aligned16(a.out);
  if constexpr (MODE != MODE_FINAL) vectors = vectors && aligned16(a.out_lo);
  if constexpr (MODE == MODE_QUAD) vectors = vectors && aligned16(a.src) && aligned16(a.src_lo);
  if constexpr (MODE == MODE_FINAL) vectors = vectors && a.out_dtype == DT_F32 && !a.transpose;
  float* out = static_cast<float*>(a.out);
  float* out_lo = static_cast<float*>(a.out_lo);

  using Share = F32Share<SPLIT, SEGMENTS>;
  constexpr int SUMS = Share::SUMS;
  uint32_t part[SUMS];
#pragma unroll
  for (int s = 0; s < SUMS; ++s) {
    const int rank_of = Share::APART && s > 0 ? 1 : s, slot = Share::APART && s == 2 ? 1 : 0;
    part[s] = park + uint32_t(slot * F32C_PARK_BYTES);
    if (SPLIT > 1) part[s] = cluster_map(part[s], uint32_t(rank_of));
  }
  auto add4 = [](float4& a, const float4& b) {
    a.x = __fadd_rn(a.x, b.x); a.y = __fadd_rn(a.y, b.y); a.z = __fadd_rn(a.z, b.z); a.w = __fadd_rn(a.w, b.w);
  };
  auto total4 = [&](int r, int c) {       // the elements (r, c .. c + 3) of the tile, segments added in their order
    const uint32_t at = uint32_t(r * F32C_PARK_PITCH + c) * 4u;
    float4 w[SUMS];
#pragma unroll
    for (int s = 0; s < SUMS; ++s) w[s] = SPLIT == 1 ? lds128(part[s] + at) : ldc128(part[s] + at);
    constexpr int PAIR = SPLIT == SEGMENTS && SPLIT > 1 ? 2 : 1;      // one sum per segment: pairs first
#pragma unroll
    for (int s = 0; s < SUMS; s += PAIR) {
      if constexpr (PAIR == 2) add4(w[s], w[s + 1]);
      if (s > 0) add4(w[0], w[s]);
    }
    return w[0];
  };

  if (diag_tile) {
    // The stored matrix is exactly symmetric: the upper half of a diagonal tile is its lower half.  Band row r takes
    // columns 0..r from row r and columns c > r from rows c.  Word-wise stores: both halves of a quad may be mixed.
    for (int rb = warp; rb < R; rb += WARPS) {
      const int r = rank * R + rb, c = 4 * lane;
      if (c > r) continue;
      const float4 v = total4(r, c);
      const float x[4] = {v.x, v.y, v.z, v.w};
      const uint32_t at = band_quad(band, rb, lane);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (c + j <= r) sts32(at + 4u * uint32_t(j), x[j]);
    }
    constexpr int QUADS = R / 4;
    const int k = tid % QUADS, r = rank * R + 4 * k;     // rows c, columns r .. r + 3
    for (int c = rank * R + tid / QUADS; c < TILE; c += F32C_THREADS / QUADS) {
      if (c <= r) continue;
      const float4 v = total4(c, r);
      const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (c > r + j) sts32(band_quad(band, 4 * k + j, c >> 2) + 4u * uint32_t(c & 3), x[j]);
    }
    __syncthreads();
  }

  const int cl = 4 * lane, col = col0 + cl;      // this lane's four columns
#pragma unroll 2
  for (int rb = warp; rb < R; rb += WARPS) {
    const int row = row0 + rb;
    const uint32_t at = band_quad(band, rb, lane);
    const float4 v = diag_tile ? lds128(at) : total4(rank * R + rb, cl);
    float x[4] = {v.x, v.y, v.z, v.w};
    if constexpr (MODE == MODE_QUAD) {
      float r[4] = {0.f, 0.f, 0.f, 0.f};
      const size_t si = (size_t(b) * g.m + row) * g.k + col;
      const float* hi = static_cast<const float*>(a.src);
      const float* lo = static_cast<const float*>(a.src_lo);
      if (row < g.m) {
        if (vectors) {
          if (col < g.n) {
            const float4 h = *reinterpret_cast<const float4*>(hi + si), l = *reinterpret_cast<const float4*>(lo + si);
            r[0] = __fadd_rn(h.x, l.x); r[1] = __fadd_rn(h.y, l.y); r[2] = __fadd_rn(h.z, l.z); r[3] = __fadd_rn(h.w, l.w);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (col + j < g.n) r[j] = __fadd_rn(hi[si + j], lo[si + j]);
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x[j] = __fadd_rn(__fmul_rn(a.cb, r[j]), __fmul_rn(a.cc, x[j]));
        if (row == col + j) x[j] = __fadd_rn(x[j], a.ca);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (row >= g.lm || col + j >= g.ln) x[j] = 0.f;     // padding is zero
    sts128(at, make_float4(x[0], x[1], x[2], x[3]));
    if (vectors) {
      if constexpr (MODE == MODE_FINAL) {
        if (row < g.lm && col < g.ln)
          *reinterpret_cast<float4*>(out + (size_t(b) * g.lm + row) * g.ln + col) = make_float4(x[0], x[1], x[2], x[3]);
      } else if (row < g.m && col < g.n) {
        float h[4], l[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) { h[j] = tf32_hi(x[j]); l[j] = tf32_lo(x[j], h[j]); }
        const size_t o = (size_t(b) * g.m + row) * g.n + col;
        *reinterpret_cast<float4*>(out + o) = make_float4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<float4*>(out_lo + o) = make_float4(l[0], l[1], l[2], l[3]);
      }
    }
  }
  // row-major, one element per lane: rows that start anywhere, and the caller's 16-bit types
  if (!vectors && !(MODE == MODE_FINAL && a.transpose)) {
    __syncwarp();          // a warp reads the rows that it has just written
    for (int rb = warp; rb < R; rb += WARPS) {
      const int row = row0 + rb;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int cb = lane + 32 * i, c = col0 + cb;
        const float v = lds32(band_quad(band, rb, cb >> 2) + 4u * uint32_t(cb & 3));
        if constexpr (MODE == MODE_FINAL) {
          if (row < g.lm && c < g.ln) store_user(a.out, a.out_dtype, (size_t(b) * g.lm + row) * g.ln + c, v);
        } else if (row < g.m && c < g.n) {
          const size_t o = (size_t(b) * g.m + row) * g.n + c;
          const float h = tf32_hi(v);
          out[o] = h;
          out_lo[o] = tf32_lo(v, h);
        }
      }
    }
  }
  // transposed: the mirrored half of a symmetric product, the transpose that the next product reads, or a final result
  // whose matrix is tall
  float* tdst = mirror ? out : static_cast<float*>(a.out_t);
  float* tdst_lo = mirror ? out_lo : static_cast<float*>(a.out_t_lo);
  if (!(MODE == MODE_FINAL ? a.transpose != 0 : (tdst != nullptr && !diag_tile))) return;
  __syncthreads();
  const int tld = MODE == MODE_FINAL ? g.lm : mirror ? g.n : g.m;          // row length of the target
  const int rows_in = MODE == MODE_FINAL ? g.lm : g.m, cols_in = MODE == MODE_FINAL ? g.ln : g.n;
  const size_t first = size_t(b) * (MODE == MODE_FINAL ? g.ln : mirror ? g.m : g.n);
  if (MODE != MODE_FINAL && tld % 4 == 0 && aligned16(tdst) && aligned16(tdst_lo)) {
    constexpr int RB = R / 4;                 // 4 x 4 blocks of the band: RB x 32, four or more along a target row
    for (int id = tid; id < RB * (TILE / 4); id += F32C_THREADS) {
      const int rb = id % RB * 4, quad = id / RB, row = row0 + rb;
      if (row >= rows_in) continue;           // rows_in == tld here: a multiple of four
      float4 w[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) w[k] = lds128(band_quad(band, rb + k, quad));
      const float x[4][4] = {{w[0].x, w[1].x, w[2].x, w[3].x}, {w[0].y, w[1].y, w[2].y, w[3].y},
                             {w[0].z, w[1].z, w[2].z, w[3].z}, {w[0].w, w[1].w, w[2].w, w[3].w}};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = col0 + 4 * quad + j;
        if (c >= cols_in) break;
        float h[4], l[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) { h[k] = tf32_hi(x[j][k]); l[k] = tf32_lo(x[j][k], h[k]); }
        const size_t o = (first + c) * tld + row;
        *reinterpret_cast<float4*>(tdst + o) = make_float4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<float4*>(tdst_lo + o) = make_float4(l[0], l[1], l[2], l[3]);
      }
    }
    return;
  }
  // element by element, consecutive lanes along a target row
  const int rb = tid % R, row = row0 + rb;
#pragma unroll 4
  for (int cb = tid / R; cb < TILE; cb += F32C_THREADS / R) {
    const int c = col0 + cb;
    if (row >= rows_in || c >= cols_in) continue;
    const float v = lds32(band_quad(band, rb, cb >> 2) + 4u * uint32_t(cb & 3));
    const size_t o = (first + c) * tld + row;
    if constexpr (MODE == MODE_FINAL) {
      store_user(a.out, a.out_dtype, o, v);
    } else {
      const float h = tf32_hi(v);
      tdst[o] = h;
      tdst_lo[o] = tf32_lo(v, h);
    }
  }
}

template <int MODE, int SPLIT, int SEGMENTS>
__global__ void __launch_bounds__(F32C_THREADS, 1)
fp32_cluster_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    const __grid_constant__ CUtensorMap map_a2, const __grid_constant__ CUtensorMap map_b2,
                    GemmGeom g, FloatArgs args) {
  using Share = F32Share<SPLIT, SEGMENTS>;
  constexpr int STAGES = F32C_STAGES;
  constexpr int NBUF = Share::NBUF;
  constexpr uint32_t IDESC = EpiFloat<float, MODE>::IDESC;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Ctrl* ctrl = reinterpret_cast<Ctrl*>(smem + STAGES * F32C_STAGE_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = int(blockIdx.x) % SPLIT;    // clusters are runs of SPLIT blocks

  int b, tm, tn;
  decode_tile(g, int(blockIdx.x) / SPLIT, b, tm, tn);
  // this CTA's share of the K blocks: [kb0, kb0 + nkb), at least one (the launcher sees to that)
  const int kb0 = int((long long)g.num_kb * rank / SPLIT);
  const int nkb = int((long long)g.num_kb * (rank + 1) / SPLIT) - kb0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&ctrl->full[s]), 1);
      mbar_init(smem_u32(&ctrl->empty[s]), 1);
    }
    for (int i = 0; i < NBUF; ++i) {
      mbar_init(smem_u32(&ctrl->acc_full[i]), 1);
      mbar_init(smem_u32(&ctrl->acc_empty[i]), F32C_FOLD_WARPS);
    }
    ctrl->abort = 0;
    fence_mbar_init();
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_b);
    tma_prefetch_desc(&map_a2);
    tma_prefetch_desc(&map_b2);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&ctrl->tmem_base), TILE * F32C_TMEM_TILES);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  const uint32_t tmem_base = ctrl->tmem_base;
  volatile uint32_t* abort_flag = &ctrl->abort;
  const uint32_t smem_base = smem_u32(smem);

  if (warp == 0 && lane == 0) {
    // -------------------------------------------------------------- producer
    int issued = 0;
    bool ok = true;
    const int mine = (g.debug_simt & 0x100) ? 0 : nkb;   // test hook (i8m_set_debug_core(2)): issue nothing
    for (int i = 0; i < mine; ++i) {
      const int s = i % STAGES;
      if (i >= STAGES) {
        ok = mbar_wait(smem_u32(&ctrl->empty[s]), uint32_t(i / STAGES - 1) & 1u, abort_flag);
        if (!ok) break;
      }
      const uint32_t bar = smem_u32(&ctrl->full[s]), dst = smem_base + uint32_t(s * F32C_STAGE_BYTES);
      mbar_arrive_expect_tx(bar, F32C_STAGE_BYTES);
      tma_load_3d(dst, &map_a, bar, (kb0 + i) * 32, tm * TILE, b);
      tma_load_3d(dst + 2 * TILE_BYTES, &map_b, bar, (kb0 + i) * 32, tn * TILE, b);
      tma_load_3d(dst + TILE_BYTES, &map_a2, bar, (kb0 + i) * 32, tm * TILE, b);
      tma_load_3d(dst + 3 * TILE_BYTES, &map_b2, bar, (kb0 + i) * 32, tn * TILE, b);
      issued = i + 1;
    }
    if (!ok) {
      atomicCAS(g.status, 0u, unsigned(ST_PRODUCER_TIMEOUT) | unsigned(blockIdx.x & 0xff));
      // let the copies that were issued land before shared memory is used for the tail
      for (int i = issued > STAGES ? issued - STAGES : 0; i < issued; ++i) {
        const uint32_t bar = smem_u32(&ctrl->full[i % STAGES]), parity = uint32_t(i / STAGES) & 1u;
        for (int spin = 0; spin < (1 << 20) && !mbar_try_wait(bar, parity); ++spin) {
        }
      }
    }
  } else if (warp == 1 && lane == 0) {
    // ------------------------------------------------------------ MMA issuer
    bool ok = true;
    for (int i = 0; i < nkb; ++i) {
      const int s = i % STAGES, buf = i % NBUF, use = i / NBUF;
      if (use >= 1) {
        ok = mbar_wait(smem_u32(&ctrl->acc_empty[buf]), uint32_t(use - 1) & 1u, abort_flag);
        if (!ok) break;
      }
      ok = mbar_wait(smem_u32(&ctrl->full[s]), uint32_t(i / STAGES) & 1u, abort_flag);
      if (!ok) break;
      tc_fence_after();
      const uint32_t sa = smem_base + uint32_t(s * F32C_STAGE_BYTES);
      const uint64_t a_hi = make_smem_desc_sw128(sa), a_lo = make_smem_desc_sw128(sa + TILE_BYTES);
      const uint64_t b_hi = make_smem_desc_sw128(sa + 2 * TILE_BYTES), b_lo = make_smem_desc_sw128(sa + 3 * TILE_BYTES);
      const uint32_t d = tmem_base + uint32_t(buf * TILE);
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        const uint64_t adv = uint64_t(ks * 2);
        // hi * hi + hi * lo + lo * hi
        umma<KIND_TF32>(d, a_hi + adv, b_hi + adv, IDESC, ks == 0 ? 0u : 1u);
        umma<KIND_TF32>(d, a_hi + adv, b_lo + adv, IDESC, 1u);
        umma<KIND_TF32>(d, a_lo + adv, b_hi + adv, IDESC, 1u);
      }
      umma_commit(smem_u32(&ctrl->empty[s]));
      umma_commit(smem_u32(&ctrl->acc_full[buf]));
    }
    if (!ok) atomicCAS(g.status, 0u, unsigned(ST_MMA_TIMEOUT) | unsigned(blockIdx.x & 0xff));
  } else if (warp >= F32C_FOLD_WARP0) {
    // ------------------------------------------------------------------ fold
    const int q = warp & 3, half = (warp - F32C_FOLD_WARP0) >> 2;
    const uint32_t taddr = tmem_base + (uint32_t(q * 32) << 16) + uint32_t(64 * half);
    float total[64];
#pragma unroll
    for (int j = 0; j < 64; ++j) total[j] = 0.f;
    bool ok = true;
    // Sums that wait in tensor memory, behind the accumulators: HALF_PAIR the first segment of a pair, EARLIER the pairs
    // before it.
    constexpr int HALF_PAIR = 0, EARLIER = 1;
    auto held = [&](int slot) { return taddr + uint32_t((NBUF + slot) * TILE); };
    auto put = [&](int slot) {
      uint32_t v[32];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(total[32 * h + j]);
        tmem_st32(held(slot) + uint32_t(32 * h), v);
      }
      tmem_wait_st();
    };
    auto add = [&](int slot) {       // total <- held sum + total
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t v[32];
        tmem_ld32(held(slot) + uint32_t(32 * h), v);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 32; ++j) total[32 * h + j] = __fadd_rn(__uint_as_float(v[j]), total[32 * h + j]);
      }
    };
    int segment = 0;                 // of this CTA's TAKEN
    // the first K block, counted from kb0, of the next segment
    auto segment_end = [&] { return int((long long)g.num_kb * (rank * Share::TAKEN + segment + 1) / SEGMENTS) - kb0; };
    int end = segment_end();
#pragma unroll 1
    for (int i = 0; i < nkb; ++i) {
      const int buf = i % NBUF;
      ok = mbar_wait_warp_inline(smem_u32(&ctrl->acc_full[buf]), uint32_t(i / NBUF) & 1u, abort_flag);
      if (!ok) break;
      tc_fence_after();
      uint32_t v[32], w[32];
      tmem_ld32(taddr + uint32_t(buf * TILE), v);
      tmem_ld32(taddr + uint32_t(buf * TILE + 32), w);
      tmem_wait_ld();
      tc_fence_before();
      __syncwarp();
      mbar_arrive_if(smem_u32(&ctrl->acc_empty[buf]), lane == 0 ? 1u : 0u);
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        total[j] = __fadd_rn(total[j], __uint_as_float(v[j]));
        total[32 + j] = __fadd_rn(total[32 + j], __uint_as_float(w[j]));
      }
      if constexpr (Share::TAKEN > 1) {
        if (i + 1 == end && i + 1 < nkb) {               // uniform over the CTA
          // an even segment waits for its partner; an odd one completes a pair, which joins those before it
          const int partners = segment % 2 == 0 ? 0 : segment == 1 ? 1 : 2;
#pragma unroll 1
          for (int slot = 0; slot < partners; ++slot) add(slot);
          put(segment % 2 == 0 ? HALF_PAIR : EARLIER);
#pragma unroll
          for (int j = 0; j < 64; ++j) total[j] = 0.f;
          ++segment;
          end = segment_end();
        }
      }
    }
    if (!ok && lane == 0) atomicCAS(g.status, 0u, unsigned(ST_EPILOGUE_TIMEOUT) | unsigned(blockIdx.x & 0xff));
    if (ok) {
      // The last accumulator is complete: every copy of this CTA has landed and been read, the ring is free.
      uint32_t own = smem_base + uint32_t((q * 32 + lane) * F32C_PARK_PITCH + 64 * half) * 4u;
      const bool apart = Share::APART && rank == 1;
      if constexpr (Share::HELD > 0) {
#pragma unroll 1
        for (int slot = 0; slot < (apart ? 1 : Share::HELD); ++slot) add(slot);
      }
      if constexpr (Share::APART) {
        if (apart) {
          uint32_t v[32];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            tmem_ld32(held(EARLIER) + uint32_t(32 * h), v);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; j += 4)
              sts128u(own + 4u * uint32_t(32 * h + j), make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]));
          }
          own += F32C_PARK_BYTES;
        }
      }
#pragma unroll
      for (int j = 0; j < 64; j += 4)
        sts128(own + 4u * uint32_t(j), make_float4(total[j], total[j + 1], total[j + 2], total[j + 3]));
    }
  }
  // every thread comes here, whatever happened to its role; a CTA whose wait ran out has posted the status word, and
  // the band it then contributes to is meaningless but in bounds
  __syncwarp();
  tc_fence_before();
  if constexpr (SPLIT == 1) __syncthreads();
  else cluster_sync();
  if (warp == 1) tmem_dealloc(tmem_base, TILE * F32C_TMEM_TILES);
  f32c_tail<MODE, SPLIT, SEGMENTS>(g, args, b, tm, tn, smem_base, smem_base + Share::PARKED * F32C_PARK_BYTES, rank);
  if constexpr (SPLIT > 1) cluster_sync();   // nobody leaves while its partial tile is still being read
}

}  // namespace i8m
