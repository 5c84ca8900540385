// Weight-quantized GEMM for few batch rows: y[M, N] = x[M, K] * W[N, K]^T with M <= 32, and the grouped expert GEMMs of
// steps that give an expert a few rows (packed weight layout and decode arithmetic: wq_gemm_common.cuh).
//
// What bounds it.  At these sizes the weights are all there is to move, so the bound is HBM: a k-block of a weight tile (128 x 64
// 4-bit weights, 5 KB with its tables) every 180 cycles and SM.  The tcgen05 kernels need 950: a decoded tile makes a round trip
// through shared memory behind four hand-offs (codes landed, slot free, tile decoded, tile multiplied), and with 16 rows the
// tensor core has nothing to hide them with.  Here the code words go from shared memory to registers and, decoded, ARE the A
// operand of mma.sync m16n8k16 -- nothing is written back, no warp waits for another one's decode.  That works because the order
// of K inside an MMA is free as long as both operands agree: lane (g, t) of a warp decodes the 32 columns of half-block t of the
// rows g, g + 8, g + 16, g + 24, four words of 16 bytes each as they lie in memory, and takes the same columns of the activations.
//
// Split.  8 consumer warps = 4 groups of 32 rows x 2 halves of an iteration's columns (256 of 4-bit weights, 128 of bf16 ones);
// two CTAs per SM.  The iterations of all tiles are dealt evenly to the CTAs (a tile in up to a few runs, summed in part order by
// the last one to arrive), because tiles alone do not fill 296 CTAs evenly.  Grouped launches deal whole tiles.  One thread of a
// ninth warp keeps the ring full across tile boundaries: per iteration eight bulk copies of code segments (32 columns of 128
// rows, 64 bytes of padding between them so that the lanes of a quad read different banks), the metadata, and the activations as
// swizzled 64-column tiles.  (Copies by the consumers themselves, cp.async, spent 27 shared-memory cycles per instruction and a
// quarter of the issue slots: 30 us instead of 23 at 8 x 24576 x 4096.)
//
// Large 4-bit weights go to wq_gemm_ts.cu.  Measured, weights not in L2 (floor = packed bytes / 6.65 TB/s), Cubic weights, 8 rows, launches in a row whose
// starts overlap: 24576 x 4096 24 us (floor 9.5, tcgen05 kernels with decoded tiles in shared memory 34), 4096 x 12288 13.6 (4.7, 21.5), 6144 x 4096 9.5 (2.4,
// 14.8), 4096 x 4096 6.6 (1.6, 10.1); single launches behind other work 27.7, 17.5, 13.0, 10.4.  bf16 50688 x 4096 65 (62, 98).  Block-scaled e4m3 weights have nothing to decode either: their chunks and those of the e4m3
// activations are the operands of m16n8k16 once they are f16; 128 experts of 3072 x 4096, eight rows each, 263 us (floor 246, tcgen05 kernel 409),
// 4096 x 1536 140 (123, 289).  What is left above the floor of 4-bit weights is the decode (integer pipe 38 % busy, four warps a scheduler that issue in 37 % of
// the cycles) and 4 to 5 us of start, last loads and the sum of the parts.
#include "wq_gemm_common.cuh"
#include "launch.cuh"

namespace cb {

static constexpr int kSnConsumers = 256;
static constexpr int kSnThreads = kSnConsumers + 32;
static constexpr int kSnRedStride = kTileN + 4;
static constexpr int kSnMaxStages = 6;

struct SkinnyParams {
  WqGemmParams g;
  int its;                    // iterations of a tile: K / columns of an iteration
  int grid;
  int experts;                // fp8: stacked matrices
};

template <int FMT, int NB>
struct SnShape {
  static constexpr bool kBf16 = FMT == kFmtBf16, kFp8 = FMT == kFmtFp8Block, kDirect = kBf16 || kFp8;     // direct: weights as [N, K] rows
  static constexpr int kRows = NB * 8;
  static constexpr int kCols = kBf16 ? 64 : 128;                // K columns of a warp and iteration
  static constexpr int kSteps = kCols / 32;                     // eight columns of every row and lane at a time
  static constexpr int kXTile = kRows * 128, kXTileCols = kFp8 ? 128 : 64;
  static constexpr int kXBytes = 2 * kCols / kXTileCols * kXTile;
  static constexpr int kSeg = kTileN * 16 + 64;                 // 32 columns of the tile's codes
  static constexpr int kCodes = kDirect ? 2 * kATileBytes : 8 * kSeg;
  static constexpr int kMetaSeg = FMT == kFmtCubic4 ? kMetaBytesCubic : kTileN * 4 + 32;
  static constexpr int kMetaSegs = kDirect ? 0 : FMT == kFmtCubic4 ? 2 : 8;
  static constexpr int kStage = (kXBytes + kCodes + kMetaSegs * kMetaSeg + 1023) & ~1023;
  static constexpr uint32_t kTx = kXBytes + (kDirect ? 2 * kATileBytes : 4 * kCodeBytes + (FMT == kFmtCubic4 ? 2 * kMetaBytesCubic : 4 * kMetaBytes));
  static constexpr int kRed = kRows * kSnRedStride * 4;
  static constexpr int kFit = (112 * 1024 - 1024 - 128 - kRed) / kStage;      // two CTAs per SM
  static constexpr int kStages = kFit > kSnMaxStages ? kSnMaxStages : kFit;
  static constexpr int kSmem = kStages * kStage + kRed + 1024;
  static_assert(kStages >= 2, "ring");
};

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void mma_f16_f32(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// four e4m3 values -> two pairs of f16 (exact)
__device__ __forceinline__ void e4m3_to_f16(uint32_t w, uint32_t& lo, uint32_t& hi) {
  asm("{\n\t.reg .b16 a, b;\n\tmov.b32 {a, b}, %2;\n\tcvt.rn.f16x2.e4m3x2 %0, a;\n\tcvt.rn.f16x2.e4m3x2 %1, b;\n\t}" : "=r"(lo), "=r"(hi) : "r"(w));
}

// A run of iterations of one tile.
struct SnSegment {
  int n_tile, expert, tile_id;
  int m0, rows;               // batch rows [m0, m0 + rows)
  int it, it_end;
  int part, parts;
};

// The deal; every thread walks the same list.
template <int NB>
struct SnWalk {
  uint32_t u, u_end, total;   // dense: units = iterations of all tiles
  int tile, tiles, pass;      // grouped: tile = item * n_tiles + n_tile; an item of many rows is walked in passes of NB * 8
  int e, m0, rows;            // grouped: the work item of `tile`
  __device__ __forceinline__ void item(const SkinnyParams& p) {
    const int* w = p.g.group_tiles + 1 + 3 * (tile / p.g.n_tiles);
    e = w[0]; m0 = w[1]; rows = w[2];
  }
  __device__ __forceinline__ void init(const SkinnyParams& p) {
    const uint32_t cta = blockIdx.x, ctas = static_cast<uint32_t>(p.grid);
    if (p.g.group_tiles) {
      tiles = p.g.group_tiles[0] * p.g.n_tiles;
      tile = static_cast<int>(cta);
      pass = 0;
      if (tile < tiles) item(p);
    } else {
      total = static_cast<uint32_t>(p.g.n_tiles) * static_cast<uint32_t>(p.its);
      u = total * cta / ctas;
      u_end = total * (cta + 1) / ctas;
    }
  }
  __device__ __forceinline__ bool next(const SkinnyParams& p, SnSegment& s) {
    if (p.g.group_tiles) {
      if (tile >= tiles) return false;
      s.n_tile = tile % p.g.n_tiles;
      s.expert = e;
      s.tile_id = 0;
      s.m0 = m0 + pass * NB * 8;
      s.rows = min(NB * 8, rows - pass * NB * 8);
      s.it = 0; s.it_end = p.its;
      s.part = 0; s.parts = 1;
      if (++pass * NB * 8 >= rows) {
        pass = 0;
        tile += p.grid;
        if (tile < tiles) item(p);
      }
      return true;
    }
    if (u >= u_end) return false;
    const uint32_t its = static_cast<uint32_t>(p.its), ctas = static_cast<uint32_t>(p.grid);
    const uint32_t t = u / its, first = t * its;
    const uint32_t end = min(u_end, first + its);
    s.n_tile = s.tile_id = static_cast<int>(t);
    s.expert = 0;
    s.m0 = 0; s.rows = p.g.M;
    s.it = static_cast<int>(u - first);
    s.it_end = static_cast<int>(end - first);
    // CTA that owns unit v: the largest c with floor(total * c / ctas) <= v
    const uint32_t g_first = ((first + 1u) * ctas - 1u) / total, g_last = ((first + its) * ctas - 1u) / total;
    s.parts = static_cast<int>(g_last - g_first + 1u);
    s.part = static_cast<int>(blockIdx.x - g_first);
    u = end;
    return true;
  }
};

// The copies of iteration `it` of a segment into a stage: {activations | codes | metadata}.
template <int FMT, int NB>
__device__ __forceinline__ void sn_load_weights(const SkinnyParams& p, const CUtensorMap* tw, const SnSegment& s, int it, uint32_t stage, uint32_t bar) {
  using Sh = SnShape<FMT, NB>;
  const uint32_t dst = stage + Sh::kXBytes;
  if constexpr (Sh::kBf16) {
#pragma unroll
    for (int kg = 0; kg < 2; ++kg) tma_load_2d(dst + kg * kATileBytes, tw, (it * 2 + kg) * 64, s.n_tile * kTileN, bar);
  } else if constexpr (Sh::kFp8) {
#pragma unroll
    for (int kg = 0; kg < 2; ++kg) tma_load_2d(dst + kg * kATileBytes, tw, (it * 2 + kg) * 128, (s.expert * p.g.n_tiles + s.n_tile) * kTileN, bar);
  } else {
    const int kb = it * 4;
    const uint8_t* src = p.g.codes + s.expert * p.g.group_code_stride + (static_cast<size_t>(s.n_tile) * p.g.k_blocks + kb) * kCodeBytes;
#pragma unroll
    for (int i = 0; i < 8; ++i) bulk_g2s(dst + i * Sh::kSeg, src + i * (kCodeBytes / 2), kCodeBytes / 2, bar);
    const uint8_t* meta = p.g.meta + s.expert * p.g.group_meta_stride;
    const uint32_t mdst = dst + Sh::kCodes;
    if constexpr (FMT == kFmtCubic4) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
        bulk_g2s(mdst + i * Sh::kMetaSeg, meta + (static_cast<size_t>(s.n_tile) * p.g.meta_blocks + (kb + 2 * i) / p.g.meta_k_blocks) * kMetaBytesCubic, kMetaBytesCubic, bar);
    } else {
      const uint8_t* m = meta + (static_cast<size_t>(s.n_tile) * p.g.meta_blocks + kb) * kMetaBytes;
#pragma unroll
      for (int i = 0; i < 8; ++i) bulk_g2s(mdst + i * Sh::kMetaSeg, m + i * (kMetaBytes / 2), kMetaBytes / 2, bar);
    }
  }
}
template <int FMT, int NB>
__device__ __forceinline__ void sn_load_x(const CUtensorMap* tx, const SnSegment& s, int it, uint32_t stage, uint32_t bar) {
  using Sh = SnShape<FMT, NB>;
#pragma unroll
  for (int i = 0; i < 2 * Sh::kCols / Sh::kXTileCols; ++i) tma_load_2d(stage + i * Sh::kXTile, tx, it * 2 * Sh::kCols + i * Sh::kXTileCols, s.m0, bar);
}

__device__ __forceinline__ uint4 lds16(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ uint2 lds8(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t lds4(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}

// One iteration of a warp: rows 32 rg + 8 i + g, columns of its half.  Lane t takes the 32 columns of half-block t; the lanes of the
// upper two half-blocks take their words in the order 2, 3, 0, 1, so that the eight lanes that read activations together (two rows,
// four half-blocks in two 64-column tiles) touch eight different 16-byte columns of the banks.
template <int FMT, int NB>
__device__ __forceinline__ void sn_compute(float (&acc)[2][NB][4], uint32_t stage, int nb_used, int rg, int kg, int g, int t) {
  using Sh = SnShape<FMT, NB>;
  const uint32_t cb = stage + Sh::kXBytes;
  uint32_t c[4][4];
  uint4 tab[FMT == kFmtCubic4 ? 4 : 1];
  uint32_t m0[4], m1[4];
  uint32_t xa, arow = 0;
  if constexpr (Sh::kBf16) {
    // 64 columns: lane t takes the chunks 2 t and 2 t + 1 of every row
    arow = cb + kg * kATileBytes + (rg * 32 + g) * 128;
    xa = stage + kg * Sh::kXTile + g * 128 + (((2 * t) ^ g) << 4);
  } else {
    const uint32_t h = static_cast<uint32_t>(t) >> 1;
    const uint32_t ca = cb + (kg * 4 + t) * Sh::kSeg + (rg * 32 + g) * 16;
    const uint32_t ma = cb + Sh::kCodes + (FMT == kFmtCubic4 ? kg * Sh::kMetaSeg + (rg * 32 + g) * 16 : (kg * 4 + t) * Sh::kMetaSeg + (rg * 32 + g) * 4);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint2 a = lds8(ca + i * 128 + h * 8), b = lds8(ca + i * 128 + 8 - h * 8);
      c[i][0] = a.x; c[i][1] = a.y; c[i][2] = b.x; c[i][3] = b.y;
      if constexpr (FMT == kFmtCubic4) {
        tab[i] = lds16(ma + i * 128);
      } else {
        const uint32_t so = lds4(ma + i * 32);
        const uint32_t d0 = bf2_dup(so), d1 = bf2_dup_hi(so);
        // NVFP4: the scales of columns 0..15 and 16..31, in the order of the words
        m0[i] = FMT == kFmtNvfp4 && h ? d1 : d0;
        m1[i] = FMT == kFmtNvfp4 && h ? d0 : d1;
      }
    }
    xa = stage + (kg * 2 + h) * Sh::kXTile + g * 128 + ((((t & 1) * 4 + h * 2) ^ g) << 4);
  }
#pragma unroll
  for (int j = 0; j < Sh::kSteps; ++j) {
    uint4 b[NB];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb)
      if (NB == 1 || nb < nb_used) b[nb] = lds16((xa ^ (j << 4)) + nb * 1024);
#pragma unroll
    for (int rt = 0; rt < 2; ++rt) {
      uint32_t lo[4], hi[4];                       // rows g and g + 8 of the 16-row tile, eight columns each
      if constexpr (Sh::kBf16) {
        const uint32_t o = ((2 * t + j) ^ g) << 4;
        const uint4 l = lds16(arow + 2 * rt * 1024 + o), u = lds16(arow + (2 * rt + 1) * 1024 + o);
        lo[0] = l.x; lo[1] = l.y; lo[2] = l.z; lo[3] = l.w;
        hi[0] = u.x; hi[1] = u.y; hi[2] = u.z; hi[3] = u.w;
      } else if constexpr (FMT == kFmtCubic4) {
        cubic_lut8(c[2 * rt][j], tab[2 * rt], lo);
        cubic_lut8(c[2 * rt + 1][j], tab[2 * rt + 1], hi);
      } else if constexpr (FMT == kFmtNvfp4) {
        decode8<FMT>(c[2 * rt][j], j < 2 ? m0[2 * rt] : m1[2 * rt], 0u, 0u, lo);
        decode8<FMT>(c[2 * rt + 1][j], j < 2 ? m0[2 * rt + 1] : m1[2 * rt + 1], 0u, 0u, hi);
      } else {
        decode8<FMT>(c[2 * rt][j], m0[2 * rt], m1[2 * rt], 0u, lo);
        decode8<FMT>(c[2 * rt + 1][j], m0[2 * rt + 1], m1[2 * rt + 1], 0u, hi);
      }
#pragma unroll
      for (int nb = 0; nb < NB; ++nb)
        if (NB == 1 || nb < nb_used) {
          mma_bf16(acc[rt][nb], lo[0], hi[0], lo[1], hi[1], b[nb].x, b[nb].y);
          mma_bf16(acc[rt][nb], lo[2], hi[2], lo[3], hi[3], b[nb].z, b[nb].w);
        }
    }
  }
}

// One iteration of a warp with e4m3 weights and activations: the 128 columns of its half are a scale block, whose product is summed from zero
// and joins the accumulators times the block's scale.  Lane t takes the chunks 2 t and 2 t + 1 of every row.  Both operands become f16, which has
// every e4m3 value: a weight is converted once for sixteen batch rows and an activation once for the warp's 32 features, where m16n8k32 of e4m3
// took as long as if it converted both for each product.  128 experts of 3072 x 4096, 16 rows each, 411 -> 394 us, of 4096 x 1536 210 -> 185; 1024 routes
// on 8 of them (128 rows each, in eight passes) 162 + 90 -> 125 + 72, where the tcgen05 kernel takes 120 + 96.
template <int NB>
__device__ __forceinline__ void sn_compute_fp8(float (&acc)[2][NB][4], uint32_t stage, int nb_used, int rg, int kg, int g, int t, float scale) {
  using Sh = SnShape<kFmtFp8Block, NB>;
  const uint32_t arow = stage + Sh::kXBytes + kg * kATileBytes + (rg * 32 + g) * 128, xa = stage + kg * Sh::kXTile + g * 128;
  constexpr int W = NB < 2 ? NB : 2;
#pragma unroll
  for (int n0 = 0; n0 < NB; n0 += W) {
    if (n0 > 0 && n0 >= nb_used) break;
    float part[2][W][4];
#pragma unroll
    for (int rt = 0; rt < 2; ++rt)
#pragma unroll
      for (int nb = 0; nb < W; ++nb)
#pragma unroll
        for (int c = 0; c < 4; ++c) part[rt][nb][c] = 0.f;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint32_t o = ((2 * t + j) ^ g) << 4;
      uint32_t b[W][8];
#pragma unroll
      for (int nb = 0; nb < W; ++nb)
        if (NB == 1 || n0 + nb < nb_used) {
          const uint4 x = lds16(xa + (n0 + nb) * 1024 + o);
          e4m3_to_f16(x.x, b[nb][0], b[nb][1]);
          e4m3_to_f16(x.y, b[nb][2], b[nb][3]);
          e4m3_to_f16(x.z, b[nb][4], b[nb][5]);
          e4m3_to_f16(x.w, b[nb][6], b[nb][7]);
        }
#pragma unroll
      for (int rt = 0; rt < 2; ++rt) {
        const uint4 l = lds16(arow + 2 * rt * 1024 + o), u = lds16(arow + (2 * rt + 1) * 1024 + o);
        const uint32_t lw[4] = {l.x, l.y, l.z, l.w}, uw[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          uint32_t a0, a1, a2, a3;
          e4m3_to_f16(lw[w], a0, a2);
          e4m3_to_f16(uw[w], a1, a3);
#pragma unroll
          for (int nb = 0; nb < W; ++nb)
            if (NB == 1 || n0 + nb < nb_used) mma_f16_f32(part[rt][nb], a0, a1, a2, a3, b[nb][2 * w], b[nb][2 * w + 1]);
        }
      }
    }
#pragma unroll
    for (int rt = 0; rt < 2; ++rt)
#pragma unroll
      for (int nb = 0; nb < W; ++nb)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[rt][n0 + nb][c] = fmaf(scale, part[rt][nb][c], acc[rt][n0 + nb][c]);
  }
}

__device__ __forceinline__ void sn_bar() { asm volatile("bar.sync 1, %0;" ::"r"(kSnConsumers) : "memory"); }

template <int FMT>
__device__ __forceinline__ void sn_write(const SkinnyParams& p, const SnSegment& s, const float* v, int stride, int items_tid) {
  // v: the tile's sums [rows][stride]
  if (p.g.swiglu) {
    for (int i = items_tid; i < s.rows * 16; i += kSnConsumers) {
      const float* r = v + (i >> 4) * stride + act_gate_col((i & 15) * 4);
      float4 a = *reinterpret_cast<const float4*>(r), u = *reinterpret_cast<const float4*>(r + 16);
      a.x *= p.g.alpha; a.y *= p.g.alpha; a.z *= p.g.alpha; a.w *= p.g.alpha;
      u.x *= p.g.alpha; u.y *= p.g.alpha; u.z *= p.g.alpha; u.w *= p.g.alpha;
      store_act4(p.g, s.m0 + (i >> 4), s.n_tile, (i & 15) * 4, a, u);
    }
  } else {
    for (int i = items_tid; i < s.rows * 32; i += kSnConsumers)
      sk_store4<FMT>(p.g, s.m0 + (i >> 5), s.n_tile * kTileN + (i & 31) * 4, *reinterpret_cast<const float4*>(v + (i >> 5) * stride + (i & 31) * 4));
  }
}

template <int FMT, int NB>
__global__ void __launch_bounds__(kSnThreads, 2)
wq_gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ SkinnyParams p) {
  using Sh = SnShape<FMT, NB>;
  constexpr int S = Sh::kStages;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full[S], empty[S];
  __shared__ uint32_t is_last, abort_word;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* red = reinterpret_cast<float*>(smem + S * Sh::kStage);
  const uint32_t ring = smem_u32(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rg = warp & 3, kg = warp >> 2, g = lane >> 2, t = lane & 3;
  volatile uint32_t* abort_flag = &abort_word;

  if (threadIdx.x == 0) {
    for (int i = 0; i < S; ++i) {
      mbar_init(smem_u32(&full[i]), 1);
      mbar_init(smem_u32(&empty[i]), kSnConsumers / 32);
    }
    abort_word = 0;
    mbar_fence_init();
  }
  __syncthreads();
  pdl_launch_dependents();
  if (p.g.group_tiles) pdl_wait();           // the work list is written by the routing kernels
  SnWalk<NB> walk;
  SnSegment seg;
  walk.init(p);

  if (warp == kSnConsumers / 32) {
    if (lane == 0) {
      tma_prefetch_desc(&tmap_x);
      // the first weights go out before the previous kernel has finished, the activations after it
      SnWalk<NB> first = walk;
      bool more = walk.next(p, seg);
      int filled = 0;
      for (bool ok = more; ok && filled < S;) {
        const uint32_t bar = smem_u32(&full[filled]);
        mbar_expect_tx(bar, Sh::kTx);
        sn_load_weights<FMT, NB>(p, &tmap_w, seg, seg.it, ring + filled * Sh::kStage, bar);
        ++filled;
        if (++seg.it == seg.it_end) ok = walk.next(p, seg);
      }
      pdl_wait();
      walk = first;
      more = walk.next(p, seg);
      uint32_t n = 0;                        // iterations issued
      int slot = 0;
      while (more) {
        const uint32_t bar = smem_u32(&full[slot]), stage = ring + slot * Sh::kStage;
        if (n >= static_cast<uint32_t>(filled)) {
          if (!mbar_wait_park(smem_u32(&empty[slot]), ((n / S) - 1u) & 1u, abort_flag)) break;
          mbar_expect_tx(bar, Sh::kTx);
          sn_load_weights<FMT, NB>(p, &tmap_w, seg, seg.it, stage, bar);
        }
        sn_load_x<FMT, NB>(&tmap_x, seg, seg.it, stage, bar);
        ++n;
        if (++slot == S) slot = 0;
        if (++seg.it == seg.it_end) more = walk.next(p, seg);
      }
      if (*abort_flag) {                     // the copies in flight land (for a bounded time) before the CTA goes
        const long long t0 = clock64();
        for (uint32_t i = n > S ? n - S : 0; i < n; ++i)
          while (!mbar_try_wait(smem_u32(&full[i % S]), (i / S) & 1u) && clock64() - t0 < kWaitBudgetCycles / 8) {
          }
        atomicExch(p.g.status, static_cast<uint32_t>(kErrBarrierTimeout));
      }
    }
    return;
  }
  pdl_wait();
  int slot = 0;
  uint32_t phase = 0;
  bool ok = true;                            // after a wait that ran out the rest runs through on whatever is there: barriers stay aligned
  while (walk.next(p, seg)) {
    float acc[2][NB][4];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int n = 0; n < NB; ++n)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][n][c] = 0.f;
    const int nb_used = (seg.rows + 7) >> 3;
    const float* block_scale = nullptr;
    if constexpr (Sh::kFp8) block_scale = p.g.row_scale + (static_cast<size_t>(seg.expert) * p.g.n_tiles + seg.n_tile) * p.g.k_blocks + kg;
    for (int it = seg.it; it < seg.it_end; ++it) {
      float scale = 0.f;
      if constexpr (Sh::kFp8) scale = __ldg(block_scale + 2 * it);
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait_park(smem_u32(&full[slot]), phase, abort_flag));
      if constexpr (Sh::kFp8) sn_compute_fp8<NB>(acc, ring + slot * Sh::kStage, nb_used, rg, kg, g, t, scale);
      else sn_compute<FMT, NB>(acc, ring + slot * Sh::kStage, nb_used, rg, kg, g, t);
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&empty[slot]));
      if (++slot == S) { slot = 0; phase ^= 1u; }
    }
    // the two column halves meet in shared memory as [batch row][feature]
    float* mine = red + (2 * t) * kSnRedStride + rg * 32 + g;
    float xs[NB][2];                           // scales of the activation rows
    if constexpr (Sh::kFp8) {
#pragma unroll
      for (int nb = 0; nb < NB; ++nb)
#pragma unroll
        for (int c = 0; c < 2; ++c) xs[nb][c] = nb * 8 + 2 * t + c < seg.rows ? p.g.col_scale[seg.m0 + nb * 8 + 2 * t + c] : 0.f;
    }
    auto each = [&](auto&& f) {
#pragma unroll
      for (int rt = 0; rt < 2; ++rt)
#pragma unroll
        for (int nb = 0; nb < NB; ++nb)
          if (NB == 1 || nb < nb_used)
#pragma unroll
            for (int c = 0; c < 4; ++c) f(mine[(nb * 8 + (c & 1)) * kSnRedStride + rt * 16 + (c >> 1) * 8], acc[rt][nb][c] * (Sh::kFp8 ? xs[nb][c & 1] : 1.f));
    };
    sn_bar();                                  // the previous segment's sums have been read: nothing else holds a warp back that is a run ahead
    if (kg == 1) each([](float& m, float v) { m = v; });
    sn_bar();
    if (kg == 0) each([](float& m, float v) { m += v; });
    sn_bar();
    if (seg.parts == 1) {
      sn_write<FMT>(p, seg, red, kSnRedStride, threadIdx.x);
    } else {
      constexpr size_t kElems = static_cast<size_t>(NB) * 8 * kTileN;
      float* slots = p.g.workspace + static_cast<size_t>(blockIdx.x - seg.part) * 2 * kElems;   // part q > 0 at q * 2 * kElems, part 0 one further
      auto slot_of = [&](int q) { return slots + (static_cast<size_t>(q) * 2 + (q == 0 ? 1 : 0)) * kElems; };
      float* own = slot_of(seg.part);
      for (int i = threadIdx.x; i < seg.rows * 32; i += kSnConsumers)
        __stcg(reinterpret_cast<float4*>(own + i * 4), *reinterpret_cast<const float4*>(red + (i >> 5) * kSnRedStride + (i & 31) * 4));
      sn_bar();
      if (threadIdx.x == 0) {
        const uint32_t prev = atom_add_acq_rel_gpu(p.g.counters + seg.tile_id, 1u);
        is_last = prev == static_cast<uint32_t>(seg.parts) - 1u;
        if (is_last) p.g.counters[seg.tile_id] = 0;
      }
      sn_bar();
      if (is_last) {
        for (int i = threadIdx.x; i < seg.rows * 32; i += kSnConsumers) {
          float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
          for (int q = 0; q < seg.parts; ++q) {
            const float4 v = __ldcg(reinterpret_cast<const float4*>(slot_of(q) + i * 4));
            a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
          }
          *reinterpret_cast<float4*>(red + (i >> 5) * kSnRedStride + (i & 31) * 4) = a;
        }
        sn_bar();
        sn_write<FMT>(p, seg, red, kSnRedStride, threadIdx.x);
      }
    }
  }
  if (!ok && lane == 0) atomicExch(p.g.status, static_cast<uint32_t>(kErrBarrierTimeout));
}

template <int FMT, int NB>
static int launch_skinny(SkinnyParams p, const void* x, int ldx, int max_grid, cudaStream_t stream) {
  using Sh = SnShape<FMT, NB>;
  CUtensorMap tx, tw;
  if ((Sh::kFp8 ? make_tmap_u8(&tx, x, p.g.M, p.g.K, ldx, Sh::kRows) : make_tmap_bf16(&tx, x, p.g.M, p.g.K, ldx, Sh::kRows)) != 0) return -20;
  tw = tx;
  if (Sh::kFp8 && make_tmap_u8(&tw, p.g.codes, static_cast<uint64_t>(p.g.N) * p.experts, p.g.K, p.g.K, kTileN) != 0) return -21;
  if (FMT == kFmtBf16 && make_tmap_bf16(&tw, p.g.codes, p.g.N, p.g.K, p.g.K, kTileN) != 0) return -21;
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -18;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(wq_gemm_skinny_kernel<FMT, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sh::kSmem);
    if (e != cudaSuccess) return static_cast<int>(e);
    configured[dev] = true;
  }
  p.its = p.g.K / (2 * Sh::kCols);
  const long long units = p.g.group_tiles ? max_grid : static_cast<long long>(p.g.n_tiles) * p.its;
  p.grid = static_cast<int>(units < max_grid ? units : max_grid);
  // Few tiles: whole divisions of K, so that a CTA has one run and joins one sum (4096 x 4096: 6.4 us on 256 CTAs, 8.8 us on 296
  // whose runs straddle tiles), unless that would leave two fifths of the machine idle
  if (!p.g.group_tiles && 2 * p.g.n_tiles <= max_grid) {
    int parts = 1;
    for (int q = 2; q <= p.its && q * p.g.n_tiles <= max_grid; ++q)
      if (p.its % q == 0) parts = q;
    if (parts * p.g.n_tiles * 5 >= max_grid * 3) p.grid = parts * p.g.n_tiles;
  }
  return static_cast<int>(launch(wq_gemm_skinny_kernel<FMT, NB>, dim3(static_cast<unsigned>(p.grid)), dim3(kSnThreads), Sh::kSmem, stream, tx, tw, p));
}

template <int FMT>
static int launch_skinny_rows(const SkinnyParams& p, const void* x, int ldx, int rows, int max_grid, cudaStream_t stream) {
  if (rows <= 8) return launch_skinny<FMT, 1>(p, x, ldx, max_grid, stream);
  if (rows <= 16) return launch_skinny<FMT, 2>(p, x, ldx, max_grid, stream);
  return launch_skinny<FMT, 4>(p, x, ldx, max_grid, stream);
}

static int skinny(int fmt, const void* x, int ldx, const void* codes, const void* meta, void* y, int ldy, const void* residual, float alpha, int M, int N, int K,
                  int group_k, int swiglu, const void* tiles, int rows, size_t code_stride, size_t meta_stride, void* workspace, long long workspace_bytes,
                  void* counters, void* status, void* stream, const void* x_scale = nullptr, int experts = 1) {
  if (fmt != kFmtBf16 && fmt != kFmtCubic4 && fmt != kFmtAffine4 && fmt != kFmtNvfp4 && fmt != kFmtFp8Block) return -11;
  if (M <= 0 || N <= 0 || K <= 0 || K % (fmt == kFmtBf16 ? 128 : 256) != 0 || ldx % (fmt == kFmtFp8Block ? 16 : 8) != 0 || (reinterpret_cast<uintptr_t>(x) & 15) != 0) return -10;
  if (fmt == kFmtFp8Block && (!x_scale || !meta || swiglu || (reinterpret_cast<uintptr_t>(codes) & 15) != 0 || experts <= 0 || (tiles && N % kTileN != 0))) return -15;
  if (fmt == kFmtCubic4 && group_k % 128 != 0) return -12;
  if (rows <= 0 || rows > 32) return -17;
  if (swiglu && (residual || (N % 32) != 0 || ldy < N / 2)) return -51;
  int dev = 0;
  static int sms[64] = {};
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -18;
  if (sms[dev] == 0 && cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -18;
  SkinnyParams p = {};
  p.g.codes = static_cast<const uint8_t*>(codes);
  p.g.meta = static_cast<const uint8_t*>(meta);
  p.g.y = static_cast<__nv_bfloat16*>(y);
  p.g.residual = static_cast<const __nv_bfloat16*>(residual);
  p.g.workspace = static_cast<float*>(workspace);
  p.g.counters = static_cast<uint32_t*>(counters);
  p.g.status = static_cast<uint32_t*>(status);
  p.g.M = M; p.g.N = N; p.g.K = K; p.g.ldy = ldy; p.g.alpha = alpha;
  p.g.swiglu = swiglu;
  p.experts = experts;
  p.g.row_scale = static_cast<const float*>(meta);
  p.g.col_scale = static_cast<const float*>(x_scale);
  p.g.k_blocks = K / (fmt == kFmtFp8Block ? 128 : kBlockK);
  p.g.meta_k_blocks = fmt == kFmtCubic4 ? group_k / kBlockK : 1;
  p.g.meta_blocks = (p.g.k_blocks + p.g.meta_k_blocks - 1) / p.g.meta_k_blocks;
  p.g.n_tiles = (N + kTileN - 1) / kTileN;
  p.g.group_tiles = static_cast<const int*>(tiles);
  p.g.group_code_stride = code_stride;
  p.g.group_meta_stride = meta_stride;
  const int max_grid = 2 * sms[dev];
  if (static_cast<long long>(p.g.n_tiles) * (K / 128) * max_grid >= (1ll << 31)) return -19;      // the deal counts in 32 bits
  if (!tiles) {
    const long long rows_up = rows <= 8 ? 8 : rows <= 16 ? 16 : 32;
    if (!workspace || !counters || workspace_bytes < 2ll * max_grid * rows_up * kTileN * 4) return -13;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (fmt) {
    case kFmtCubic4: return launch_skinny_rows<kFmtCubic4>(p, x, ldx, rows, max_grid, st);
    case kFmtAffine4: return launch_skinny_rows<kFmtAffine4>(p, x, ldx, rows, max_grid, st);
    case kFmtNvfp4: return launch_skinny_rows<kFmtNvfp4>(p, x, ldx, rows, max_grid, st);
    case kFmtFp8Block: return launch_skinny_rows<kFmtFp8Block>(p, x, ldx, rows, max_grid, st);
    default: return launch_skinny_rows<kFmtBf16>(p, x, ldx, rows, max_grid, st);
  }
}

}  // namespace cb

extern "C" {

// y[M, N] (or, with `swiglu`, the N / 2 activations of interleaved gate / up rows) for M <= 32, K a multiple of 256 (bf16 weights:
// 128) and, for Cubic weights, a scale group that is a multiple of 128 columns.  `counters`: one word per weight tile, zero.
int cb_wq_gemm_skinny(int fmt, const void* x, int ldx, const void* codes, const void* meta, void* y, int ldy, const void* residual, float alpha, int M, int N,
                      int K, int group_k, int swiglu, void* workspace, long long workspace_bytes, void* counters, void* status, void* stream) {
  return cb::skinny(fmt, x, ldx, codes, meta, y, ldy, residual, alpha, M, N, K, group_k, swiglu, nullptr, M, 0, 0, workspace, workspace_bytes, counters, status, stream);
}

// The grouped form over a device work list {count, then {expert, first row, rows}}: `rows` (<= 32) rows of an item at a time.
int cb_wq_gemm_skinny_grouped(int fmt, const void* x, int ldx, const void* codes, const void* meta, void* y, int ldy, float alpha, int total_rows, int N, int K,
                              int group_k, int swiglu, const void* tiles, int rows, long long code_stride, long long meta_stride, void* status, void* stream) {
  if (!tiles || fmt == cb::kFmtBf16 || fmt == cb::kFmtFp8Block) return -40;
  return cb::skinny(fmt, x, ldx, codes, meta, y, ldy, nullptr, alpha, total_rows, N, K, group_k, swiglu, tiles, rows, static_cast<size_t>(code_stride),
                    static_cast<size_t>(meta_stride), nullptr, 0, nullptr, status, stream);
}

// Block-scaled e4m3 weights [N, K] times e4m3 activations with a scale a row, for M <= 32, or over a work list as above (`experts` matrices stacked
// in `wq` and `w_scale`, N a multiple of 128).  K a multiple of 256, rows of `xq` 16 bytes apart or a multiple.
int cb_wq_gemm_skinny_fp8(const void* xq, int ldx, const void* x_scale, const void* wq, const void* w_scale, void* y, int ldy, const void* residual, int M, int N, int K,
                          void* workspace, long long workspace_bytes, void* counters, void* status, void* stream) {
  return cb::skinny(cb::kFmtFp8Block, xq, ldx, wq, w_scale, y, ldy, residual, 1.f, M, N, K, K, 0, nullptr, M, 0, 0, workspace, workspace_bytes, counters, status, stream, x_scale);
}
int cb_wq_gemm_skinny_fp8_grouped(const void* xq, int ldx, const void* x_scale, const void* wq, const void* w_scale, void* y, int ldy, int total_rows, int N, int K,
                                  const void* tiles, int rows, int experts, void* status, void* stream) {
  if (!tiles) return -40;
  return cb::skinny(cb::kFmtFp8Block, xq, ldx, wq, w_scale, y, ldy, nullptr, 1.f, total_rows, N, K, K, 0, tiles, rows, 0, 0, nullptr, 0, nullptr, status, stream, x_scale, experts);
}

}  // extern "C"
