// Weight-quantized GEMM of batch rows in blocks of up to 128, of one matrix or of each expert of a work list: y[M, N] = x[M, K] * W[N, K]^T, 4-bit weights
// (packed weight layout and decode arithmetic: wq_gemm_common.cuh).
//
// What bounds it.  The other tcgen05 kernels write a decoded tile to shared memory, in a stage that also holds the activation tile and (per-tile
// kernel) the codes: six to eight stages of 27 KB, each of which goes release -> copies -> 2000 to 3000 cycles -> decode -> fence -> MMA before
// it comes back, 500 to 750 cycles a k-block of 64 columns whatever the rows.  Here the decoded tile is the MMA's A operand in TENSOR MEMORY: a
// decoding thread owns a weight row, its 64 decoded columns are one tcgen05.st.  Shared memory then holds nothing but copies, in two rings of
// their own: codes (10 KB a stage, up to 12 stages, on their way before the previous kernel is done) and activations.  A unit of the pipeline
// is 128 columns: the one thread that waits, counts and issues copies or MMAs for a stage takes 150 to 200 cycles for it, whatever it moves.
// Few-row, per-tile or persistent kernel -> this one, Cubic weights not in L2, single launches behind other work, 8 / 48 / 128 rows, one B200: 24576 x 4096
// 27.4 / 38.7 / 44.5 -> 21.9 / 24.0 / 29.7 us (floor 8.7), 4096 x 12288 17.2 / 25.5 / 28.3 -> 15.7 / 17.9 / 22.3 (4.3), 6144 x 4096 13.2 / 18.9 / 21.4 -> 11.7 / 13.6 / 18.8
// (2.2); launches in a row whose starts overlap, 8 rows: 23.9 -> 20.3, 13.6 -> 12.9, 9.5 -> 8.9.  About 8 us of each are start (4300 cycles to the first codes), the last run's sums and the sum of parts.  128 experts (NVFP4) of 1536 x 2048,
// 6 / 24 / 64 / 256 rows an expert: 85 / 134 / 137 / 299 -> 73 / 78 / 93 / 251 us (35 us of codes; at 256 rows 125 us of MMAs), 2048 x 768
// 48 / 88 / 102 / 287 -> 41 / 43 / 51 / 132.  Blocks of rows decode a tile once each: 24576 x 4096 at 256 / 331 / 512 rows, single cold launches,
// 57.5 / 89.5 / 93.1 -> 48.8 / 64.3 / 83.5 us.  Up to 24 rows the decode's integer pipe is half busy and its latency the rest (a unit in 740 cycles, 490
// instructions a scheduler), at 128 rows a unit takes 1150 cycles of which the MMAs are 517.  What did not help: pairs of CTAs with half of the activation
// tile each (256 rows: 51.4 us), MMAs on each half of a unit while the other is decoded (8 rows: 25.9 us, the one thread's rounds double).
//
// Split.  One CTA per SM.  One matrix: the units of all weight tiles (of each block of rows in turn) are dealt evenly, a tile in a few runs whose fp32 sums the last one to arrive
// adds in the order of K (deterministic).  Work list: whole tiles, every CTA every so many.  Roles: warps 0-3 epilogue (from one of two accumulators
// while the next run fills the other one; a lane has a feature, results leave from its registers: staged in shared memory for wider stores they set
// the pace of short K, 2048 x 768 at 256 rows 230 us), warp 4 codes, warp 7 their tables, warp 5 MMAs, warp 6 activations, warps 8-23 decode: group g
// of four takes every fourth unit, and a share of the last run's sums (24576 x 4096 at 128 rows 36.9 -> 34.6 us).
// Every wait is bounded; on a timeout the roles leave, the status word is set and tensor memory is freed.
#include "wq_gemm_common.cuh"
#include "launch.cuh"
#include <type_traits>

namespace cb {

static constexpr int kTsThreads = 768;
static constexpr int kTsGroups = 4;              // of decode warps
static constexpr int kTsCols = 128;              // K columns of a unit: two k-blocks of the packed layout
static constexpr int kTsSlots = 4;               // decoded units in tensor memory, 64 columns each
static constexpr int kTsMaxC = 12;
static constexpr int kTsBox = 64;                // activation rows of a copy
static constexpr uint32_t kTsTmemA = 256;        // first column of the decoded tiles; accumulators below
static_assert(kTsSlots % kTsGroups == 0 && kTsMaxC % kTsGroups == 0, "a slot belongs to one group");

struct __align__(16) TsCtl {
  uint64_t c_full[kTsMaxC], c_empty[kTsMaxC], full[kTsSlots], empty[kTsSlots], acc_full[2], acc_empty[2], last_full;
  int sum_tile[2], sum_part[2], sum_parts[2], sums;      // tiles whose last part was this CTA's
  uint32_t tmem, abort_word;
};

// Forms, each a kernel of its own: what blocks of rows add to every role's walk costs a matrix of one block 0.5 us (4096 x 12288 at 8 rows 16.3 against 15.7)
static constexpr int kTsOneBlock = 0, kTsGrouped = 1, kTsRowBlocks = 2;
// A run of units of one tile.
struct TsRun {
  int tile, kb, kb_end, part, parts;
  int sum;                                       // counter of the tile's (and block of rows') parts
  int expert, m0, rows;                          // batch rows [m0, m0 + rows)
};
// The deal; every role walks the same list.  Work list: tile c, c + CTAs, .. of its items, whole.  p.splits > 0: CTA c has part c % splits of
// tile c / splits; else the units of all tiles are dealt evenly.
template <int FORM>
struct TsWalk {
  static constexpr bool GROUPED = FORM == kTsGrouped, BLOCKS = FORM == kTsRowBlocks;
  uint32_t u, u_end, total;
  int m_blocks;
  int tile, tiles, e, m0, rows;                  // work list: the next tile, its item
  __device__ __forceinline__ TsWalk(const WqGemmParams& p, int m_blocks_) : m_blocks(m_blocks_) {
    const uint32_t cta = blockIdx.x, ctas = gridDim.x;
    const uint32_t kbs = static_cast<uint32_t>(p.k_blocks);
    total = static_cast<uint32_t>(BLOCKS ? p.tiles * m_blocks : p.tiles) * kbs;
    if constexpr (GROUPED) {
      tiles = p.group_tiles[0] * p.tiles;
      tile = static_cast<int>(cta);
      u = 0;
      u_end = tile < tiles ? static_cast<uint32_t>((tiles - 1 - tile) / static_cast<int>(ctas) + 1) * kbs : 0u;
      if (tile < tiles) item(p);
    } else if (p.splits > 0) {
      const uint32_t parts = static_cast<uint32_t>(p.splits), t = cta / parts, part = cta - t * parts;
      u = t * kbs + kbs * part / parts;
      u_end = t * kbs + kbs * (part + 1) / parts;
    } else {
      u = total * cta / ctas;                    // (total * CTAs is below 2^32)
      u_end = total * (cta + 1) / ctas;
    }
  }
  __device__ __forceinline__ uint32_t units() const { return u_end - u; }
  __device__ __forceinline__ void item(const WqGemmParams& p) {
    const int* w = p.group_tiles + 1 + 3 * (tile / p.tiles);
    e = w[0]; m0 = w[1]; rows = w[2];
  }
  __device__ __forceinline__ bool next(const WqGemmParams& p, TsRun& r) {
    if constexpr (GROUPED) {
      if (tile >= tiles) return false;
      r.tile = tile % p.tiles;
      r.kb = 0; r.kb_end = p.k_blocks;
      r.part = 0; r.parts = 1; r.sum = 0;
      r.expert = e; r.m0 = m0; r.rows = rows;
      tile += static_cast<int>(gridDim.x);
      if (tile < tiles) item(p);                 // on its way while this tile is worked on
      return true;
    } else {
      if (u >= u_end) return false;
      const uint32_t kbs = static_cast<uint32_t>(p.k_blocks), t = u / kbs, first = t * kbs, end = min(u_end, first + kbs);
      r.tile = r.sum = static_cast<int>(t);
      r.kb = static_cast<int>(u - first);
      r.kb_end = static_cast<int>(end - first);
      r.expert = 0; r.m0 = 0; r.rows = p.M;
      if constexpr (BLOCKS) {                    // those of a weight tile in turn
        r.tile = static_cast<int>(t) / m_blocks;
        r.m0 = (r.sum - r.tile * m_blocks) * p.mb;
        r.rows = min(p.mb, p.M - r.m0);
      }
      if (p.splits > 0) {
        r.parts = p.splits;
        r.part = static_cast<int>(blockIdx.x) - r.sum * p.splits;
      } else {
        // CTA that owns unit v: the largest c with floor(total * c / ctas) <= v
        const uint32_t ctas = gridDim.x, c0 = ((first + 1u) * ctas - 1u) / total, c1 = ((first + kbs) * ctas - 1u) / total;
        r.parts = static_cast<int>(c1 - c0 + 1u);
        r.part = static_cast<int>(blockIdx.x - c0);
      }
      u = end;
      return true;
    }
  }
};

// Bytes of a unit's codes and tables
__host__ __device__ constexpr int ts_codes() { return 2 * kCodeBytes; }
__host__ __device__ constexpr int ts_meta(int fmt) { return fmt == kFmtCubic4 ? kMetaBytesCubic : 2 * kMetaBytes; }

// 64 columns of a weight row -> bf16 pairs in the order of K; `h`: which of the unit's k-blocks
template <int FMT>
__device__ __forceinline__ void ts_decode(const uint8_t* stage, int h, int row, uint32_t (&out)[32]) {
  const uint8_t* codes = stage + h * kCodeBytes + row * 16;
  const uint4 w[2] = {*reinterpret_cast<const uint4*>(codes), *reinterpret_cast<const uint4*>(codes + kCodeBytes / 2)};
  uint4 t = make_uint4(0u, 0u, 0u, 0u);
  uint32_t so[2] = {0u, 0u};
  if constexpr (FMT == kFmtCubic4) {
    t = *reinterpret_cast<const uint4*>(stage + ts_codes() + row * 16);
  } else {
    const uint32_t* meta = reinterpret_cast<const uint32_t*>(stage + ts_codes() + h * kMetaBytes) + row;
    so[0] = meta[0];
    so[1] = meta[128];
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const uint32_t c0 = bf2_dup(so[q]), c1 = bf2_dup_hi(so[q]), words[4] = {w[q].x, w[q].y, w[q].z, w[q].w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t o[4];
      if constexpr (FMT == kFmtCubic4) cubic_lut8(words[j], t, o);
      else if constexpr (FMT == kFmtNvfp4) decode8<FMT>(words[j], j < 2 ? c0 : c1, 0u, 0u, o);
      else decode8<FMT>(words[j], c0, c1, 0u, o);
#pragma unroll
      for (int i = 0; i < 4; ++i) out[q * 16 + j * 4 + i] = o[i];
    }
  }
}

// Partial sums of a CTA: [row][128]; two places a CTA, the first part of a tile in the second
__device__ __forceinline__ float* ts_slot(const WqGemmParams& p, int cta, int part) {
  return p.workspace + (static_cast<size_t>(cta) * 2 + (part == 0 ? 1 : 0)) * p.mb * kTileN;
}
__device__ __forceinline__ void ts_bar() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// A part's sums of the rows c, c + step, .. (32 at a time), out of tensor memory into the CTA's place of the workspace
__device__ __forceinline__ void ts_part(const WqGemmParams& p, const TsRun& run, uint32_t acc, int quad, int lane, int c, int step) {
  float* own = ts_slot(p, blockIdx.x, run.part) + quad * 32 + lane;
#pragma unroll 1
  for (; c < run.rows; c += step) {              // (columns behind the rows hold nothing, and are not written)
    uint32_t r[32];
    tmem_ld_32x32(acc + (static_cast<uint32_t>(quad * 32) << 16) + c, r);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (c + j < run.rows) __stcg(own + (c + j) * kTileN, __uint_as_float(r[j]));
  }
}

// A whole tile's sums leave from the registers that tensor memory gives: a lane has a feature of 32 rows, a row of a warp is 64 bytes.  Gated: lanes
// 0-15 have the gates of 16 features, 16-31 the others of the same; a pair of rows is exchanged and each half of the warp activates one.
template <int FMT>
__device__ __forceinline__ void ts_out(const WqGemmParams& p, const TsRun& run, uint32_t acc, int warp, int lane) {
#pragma unroll 1
  for (int c = 0; c < run.rows; c += 32) {       // (columns behind the rows hold nothing, and are not written)
    uint32_t r[32];
    tmem_ld_32x32(acc + c, r);
    tmem_ld_wait();
    const int rows = run.rows - c;
    if (p.swiglu) {
      const int n = run.tile * (kTileN / 2) + warp * 16 + (lane & 15), half = lane >> 4;
      __nv_bfloat16* y = p.y + static_cast<size_t>(run.m0 + c + half) * p.ldy + n;
#pragma unroll
      for (int j = 0; j < 32; j += 2) {
        const float a = __uint_as_float(r[j]), b = __uint_as_float(r[j + 1]), o = __shfl_xor_sync(0xffffffffu, half ? a : b, 16);
        const float v = glu_mul(p.swiglu, p.glu_limit, (half ? o : a) * p.alpha, (half ? b : o) * p.alpha);
        if (j + half < rows && 2 * n < p.N) *y = __float2bfloat16(v);
        y += 2 * p.ldy;
      }
    } else {
      const int n = run.tile * kTileN + warp * 32 + lane;
      const size_t off = static_cast<size_t>(run.m0 + c) * p.ldy + n;
      __nv_bfloat16* y = p.y + off;
      const __nv_bfloat16* res = p.residual ? p.residual + off : nullptr;
      if (n < p.N) {
#pragma unroll
        for (int j0 = 0; j0 < 32; j0 += 8) {
          float v[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r[j0 + j]) * p.alpha;
          if (res) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (j0 + j < rows) v[j] += __bfloat162float(res[static_cast<size_t>(j0 + j) * p.ldy]);
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (j0 + j < rows) *y = __float2bfloat16(v[j]);
            y += p.ldy;
          }
        }
      }
    }
  }
}

// k_blocks counts units here, meta_k_blocks units of a table; tiles: weight tiles of a matrix; c_stages: depth of the code ring;
// mb: most batch rows of a run, rounded up to 16
template <int FMT, int FORM>
__global__ void __launch_bounds__(kTsThreads, 1)
wq_gemm_ts_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ WqGemmParams p, const int m_blocks, const int box, const int boxes) {
  constexpr bool GROUPED = FORM == kTsGrouped, BLOCKS = FORM == kTsRowBlocks;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  constexpr uint32_t kC = ts_codes() + ts_meta(FMT);
  const uint32_t box_bytes = static_cast<uint32_t>(box) * 128u, x_half = box_bytes * boxes, x_bytes = 2 * x_half;
  uint8_t* xs = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* cs = xs + kTsSlots * x_bytes;
  TsCtl& ctl = *reinterpret_cast<TsCtl*>(cs + p.c_stages * kC);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int S = kTsSlots;
  const int NC = p.c_stages;
  volatile uint32_t* abort_flag = &ctl.abort_word;
  if (threadIdx.x == 0) {
    for (int i = 0; i < NC; ++i) {
      mbar_init(smem_u32(&ctl.c_full[i]), 2);    // codes, tables
      mbar_init(smem_u32(&ctl.c_empty[i]), 4);
    }
    for (int i = 0; i < S; ++i) {
      mbar_init(smem_u32(&ctl.full[i]), 5);       // four decode warps a CTA, the copies of the activations
      mbar_init(smem_u32(&ctl.empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&ctl.acc_full[i]), 1);
      mbar_init(smem_u32(&ctl.acc_empty[i]), 4);
    }
    mbar_init(smem_u32(&ctl.last_full), 1);
    ctl.abort_word = 0;
    ctl.sums = 0;
    mbar_fence_init();
  }
  if (warp == 5) {
    tmem_alloc(smem_u32(&ctl.tmem), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch_dependents();
  if constexpr (GROUPED) pdl_wait();             // the work list is written by the routing kernels
  const uint32_t tmem = ctl.tmem;
  TsWalk<FORM> walk(p, m_blocks);
  TsRun run;
  bool ok = true;

  if (warp >= 8) {
    // ---------------------------------------------------------------- decode
    const int grp = (warp - 8) >> 2, quad = warp & 3, row = quad * 32 + lane;
    const int total = static_cast<int>(walk.units());
    int c = grp;                                 // slots and phases are counted along: divisions by ring lengths take longer than the decode
    uint32_t c_phase = 0, a_phase = 1;
    for (int n = grp; ok && n < total; n += kTsGroups) {
      ok = mbar_wait_park(smem_u32(&ctl.c_full[c]), c_phase, abort_flag);
      uint32_t out[32];
      ts_decode<FMT>(cs + c * kC, 0, row, out);
      if (ok && n >= S) ok = mbar_wait_park(smem_u32(&ctl.empty[grp]), a_phase, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const uint32_t to = tmem + kTsTmemA + grp * 64 + (static_cast<uint32_t>(quad * 32) << 16);
      tmem_st_32x32(to, out);
      uint32_t out2[32];
      ts_decode<FMT>(cs + c * kC, 1, row, out2);
      tmem_st_32x32(to + 32, out2);
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl.c_empty[c]));
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl.full[grp]));
      c += kTsGroups;
      if (c >= NC) { c -= NC; c_phase ^= 1u; }
      a_phase ^= 1u;
    }
    if constexpr (!GROUPED) {
      // the last run, if it is a part: group g takes its rows from 32 (g + 1) on, every fifth 32
      int runs = 0;
      while (walk.next(p, run)) ++runs;
      if (runs > 0 && run.parts > 1 && run.rows > 32) {
        ok = __all_sync(0xffffffffu, ok && mbar_wait_park(smem_u32(&ctl.last_full), 0, abort_flag));
        pdl_wait();
        tc_fence_after();
        ts_part(p, run, tmem + ((runs - 1) & 1) * 128, quad, lane, 32 * (grp + 1), 160);
        asm volatile("bar.arrive 2, 640;" ::: "memory");
      }
    }
  } else if (warp == 4 || warp == 7) {
    // ------------------------------- codes (warp 4) and their tables (warp 7): a copy takes its thread longer than a unit's share of the decode
    if (lane == 0) {
      const bool tables = warp == 7;
      const uint32_t bytes = tables ? ts_meta(FMT) : ts_codes();
      int n = 0, c = 0;
      uint32_t phase = 1;
      while (ok && walk.next(p, run)) {
        const size_t tile = static_cast<size_t>(run.tile);
        const uint8_t* src = tables ? p.meta + run.expert * p.group_meta_stride + (tile * p.meta_blocks + run.kb / p.meta_k_blocks) * ts_meta(FMT)
                                    : p.codes + run.expert * p.group_code_stride + (tile * p.k_blocks + run.kb) * ts_codes();
        int left = tables ? p.meta_k_blocks - run.kb % p.meta_k_blocks : 1;      // units before the next table
        for (int kb = run.kb; kb < run.kb_end; ++kb, ++n) {
          if (n >= NC) ok = mbar_wait_park(smem_u32(&ctl.c_empty[c]), phase, abort_flag);
          if (!ok) break;
          const uint32_t bar = smem_u32(&ctl.c_full[c]), dst = smem_u32(cs) + c * kC + (tables ? ts_codes() : 0);
          mbar_expect_tx(bar, bytes);
          bulk_g2s(dst, src, bytes, bar);
          if (--left == 0) { left = tables ? p.meta_k_blocks : 1; src += bytes; }
          if (++c == NC) { c = 0; phase ^= 1u; }
        }
      }
      if (*abort_flag) {                         // copies in flight land before the CTA goes (their barriers count other roles, which may be gone: a fixed time)
        const long long t0 = clock64();
        while (clock64() - t0 < kWaitBudgetCycles / 256) {
        }
      }
    }
  } else if (warp == 6) {
    // ------------------------------------------------------------ activations: a lane a copy
    if (lane == 0) tma_prefetch_desc(&tmap_x);
    pdl_wait();
    const int h = lane & 1, at = lane >> 1;
    const uint32_t mine = smem_u32(xs) + h * x_half + at * box_bytes;
    int n = 0, s = 0;
    uint32_t phase = 1;
    while (ok && walk.next(p, run)) {
      const int each = (run.rows + 15) & ~15, copies = (each + box - 1) / box, row = run.m0 + at * box;
      const uint32_t bytes = 2u * copies * box_bytes;
      int col = run.kb * kTsCols + h * 64;
      for (int kb = run.kb; kb < run.kb_end; ++kb, ++n, col += kTsCols) {
        if (n >= S) ok = __all_sync(0xffffffffu, mbar_wait_park(smem_u32(&ctl.empty[s]), phase, abort_flag));
        if (!ok) break;
        const uint32_t bar = smem_u32(&ctl.full[s]), dst = mine + s * x_bytes;
        if (lane == 0) mbar_expect_tx(bar, bytes);
        __syncwarp();
        if (at < copies) tma_load_2d(dst, &tmap_x, col, row, bar);
        if (++s == S) { s = 0; phase ^= 1u; }
      }
    }
    if (*abort_flag) {
      const long long t0 = clock64();
      while (clock64() - t0 < kWaitBudgetCycles / 256) {
      }
    }
  } else if (warp == 5) {
    // ------------------------------------------------------------------ MMAs
    const bool leader = elect_one();
    const uint64_t dx = umma_desc_sw128(smem_u32(xs));
    const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
    int runs = 0, s = 0;
    uint32_t phase = 0;
    TsRun next;
    bool more = walk.next(p, next);
    while (ok && more) {
      run = next;
      more = walk.next(p, next);
      const int b = runs & 1, used = runs >> 1;
      // (from lane 0: what the MMAs take has to be known to be the same in all lanes, or every one of them moves it to uniform registers)
      const uint32_t acc = tmem_u + b * 128, idesc = __shfl_sync(0xffffffffu, umma_idesc(kTileN, static_cast<uint32_t>(FORM == kTsOneBlock ? p.mb : (run.rows + 15) & ~15), 1u, 1u), 0);
      if (used > 0) ok = mbar_wait_park(smem_u32(&ctl.acc_empty[b]), (used - 1) & 1, abort_flag);
      for (int kb = run.kb; kb < run.kb_end; ++kb) {
        ok = __all_sync(0xffffffffu, ok && mbar_wait_park(smem_u32(&ctl.full[s]), phase, abort_flag));
        if (!ok) break;
        tc_fence_after();
        if (leader) {
          const uint64_t d = dx + (static_cast<uint32_t>(s) * x_bytes >> 4);
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_f16_ts(acc, tmem_u + kTsTmemA + s * 64 + h * 32 + k * 8, d + (h * x_half >> 4) + k * 2, idesc, kb > run.kb || h > 0 || k > 0);
          tc_commit(smem_u32(&ctl.empty[s]));
        }
        __syncwarp();
        if (++s == S) { s = 0; phase ^= 1u; }
      }
      if (!ok) break;
      if (leader) {
        tc_commit(smem_u32(&ctl.acc_full[b]));
        if (!more) tc_commit(smem_u32(&ctl.last_full));
      }
      __syncwarp();
      ++runs;
    }
  } else if (warp < 4) {
    // -------------------------------------------------------------- epilogue
    pdl_wait();
    int runs = 0;
    TsRun next;
    bool more = walk.next(p, next);
    while (more) {
      run = next;
      more = walk.next(p, next);
      const bool helped = !GROUPED && !more && run.parts > 1 && run.rows > 32;                // by the decode warps
      const int b = runs & 1, used = runs >> 1;
      ++runs;
      // after a wait that ran out the rest runs through on whatever is there: barriers stay aligned
      if (ok) ok = mbar_wait_park(smem_u32(&ctl.acc_full[b]), used & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      tc_fence_after();
      const uint32_t acc = tmem + b * 128;
      if (run.parts > 1) {
        ts_part(p, run, acc, warp, lane, 0, helped ? 160 : 32);
      } else {
        ts_out<FMT>(p, run, acc + (static_cast<uint32_t>(warp * 32) << 16), warp, lane);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl.acc_empty[b]));
      if (run.parts > 1) {
        if (helped) asm volatile("bar.sync 2, 640;" ::: "memory");
        else ts_bar();
        if (threadIdx.x == 0) {
          const uint32_t prev = atom_add_acq_rel_gpu(p.counters + run.sum, 1u);
          if (prev == static_cast<uint32_t>(run.parts) - 1u) {
            p.counters[run.sum] = 0;
            ctl.sum_tile[ctl.sums] = run.sum;
            ctl.sum_part[ctl.sums] = run.part;
            ctl.sum_parts[ctl.sums] = run.parts;
            ++ctl.sums;                          // the first and the last run of a CTA are all that can be parts
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  // tiles in parts that are complete with this CTA's: summed by all threads, two parts (most weights have no more) of several places in flight
  for (int d = 0; !GROUPED && d < ctl.sums; ++d) {
    const int parts = ctl.sum_parts[d], t = ctl.sum_tile[d], tile = BLOCKS ? t / m_blocks : t, m0 = BLOCKS ? (t - tile * m_blocks) * p.mb : 0, c0 = static_cast<int>(blockIdx.x) - ctl.sum_part[d], shift = p.swiglu ? 4 : 5;
    auto part = [&](int q, int at) { return __ldcg(reinterpret_cast<const float4*>(ts_slot(p, c0 + q, q) + at)); };
    auto out = [&](int i, auto sum) {
      const int m = i >> shift, j = i & ((1 << shift) - 1);
      if (p.swiglu) {
        float4 g = sum(m * kTileN + act_gate_col(j * 4)), u = sum(m * kTileN + act_gate_col(j * 4) + 16);
        g.x *= p.alpha; g.y *= p.alpha; g.z *= p.alpha; g.w *= p.alpha;
        u.x *= p.alpha; u.y *= p.alpha; u.z *= p.alpha; u.w *= p.alpha;
        store_act4(p, m0 + m, tile, j * 4, g, u);
      } else {
        sk_store4<FMT>(p, m0 + m, tile * kTileN + j * 4, sum(i * 4));
      }
    };
    const int n = (BLOCKS ? min(p.mb, p.M - m0) : p.M) << shift;
    if (parts == 2) {
      for (int i = threadIdx.x; i < n; i += 2 * kTsThreads) {
        const int i2 = i + kTsThreads;
        if (p.swiglu || i2 >= n) {               // (of gates and the others, four loads are on their way as it is)
          auto two = [&](int at) {
            float4 a = part(0, at);
            const float4 b = part(1, at);
            a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
            return a;
          };
          out(i, two);
          if (i2 < n) out(i2, two);
        } else {
          float4 a = part(0, i * 4), c = part(0, i2 * 4);
          const float4 b = part(1, i * 4), e = part(1, i2 * 4);
          a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
          c.x += e.x; c.y += e.y; c.z += e.z; c.w += e.w;
          out(i, [&](int) { return a; });
          out(i2, [&](int) { return c; });
        }
      }
    } else {
      auto all = [&](int at) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int q = 0; q < parts; ++q) {
          const float4 v = part(q, at);
          a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
        }
        return a;
      };
#pragma unroll 2
      for (int i = threadIdx.x; i < n; i += kTsThreads) out(i, all);
    }
  }
  if (threadIdx.x == 0 && ctl.abort_word) atomicExch(p.status, static_cast<uint32_t>(kErrBarrierTimeout));
}

template <int FMT, int FORM>
static int launch_ts(const CUtensorMap& tx, const WqGemmParams& p, int m_blocks, int box, int boxes, int grid, size_t smem, cudaStream_t stream) {
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -18;
  if (!configured[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(wq_gemm_ts_kernel<FMT, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
    if (e != cudaSuccess) return static_cast<int>(e);
    configured[dev] = true;
  }
  return static_cast<int>(launch(wq_gemm_ts_kernel<FMT, FORM>, dim3(static_cast<unsigned>(grid)), dim3(kTsThreads), smem, stream, tx, p, m_blocks, box, boxes));
}

// A matrix (mb = M), or with `items` the experts of a work list of at most `max_items` items of at most mb rows
static int ts_gemm(int fmt, const void* x, int ldx, const void* codes, const void* meta, void* y, int ldy, const void* residual, float alpha, int M, int mb, int N, int K,
                   int group_k, int swiglu, const void* items, int max_items, size_t code_stride, size_t meta_stride, void* workspace, long long workspace_bytes, void* counters,
                   void* status, void* stream) {
  if (fmt != kFmtCubic4 && fmt != kFmtAffine4 && fmt != kFmtNvfp4) return -11;
  if (M <= 0 || mb <= 0 || mb > 128 || N <= 0 || K <= 0 || K % kTsCols != 0 || ldx % 8 != 0 || (reinterpret_cast<uintptr_t>(x) & 15) != 0) return -10;
  if (fmt == kFmtCubic4 && group_k % kTsCols != 0) return -12;
  if (swiglu && (residual || (N % 32) != 0 || ldy < N / 2)) return -51;
  int dev = 0;
  static int sms[64] = {};
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -18;
  if (sms[dev] == 0 && cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -18;
  WqGemmParams p = {};
  p.codes = static_cast<const uint8_t*>(codes);
  p.meta = static_cast<const uint8_t*>(meta);
  p.y = static_cast<__nv_bfloat16*>(y);
  p.residual = static_cast<const __nv_bfloat16*>(residual);
  p.workspace = static_cast<float*>(workspace);
  p.counters = static_cast<uint32_t*>(counters);
  p.status = static_cast<uint32_t*>(status);
  p.M = M; p.N = N; p.K = K; p.ldy = ldy; p.alpha = alpha;
  p.swiglu = swiglu;
  p.mb = (mb + 15) / 16 * 16;
  p.k_blocks = K / kTsCols;
  p.meta_k_blocks = fmt == kFmtCubic4 ? group_k / kTsCols : 1;
  p.meta_blocks = (p.k_blocks + p.meta_k_blocks - 1) / p.meta_k_blocks;
  p.n_tiles = p.tiles = (N + kTileN - 1) / kTileN;
  p.group_tiles = static_cast<const int*>(items);
  p.group_code_stride = code_stride;
  p.group_meta_stride = meta_stride;
  const int m_blocks = items ? 1 : (M + p.mb - 1) / p.mb;
  const long long units = static_cast<long long>(p.tiles) * m_blocks * p.k_blocks, most = items ? static_cast<long long>(max_items) * p.tiles : units;
  if (units * sms[dev] >= (1ll << 32) || most * p.k_blocks >= (1ll << 31)) return -19;
  if (!items && (!workspace || !counters || workspace_bytes < 2ll * sms[dev] * p.mb * kTileN * 4)) return -13;
  int grid = static_cast<int>(most < sms[dev] ? most : sms[dev]);
  // Few tiles: parts of one tile each, so that a CTA has one run and joins one sum
  const int all = p.tiles * m_blocks;
  if (!items && 2 * all <= grid) {
    p.splits = grid / all < p.k_blocks ? grid / all : p.k_blocks;
    grid = p.splits * all;
  }
  const int box = p.mb < kTsBox ? p.mb : kTsBox, boxes = (p.mb + box - 1) / box;
  const size_t kC = ts_codes() + ts_meta(fmt), xb = static_cast<size_t>(kTsSlots) * box * boxes * 256;
  const int fit = static_cast<int>((232448 - 1024 - sizeof(TsCtl) - xb) / kC);
  p.c_stages = fit >= kTsMaxC ? kTsMaxC : fit / kTsGroups * kTsGroups;       // a slot belongs to one group
  const size_t smem = 1024 + xb + p.c_stages * kC + sizeof(TsCtl);
  CUtensorMap tx;
  if (make_tmap_bf16(&tx, x, M, K, ldx, box) != 0) return -20;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto go = [&](auto f) {
    constexpr int F = decltype(f)::value;
    if (items) return launch_ts<F, kTsGrouped>(tx, p, m_blocks, box, boxes, grid, smem, st);
    if (m_blocks > 1) return launch_ts<F, kTsRowBlocks>(tx, p, m_blocks, box, boxes, grid, smem, st);
    return launch_ts<F, kTsOneBlock>(tx, p, m_blocks, box, boxes, grid, smem, st);
  };
  switch (fmt) {
    case kFmtCubic4: return go(std::integral_constant<int, kFmtCubic4>());
    case kFmtAffine4: return go(std::integral_constant<int, kFmtAffine4>());
    default: return go(std::integral_constant<int, kFmtNvfp4>());
  }
}

}  // namespace cb

extern "C" {

// Arguments as cb_wq_gemm_skinny; 4-bit weights, K a multiple of 128; M in blocks of one size of up to 128 rows.
// `workspace`: two fp32 tiles of a block's rows rounded up to 16 for every SM; `counters`: one for every weight tile and block.
int cb_wq_gemm_ts(int fmt, const void* x, int ldx, const void* codes, const void* meta, void* y, int ldy, const void* residual, float alpha, int M, int N, int K,
                  int group_k, int swiglu, void* workspace, long long workspace_bytes, void* counters, void* status, void* stream) {
  if (M <= 0) return -10;
  const int blocks = (M + 127) / 128, mb = (M + blocks - 1) / blocks;
  return cb::ts_gemm(fmt, x, ldx, codes, meta, y, ldy, residual, alpha, M, mb, N, K, group_k, swiglu, nullptr, 0, 0, 0, workspace, workspace_bytes, counters, status, stream);
}

// The grouped form over a device work list {count, then {expert, first row, rows}} of at most `max_items` items of at most `mb` <= 128 rows.
int cb_wq_gemm_ts_grouped(int fmt, const void* x, int ldx, const void* codes, const void* meta, void* y, int ldy, float alpha, int total_rows, int N, int K, int group_k,
                          int swiglu, const void* tiles, int max_items, int mb, long long code_stride, long long meta_stride, void* status, void* stream) {
  if (!tiles || max_items <= 0) return -40;
  return cb::ts_gemm(fmt, x, ldx, codes, meta, y, ldy, nullptr, alpha, total_rows, mb, N, K, group_k, swiglu, tiles, max_items, static_cast<size_t>(code_stride),
                     static_cast<size_t>(meta_stride), nullptr, 0, nullptr, status, stream);
}

}  // extern "C"
