// Weight-quantized GEMM for decode batches of more rows than wq_gemm_skinny.cu takes: y[M, N] = x[M, K] * W[N, K]^T, 4-bit weights, M <= 128
// (packed weight layout and decode arithmetic: wq_gemm_common.cuh).
//
// What bounds it.  The other tcgen05 kernels write a decoded tile to shared memory, in a stage that also holds the activation tile and (per-tile
// kernel) the codes: six to eight stages of 27 KB, each of which goes release -> copies -> 2000 to 3000 cycles -> decode -> fence -> MMA before
// it comes back, 500 to 750 cycles a k-block of 64 columns whatever the rows.  Here the decoded tile is the MMA's A operand in TENSOR MEMORY: a decoding thread owns
// a weight row, its 64 decoded columns are one tcgen05.st.  Shared memory then holds nothing but copies, in two rings of their own: codes
// (10 KB a stage, up to 12 stages, on their way before the previous kernel is done) and activations.  A unit of the pipeline is 128 columns: the one thread that
// waits, counts and issues copies or MMAs for a stage takes 150 to 200 cycles for it, whatever it moves.
// Few-row, per-tile or persistent kernel -> this one, Cubic weights not in L2, 17 / 48 / 128 rows, one B200: 24576 x 4096 37.6 / 38.7 / 44.5 -> 23.9 / 26.9 / 36.9
// us (floor 8.7), 4096 x 12288 24.4 / 25.5 / 28.3 -> 16.0 / 17.5 / 22.6 (4.3), 6144 x 4096 17.9 / 18.9 / 21.4 -> 12.4 / 13.9 / 18.9 (2.2).  About 9 us of
// each are start (4300 cycles to the first codes), the last run's sums and the sum of parts.
//
// Split.  One CTA per SM; the units of all weight tiles are dealt evenly, a tile in a few runs whose fp32 sums the last one to arrive adds in
// the order of K (deterministic).  Roles: warps 0-3 epilogue (from one of two accumulators while the next run fills the other one), warp 4 codes, warp 7 their tables, warp 5 MMAs, warp 6 activations, warps 8-23 decode: group g of four takes every fourth unit.
// Every wait is bounded; on a timeout the roles leave, the status word is set and tensor memory is freed.
#include "wq_gemm_common.cuh"
#include "launch.cuh"

namespace cb {

static constexpr int kTsThreads = 768;
static constexpr int kTsGroups = 4;              // of decode warps
static constexpr int kTsCols = 128;              // K columns of a unit: two k-blocks of the packed layout
static constexpr int kTsSlots = 4;               // decoded units in tensor memory, 64 columns each
static constexpr int kTsMaxC = 12;
static constexpr int kTsScratch = kTileN + 4;    // floats of a row of the epilogue's staging
static constexpr uint32_t kTsTmemA = 256;        // first column of the decoded tiles; accumulators below
static_assert(kTsSlots % kTsGroups == 0 && kTsMaxC % kTsGroups == 0, "a slot belongs to one group");

struct __align__(16) TsCtl {
  uint64_t c_full[kTsMaxC], c_empty[kTsMaxC], full[kTsSlots], empty[kTsSlots], acc_full[2], acc_empty[2];
  float scratch[16][kTsScratch];
  int sum_tile[2], sum_part[2], sum_parts[2], sums;      // tiles whose last part was this CTA's
  uint32_t tmem, abort_word;
};

// A run of units of one tile.
struct TsRun {
  int tile, kb, kb_end, part, parts;
};
// The deal; every role walks the same list.  p.splits > 0: CTA c has part c % splits of tile c / splits; else the units of all tiles are dealt evenly.
struct TsWalk {
  uint32_t u, u_end, total;
  __device__ __forceinline__ TsWalk(const WqGemmParams& p) {
    const uint32_t kbs = static_cast<uint32_t>(p.k_blocks);
    total = static_cast<uint32_t>(p.n_tiles) * kbs;
    if (p.splits > 0) {
      const uint32_t parts = static_cast<uint32_t>(p.splits), tile = blockIdx.x / parts, part = blockIdx.x - tile * parts;
      u = tile * kbs + kbs * part / parts;
      u_end = tile * kbs + kbs * (part + 1) / parts;
    } else {
      u = static_cast<uint32_t>(static_cast<unsigned long long>(total) * blockIdx.x / gridDim.x);
      u_end = static_cast<uint32_t>(static_cast<unsigned long long>(total) * (blockIdx.x + 1) / gridDim.x);
    }
  }
  __device__ __forceinline__ bool next(const WqGemmParams& p, TsRun& r) {
    if (u >= u_end) return false;
    const uint32_t kbs = static_cast<uint32_t>(p.k_blocks), t = u / kbs, first = t * kbs, end = min(u_end, first + kbs);
    r.tile = static_cast<int>(t);
    r.kb = static_cast<int>(u - first);
    r.kb_end = static_cast<int>(end - first);
    if (p.splits > 0) {
      r.parts = p.splits;
      r.part = static_cast<int>(blockIdx.x) - r.tile * p.splits;
    } else {
      // CTA that owns unit v: the largest c with floor(total * c / ctas) <= v
      const unsigned long long ctas = gridDim.x;
      const uint32_t c0 = static_cast<uint32_t>(((first + 1ull) * ctas - 1ull) / total), c1 = static_cast<uint32_t>(((first + static_cast<unsigned long long>(kbs)) * ctas - 1ull) / total);
      r.parts = static_cast<int>(c1 - c0 + 1u);
      r.part = static_cast<int>(blockIdx.x - c0);
    }
    u = end;
    return true;
  }
};

__device__ __forceinline__ void ts_umma_bf16(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void ts_tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]),
      "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]),
      "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}

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

// Partial sums of part q of a tile whose first part is CTA c0's: [row][128]
__device__ __forceinline__ float* ts_slot(const WqGemmParams& p, int c0, int q) {
  return p.workspace + (static_cast<size_t>(c0 + q) * 2 + (q == 0 ? 1 : 0)) * p.mb * kTileN;
}
// Four features of a row, or four activations of gate and up rows; sum(col): the tile's sums of four of its 128 features
template <int FMT, typename Sum>
__device__ __forceinline__ void ts_write(const WqGemmParams& p, int tile, int m, int i, Sum&& sum) {
  if (p.swiglu) {
    float4 g = sum(act_gate_col(i * 4)), u = sum(act_gate_col(i * 4) + 16);
    g.x *= p.alpha; g.y *= p.alpha; g.z *= p.alpha; g.w *= p.alpha;
    u.x *= p.alpha; u.y *= p.alpha; u.z *= p.alpha; u.w *= p.alpha;
    store_act4(p, m, tile, i * 4, g, u);
  } else {
    sk_store4<FMT>(p, m, tile * kTileN + i * 4, sum(i * 4));
  }
}

__device__ __forceinline__ void ts_bar() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// k_blocks counts units here, meta_k_blocks units of a table; c_stages: depth of the code ring
template <int FMT>
__global__ void __launch_bounds__(kTsThreads, 1)
wq_gemm_ts_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ WqGemmParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  constexpr uint32_t kC = ts_codes() + ts_meta(FMT);
  const uint32_t x_half = static_cast<uint32_t>(p.mb) * 128u, x_bytes = 2 * x_half;
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
      mbar_init(smem_u32(&ctl.full[i]), 5);      // four decode warps, the copy of the activations
      mbar_init(smem_u32(&ctl.empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&ctl.acc_full[i]), 1);
      mbar_init(smem_u32(&ctl.acc_empty[i]), 4);
    }
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
  const uint32_t tmem = ctl.tmem;
  TsWalk walk(p);
  TsRun run;
  bool ok = true;

  if (warp >= 8) {
    // ---------------------------------------------------------------- decode
    const int grp = (warp - 8) >> 2, quad = warp & 3, row = quad * 32 + lane;
    const int total = static_cast<int>(walk.u_end - walk.u);      // k-blocks of the CTA
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
        ts_tmem_st32(to, out);
        uint32_t out2[32];
        ts_decode<FMT>(cs + c * kC, 1, row, out2);
        ts_tmem_st32(to + 32, out2);
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctl.c_empty[c]));
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctl.full[grp]));
        c += kTsGroups;
        if (c >= NC) { c -= NC; c_phase ^= 1u; }
        a_phase ^= 1u;
    }
  } else if (warp == 4 || warp == 7) {
    // ------------------------------- codes (warp 4) and their tables (warp 7): a copy takes its thread longer than a unit's share of the decode
    if (lane == 0) {
      const bool tables = warp == 7;
      const uint32_t bytes = tables ? ts_meta(FMT) : ts_codes();
      int n = 0, c = 0;
      uint32_t phase = 1;
      while (ok && walk.next(p, run)) {
        const uint8_t* src = tables ? p.meta + (static_cast<size_t>(run.tile) * p.meta_blocks + run.kb / p.meta_k_blocks) * ts_meta(FMT)
                                    : p.codes + (static_cast<size_t>(run.tile) * p.k_blocks + run.kb) * ts_codes();
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
    // ------------------------------------------------------------ activations
    if (lane == 0) {
      tma_prefetch_desc(&tmap_x);
      pdl_wait();
      int n = 0, s = 0;
      uint32_t phase = 1;
      while (ok && walk.next(p, run)) {
        for (int kb = run.kb; kb < run.kb_end; ++kb, ++n) {
          if (n >= S) ok = mbar_wait_park(smem_u32(&ctl.empty[s]), phase, abort_flag);
          if (!ok) break;
          mbar_expect_tx(smem_u32(&ctl.full[s]), x_bytes);
#pragma unroll
          for (int h = 0; h < 2; ++h) tma_load_2d(smem_u32(xs) + s * x_bytes + h * x_half, &tmap_x, kb * kTsCols + h * 64, 0, smem_u32(&ctl.full[s]));
          if (++s == S) { s = 0; phase ^= 1u; }
        }
      }
      if (*abort_flag) {
        const long long t0 = clock64();
        while (clock64() - t0 < kWaitBudgetCycles / 256) {
        }
      }
    }
  } else if (warp == 5) {
    // ------------------------------------------------------------------ MMAs
    const bool leader = elect_one();
    const uint32_t idesc = umma_idesc(kTileN, static_cast<uint32_t>(p.mb), 1u, 1u);
    const uint64_t dx = umma_desc_sw128(smem_u32(xs));
    int runs = 0, s = 0;
    uint32_t phase = 0;
    while (ok && walk.next(p, run)) {
      const int b = runs & 1, used = runs >> 1;
      const uint32_t acc = tmem + b * 128;
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
              ts_umma_bf16(acc, tmem + kTsTmemA + s * 64 + h * 32 + k * 8, d + (h * x_half >> 4) + k * 2, idesc, kb > run.kb || h > 0 || k > 0);
          tc_commit(smem_u32(&ctl.empty[s]));
        }
        __syncwarp();
        if (++s == S) { s = 0; phase ^= 1u; }
      }
      if (!ok) break;
      if (leader) tc_commit(smem_u32(&ctl.acc_full[b]));
      __syncwarp();
      ++runs;
    }
  } else if (warp < 4) {
    // -------------------------------------------------------------- epilogue
    pdl_wait();
    int runs = 0;
    while (walk.next(p, run)) {
      const int b = runs & 1, used = runs >> 1;
      ++runs;
      // after a wait that ran out the rest runs through on whatever is there: barriers stay aligned
      if (ok) ok = mbar_wait_park(smem_u32(&ctl.acc_full[b]), used & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      tc_fence_after();
      float* own = ts_slot(p, blockIdx.x - run.part, run.part);
      const int per = p.swiglu ? 16 : 32, shift = p.swiglu ? 4 : 5;
      const uint32_t acc = tmem + b * 128 + (static_cast<uint32_t>(warp * 32) << 16);
      if (run.parts > 1) {
#pragma unroll 1
        for (int c = 0; c < p.M; c += 32) {      // (columns behind the rows hold nothing, and are not written)
          uint32_t r[32];
          tmem_ld_32x32(acc + c, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (c + j < p.M) __stcg(own + (c + j) * kTileN + warp * 32 + lane, __uint_as_float(r[j]));
        }
      } else {
#pragma unroll 1
        for (int c = 0; c < p.M; c += 16) {
          uint32_t r[16];
          tmem_ld_32x16(acc + c, r);
          tmem_ld_wait();
          const int rows = min(16, p.M - c);
#pragma unroll
          for (int j = 0; j < 16; ++j) ctl.scratch[j][warp * 32 + lane] = __uint_as_float(r[j]);
          ts_bar();
#pragma unroll 4
          for (int i = threadIdx.x; i < rows * per; i += 128)
            ts_write<FMT>(p, run.tile, c + (i >> shift), i & (per - 1), [&](int col) { return *reinterpret_cast<const float4*>(&ctl.scratch[i >> shift][col]); });
          ts_bar();
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl.acc_empty[b]));
      if (run.parts > 1) {
        ts_bar();
        if (threadIdx.x == 0) {
          const uint32_t prev = atom_add_acq_rel_gpu(p.counters + run.tile, 1u);
          if (prev == static_cast<uint32_t>(run.parts) - 1u) {
            p.counters[run.tile] = 0;
            ctl.sum_tile[ctl.sums] = run.tile;
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
  if (warp == 5) tmem_dealloc(tmem, 512);
  // tiles in parts that are complete with this CTA's: summed by all threads, each of a tile's parts in flight at once
  for (int d = 0; d < ctl.sums; ++d) {
    const int parts = ctl.sum_parts[d], c0 = static_cast<int>(blockIdx.x) - ctl.sum_part[d], shift = p.swiglu ? 4 : 5;
#pragma unroll 2
    for (int i = threadIdx.x; i < p.M << shift; i += kTsThreads) {
      const int m = i >> shift;
      ts_write<FMT>(p, ctl.sum_tile[d], m, i & ((1 << shift) - 1), [&](int col) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int q = 0; q < parts; ++q) {
          const float4 v = __ldcg(reinterpret_cast<const float4*>(ts_slot(p, c0, q) + m * kTileN + col));
          a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
        }
        return a;
      });
    }
  }
  if (threadIdx.x == 0 && ctl.abort_word) atomicExch(p.status, static_cast<uint32_t>(kErrBarrierTimeout));
}

template <int FMT>
static int launch_ts(const CUtensorMap& tx, const WqGemmParams& p, int grid, size_t smem, cudaStream_t stream) {
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -18;
  if (!configured[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(wq_gemm_ts_kernel<FMT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
    if (e != cudaSuccess) return static_cast<int>(e);
    configured[dev] = true;
  }
  return static_cast<int>(launch(wq_gemm_ts_kernel<FMT>, dim3(static_cast<unsigned>(grid)), dim3(kTsThreads), smem, stream, tx, p));
}

}  // namespace cb

extern "C" {

// Arguments as cb_wq_gemm_skinny; 4-bit weights, M <= 128, K a multiple of 128.  `workspace`: two fp32 tiles of the rows rounded up to 16 for every SM.
int cb_wq_gemm_ts(int fmt, const void* x, int ldx, const void* codes, const void* meta, void* y, int ldy, const void* residual, float alpha, int M, int N, int K,
                  int group_k, int swiglu, void* workspace, long long workspace_bytes, void* counters, void* status, void* stream) {
  using namespace cb;
  if (fmt != kFmtCubic4 && fmt != kFmtAffine4 && fmt != kFmtNvfp4) return -11;
  if (M <= 0 || M > 128 || N <= 0 || K <= 0 || K % kTsCols != 0 || ldx % 8 != 0 || (reinterpret_cast<uintptr_t>(x) & 15) != 0) return -10;
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
  p.mb = (M + 15) / 16 * 16;
  p.k_blocks = K / kTsCols;
  p.meta_k_blocks = fmt == kFmtCubic4 ? group_k / kTsCols : 1;
  p.meta_blocks = (p.k_blocks + p.meta_k_blocks - 1) / p.meta_k_blocks;
  p.n_tiles = (N + kTileN - 1) / kTileN;
  const long long units = static_cast<long long>(p.n_tiles) * p.k_blocks;
  if (units >= (1ll << 31)) return -19;
  if (!workspace || !counters || workspace_bytes < 2ll * sms[dev] * p.mb * kTileN * 4) return -13;
  int grid = static_cast<int>(units < sms[dev] ? units : sms[dev]);
  // Few tiles: parts of one tile each, so that a CTA has one run and joins one sum
  p.splits = 0;
  if (2 * p.n_tiles <= grid) {
    int parts = grid / p.n_tiles;
    if (parts > p.k_blocks) parts = p.k_blocks;
    p.splits = parts;
    grid = parts * p.n_tiles;
  }
  const size_t kC = ts_codes() + ts_meta(fmt), xb = static_cast<size_t>(kTsSlots) * p.mb * 256, budget = 232448 - 1024 - sizeof(TsCtl);
  const int fit = static_cast<int>((budget - xb) / kC);
  p.c_stages = fit >= kTsMaxC ? kTsMaxC : fit / kTsGroups * kTsGroups;       // a slot belongs to one group
  const size_t smem = 1024 + xb + p.c_stages * kC + sizeof(TsCtl);
  CUtensorMap tx;
  if (make_tmap_bf16(&tx, x, M, K, ldx, p.mb) != 0) return -20;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (fmt) {
    case kFmtCubic4: return launch_ts<kFmtCubic4>(tx, p, grid, smem, st);
    case kFmtAffine4: return launch_ts<kFmtAffine4>(tx, p, grid, smem, st);
    default: return launch_ts<kFmtNvfp4>(tx, p, grid, smem, st);
  }
}

}  // extern "C"
