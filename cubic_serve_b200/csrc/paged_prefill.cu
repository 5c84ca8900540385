// Paged GQA attention over the quantized KV cache for portions of prompts, on the tensor cores of tcgen05 (page layout: kv_layout.cuh;
// row blocks and arithmetic: paged_attn.cu).
//
// What bounds it.  The general kernel gives a row block (16 MMA rows: 16 / G positions x G heads) a CTA of its own: a prompt's pages
// are fetched and converted to f16 once per 16 / G positions, and mma.sync re-reads every operand for 16 rows.  Here a CTA takes
// eight consecutive row blocks -- the 128 rows of one tcgen05 MMA -- and converts a step of 64 tokens once for all of them.
// Codes stay exact in f16; the scales, one per token and 32 channels, multiply fp32 scores (K) and probabilities before their
// rounding to f16 (V), as in the general kernel.  So a step makes four score tiles in tensor memory, one per channel group, and four
// scaled copies of the probabilities; what is left to pay is that arithmetic: 256 fp32 multiply-adds, 256 multiplications, 128
// packings and 64 exponentials a row and step.
// One softmax warp a scheduler pays it, and waits for its own tensor-memory loads besides: about 5800 cycles a step.  General kernel -> this one
// (with 8 us of launch and cold operands), 32 heads over 8: 8 x 1024 tokens 707 -> 513 us, 4 x 256 behind 2048 284 -> 234; 6 bit, 64 over 4,
// 3 x 500 195 -> 136; one prompt of 331 tokens 29 -> 33, which the caller leaves to the general kernel.  What keeps values that are not finite
// to those who see them, and scaled probabilities in the range of f16, costs 0.5 % of it.
//
// Roles: warps 0-3 own a row a thread (softmax needs no exchange: tensor-memory lane = row); warps 4-7 convert raw pages, which warp 4
// copies two steps ahead, to the swizzled operands (K as [token][channel], V transposed as [channel][token]); warp 8 issues the MMAs.
// The scores of step i + 1 are computed while the softmax of step i runs.  Row blocks of several requests may meet in a CTA: it walks
// their steps one request after the other, rows of another request taking part with probability zero.  The output accumulator stays
// in tensor memory and is rescaled only when a row's maximum has grown by more than a factor of four (2 in the log2 domain): until
// then probabilities relative to the older maximum are at most 4.  A step with a V scale of which four times is more than f16 holds
// rescales at any growth, so that scaled probabilities have the range that they have in the general kernel.
// Every wait is bounded; on a timeout the roles run through without waiting, the status word is set and tensor memory is freed.
#include "paged_attn.cuh"

namespace cb {

static constexpr int kPfRows = 128;
static constexpr int kPfBlocks = kPfRows / 16;
static constexpr int kPfPages = 4;                       // pages of a step
static constexpr int kPfTok = kPfPages * kPageTokens;    // 64
static constexpr int kPfThreads = 288;
static constexpr float kPfGrowth = 2.f;
static constexpr float kPfGrowthScale = 65504.f / 4.f;   // largest V scale of a step with probabilities up to 4
static constexpr uint32_t kPfWild = 1, kPfLarge = 2;     // a V scale of the step is not finite, is finite and above that
static constexpr uint32_t kPfTmemCols = 512, kPfTmemO = 256;      // four score tiles of 64 columns, then 128 columns of output

struct PfRun {
  int first, end, req, total, pages, steps;              // row blocks [first, end) of the CTA, tokens that the last of them sees
};
struct __align__(1024) PfSmem {
  uint8_t q[2 * kPfRows * 128];                          // f16 [64-channel half][row][128 B], 16-byte chunk ^ (row & 7)
  uint8_t p[4][kPfRows * 128];                           // f16 [channel group][row][64 tokens]
  uint8_t k[2][2 * kPfTok * 128];                        // f16 [stage][64-channel half][token]
  uint8_t v[2][kD * 128];                                // f16 [stage][channel][64 tokens]
  float ks[2][4 * kPfTok], vs[2][4 * kPfTok];            // [stage][channel group][token]
  uint32_t vs_kind[2][2];                                // [stage][half of the tokens] kPfWild, kPfLarge
  uint64_t raw_full[2], kv_full[2], kv_free[2], s_full, s_free, p_full, pv_done;
  PfRun run[kPfBlocks];
  int runs, steps;
  uint32_t tmem, abort_word;
};

__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]),
      "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]),
      "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Where a role stands in the CTA's list of steps: runs one after the other.
struct PfWalk {
  int run = 0, step = 0;
  __device__ __forceinline__ void advance(const PfSmem& sm) {
    if (++step == sm.run[run].steps) { step = 0; ++run; }
  }
};

__device__ __forceinline__ uint4 conv8(uint2 w, uint32_t bias) {        // eight codes in order -> eight f16
  return make_uint4(u8x2_to_f16x2(w.x, 0x5140u, bias), u8x2_to_f16x2(w.x, 0x5342u, bias), u8x2_to_f16x2(w.y, 0x5140u, bias), u8x2_to_f16x2(w.y, 0x5342u, bias));
}

// One step's codes and scales into operands.  What a step's tail has beyond `pages` becomes zeros, and so do V scales from `visible`
// on: those slots may hold anything, and a probability of zero has to stay zero.
template <int KBITS, int VBITS>
__device__ __forceinline__ void pf_convert(PfSmem& sm, int b, const uint8_t* raw, int stride, const KvLayout& lay, int pages, int visible, int tid) {
  constexpr uint32_t kb = KBITS == 8 ? 0x64806480u : KBITS == 6 ? 0x64206420u : 0x64086408u;
  constexpr uint32_t vb = VBITS == 8 ? 0x64806480u : VBITS == 6 ? 0x64206420u : 0x64086408u;
  // K: an item is 16 channels (8 bit) or 32 (4 and 6 bit) of a token
  constexpr int kItems = KBITS == 8 ? kPageTokens * 8 : kPageTokens * 4;
#pragma unroll 4
  for (int i = tid; i < kPfPages * kItems; i += 128) {
    const int page = i / kItems, r = i % kItems, tok = r & 15, blk = r >> 4, sw = tok & 7;
    uint4* row = reinterpret_cast<uint4*>(sm.k[b] + (KBITS == 8 ? blk >> 2 : blk >> 1) * (kPfTok * 128) + (page * 16 + tok) * 128);
    const int c = KBITS == 8 ? (blk & 3) * 2 : (blk & 1) * 4;
    if (page >= pages) {
#pragma unroll
      for (int j = 0; j < (KBITS == 8 ? 2 : 4); ++j) row[(c + j) ^ sw] = make_uint4(0u, 0u, 0u, 0u);
      continue;
    }
    const uint8_t* src = raw + page * stride;
    const uint4 w = *reinterpret_cast<const uint4*>(src + blk * 256 + tok * 16);
    if constexpr (KBITS == 8) {
      row[c ^ sw] = conv8(make_uint2(w.x, w.y), kb);
      row[(c + 1) ^ sw] = conv8(make_uint2(w.z, w.w), kb);
    } else {
      const uint32_t n[4] = {w.x, w.y, w.z, w.w};
      uint32_t lo[4], hi[4];
      uint4 hb = make_uint4(0u, 0u, 0u, 0u);
      if constexpr (KBITS == 6) hb = *reinterpret_cast<const uint4*>(src + kPageTokens * kD / 2 + blk * 128 + (tok & 7) * 16);
      const uint32_t hw[4] = {hb.x, hb.y, hb.z, hb.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        lo[q] = n[q] & 0x0F0F0F0Fu;
        hi[q] = (n[q] >> 4) & 0x0F0F0F0Fu;
        if constexpr (KBITS == 6) {
          lo[q] |= (tok < 8 ? hw[q] : hw[q] << 4) & 0x30303030u;
          hi[q] |= (tok < 8 ? hw[q] >> 2 : hw[q] << 2) & 0x30303030u;
        }
      }
      row[c ^ sw] = conv8(make_uint2(lo[0], lo[1]), kb);
      row[(c + 1) ^ sw] = conv8(make_uint2(lo[2], lo[3]), kb);
      row[(c + 2) ^ sw] = conv8(make_uint2(hi[0], hi[1]), kb);
      row[(c + 3) ^ sw] = conv8(make_uint2(hi[2], hi[3]), kb);
    }
  }
  // V: lane = token pair of the step; a warp's lanes take four neighbouring chunks (4 channels) in turns, shifted so that neither the
  // loads nor the stores, one 32-bit pair per channel row, meet in a bank
  const int lane = tid & 31, page = lane >> 3, pair = lane & 7, j8 = lane >> 2;
  const uint8_t* src = raw + page * stride + lay.v_code_off;
#pragma unroll 2
  for (int c0 = (tid >> 5) * 8; c0 < (tid >> 5) * 8 + 8; c0 += 4)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = c0 + ((j8 + i) & 3), at = c ^ ((pair & 3) << 2);
      uint4 w = make_uint4(0u, 0u, 0u, 0u);
      if (page < pages) {
        if constexpr (VBITS == 8) {
          w = conv8(*reinterpret_cast<const uint2*>(src + pair * 256 + at * 8), vb);
        } else {
          const uint32_t n = *reinterpret_cast<const uint32_t*>(src + pair * 128 + at * 4);
          uint32_t e = n & 0x0F0F0F0Fu, o = (n >> 4) & 0x0F0F0F0Fu;
          if constexpr (VBITS == 6) {
            const uint32_t hw = *reinterpret_cast<const uint32_t*>(src + kPageTokens * kD / 2 + (pair & 3) * 128 + at * 4);
            e |= (pair < 4 ? hw : hw << 4) & 0x30303030u;
            o |= (pair < 4 ? hw >> 2 : hw << 2) & 0x30303030u;
          }
          w = conv8(make_uint2(prmt(e, o, 0x5140u), prmt(e, o, 0x7362u)), vb);
        }
      }
      uint8_t* dst = sm.v[b] + 4 * c * 128 + (lane & 3) * 4;
      const int sw = (4 * c) & 7;
      *reinterpret_cast<uint32_t*>(dst + ((j8 ^ sw) << 4)) = w.x;
      *reinterpret_cast<uint32_t*>(dst + 128 + ((j8 ^ (sw + 1)) << 4)) = w.y;
      *reinterpret_cast<uint32_t*>(dst + 256 + ((j8 ^ (sw + 2)) << 4)) = w.z;
      *reinterpret_cast<uint32_t*>(dst + 384 + ((j8 ^ (sw + 3)) << 4)) = w.w;
    }
  {
    const int tok = tid & 63, pg = tok >> 4;
    const bool is_v = tid >= 64;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (pg < pages && (!is_v || tok < visible))
      s = *reinterpret_cast<const float4*>(raw + pg * stride + (is_v ? lay.v_scale_off : lay.k_scale_off) + (tok & 15) * 16);
    float* dst = (is_v ? sm.vs[b] : sm.ks[b]) + tok;
    dst[0] = s.x; dst[kPfTok] = s.y; dst[2 * kPfTok] = s.z; dst[3 * kPfTok] = s.w;
    if (is_v) {                                          // both warps of V
      auto of = [](float x) { return fabsf(x) <= kPfGrowthScale ? 0u : fabsf(x) < INFINITY ? kPfLarge : kPfWild; };
      const uint32_t kind = __reduce_or_sync(0xffffffffu, of(s.x) | of(s.y) | of(s.z) | of(s.w));
      if ((tid & 31) == 0) sm.vs_kind[b][(tid >> 5) & 1] = kind;
    }
  }
}

// A step with a V scale that is not finite: zero times it, and it may be another request's, is not zero.  The warp of the MMAs clears the
// tokens that a row does not see before it multiplies (in the softmax warps, which have no register left for it, the check alone was 1 % of the kernel).
// `rb_qcount`, `rb_ctx`: of the CTA's first row block; `blocks`: from there to the last; `i`: the step.
__device__ __noinline__ void pf_unseen(PfSmem& sm, const int* rb_qcount, const int* rb_ctx, int blocks, int G, int i, int lane) {
  int run = 0;
  while (i >= sm.run[run].steps) i -= sm.run[run++].steps;
  for (int row = lane; row < kPfRows; row += 32) {
    const int blk = row >> 4, qp = (row & 15) / G;
    int sees = 0;
    if (blk >= sm.run[run].first && blk < sm.run[run].end && blk < blocks && qp < rb_qcount[blk]) sees = rb_ctx[blk] + qp - i * kPfTok;
    for (int c = max(sees, 0) >> 3; c < 8; ++c) {
      const int keep = min(max(sees - 8 * c, 0), 8);                 // tokens of the chunk
      for (int cg = 0; cg < 4; ++cg) {
        uint32_t* at = reinterpret_cast<uint32_t*>(sm.p[cg] + row * 128 + ((c ^ (row & 7)) << 4));
#pragma unroll
        for (int k = 0; k < 4; ++k) at[k] &= keep >= 2 * k + 2 ? 0xFFFFFFFFu : keep == 2 * k + 1 ? 0xFFFFu : 0u;
      }
    }
  }
  fence_proxy_async_smem();
  __syncwarp();
}

template <int KBITS, int VBITS>
__global__ void __launch_bounds__(kPfThreads, 1)
paged_prefill_kernel(const AttnParams p, const int row_blocks) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  PfSmem& sm = *reinterpret_cast<PfSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* raw = reinterpret_cast<uint8_t*>(&sm + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int kvh = blockIdx.x;
  const int rb0 = static_cast<int>(gridDim.y - 1 - blockIdx.y) * kPfBlocks;     // the blocks that see most first
  const int stride = (p.lay.blob_bytes + 127) & ~127;
  volatile uint32_t* abort_flag = &sm.abort_word;
  if (tid == 0) {
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&sm.raw_full[b]), 1);
      mbar_init(smem_u32(&sm.kv_full[b]), 4);
      mbar_init(smem_u32(&sm.kv_free[b]), 1);
    }
    mbar_init(smem_u32(&sm.s_full), 1);
    mbar_init(smem_u32(&sm.s_free), 4);
    mbar_init(smem_u32(&sm.p_full), 4);
    mbar_init(smem_u32(&sm.pv_done), 1);
    sm.abort_word = 0;
    mbar_fence_init();
  }
  if (warp == 8) {
    tmem_alloc(smem_u32(&sm.tmem), kPfTmemCols);
    tmem_relinquish();
  }
  pdl_wait();
  pdl_launch_dependents();
  if (tid == 32) {
    // the CTA's row blocks as runs of one request
    int n = 0, steps = 0;
    for (int i = 0; i < kPfBlocks && rb0 + i < row_blocks;) {
      if (p.rb_qcount[rb0 + i] <= 0) { ++i; continue; }
      PfRun r;
      r.first = i;
      r.req = p.rb_req[rb0 + i];
      r.total = 0;
      while (i < kPfBlocks && rb0 + i < row_blocks && p.rb_qcount[rb0 + i] > 0 && p.rb_req[rb0 + i] == r.req) {
        r.total = max(r.total, p.rb_ctx[rb0 + i] + p.rb_qcount[rb0 + i] - 1);
        ++i;
      }
      r.end = i;
      r.pages = (r.total + kPageTokens - 1) / kPageTokens;
      r.steps = (r.pages + kPfPages - 1) / kPfPages;
      if (r.steps > 0) {
        sm.run[n++] = r;
        steps += r.steps;
      }
    }
    sm.runs = n;
    sm.steps = steps;
  }
  // rows: thread = row of the MMA
  const int G = p.G, blk = tid >> 4, rb = rb0 + blk;
  int qp = 0, hh = 0, limit = 0;
  __nv_bfloat16* out_row = nullptr;
  if (warp < 4) {
    qp = (tid & 15) / G;
    hh = (tid & 15) - qp * G;
    const int qcount = rb < row_blocks ? p.rb_qcount[rb] : 0;
    const bool valid = qp < qcount;
    const __nv_bfloat16* q = nullptr;
    if (valid) {
      limit = p.rb_ctx[rb] + qp;
      const size_t at = (static_cast<size_t>(p.rb_qstart[rb] + qp) * p.Hq + kvh * G + hh) * kD;
      q = p.q + at;
      out_row = p.out + at;
    }
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      uint4 w = make_uint4(0u, 0u, 0u, 0u);
      if (valid) w = reinterpret_cast<const uint4*>(q)[c];
      uint32_t x[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x[j]));
        x[j] = pack_f16x2(v.x * p.scale_log2, v.y * p.scale_log2);
      }
      *reinterpret_cast<uint4*>(sm.q + (c >> 3) * (kPfRows * 128) + tid * 128 + (((c & 7) ^ (tid & 7)) << 4)) = make_uint4(x[0], x[1], x[2], x[3]);
    }
    fence_proxy_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem;
  const int steps = sm.steps;
  bool ok = true;

  if (warp == 8) {
    // ------------------------------------------------------------------ MMAs
    const bool leader = elect_one();
    const uint32_t idesc_s = umma_idesc(kPfRows, kPfTok, 0u, 0u), idesc_o = umma_idesc(kPfRows, 32u, 0u, 0u);
    const uint64_t dq = umma_desc_sw128(smem_u32(sm.q)), dp = umma_desc_sw128(smem_u32(sm.p[0]));
    const uint64_t dk = umma_desc_sw128(smem_u32(sm.k[0])), dv = umma_desc_sw128(smem_u32(sm.v[0]));
    auto scores = [&](int i) {
      const int b = i & 1;
      if (ok) ok = mbar_wait_park(smem_u32(&sm.kv_full[b]), (i >> 1) & 1, abort_flag);
      if (ok && i > 0) ok = mbar_wait_park(smem_u32(&sm.s_free), (i - 1) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      tc_fence_after();
      if (ok && leader) {
#pragma unroll
        for (int cg = 0; cg < 4; ++cg)
#pragma unroll
          for (int k = 0; k < 2; ++k)
            umma_f16(tmem + cg * kPfTok, dq + ((cg >> 1) * (kPfRows * 128) >> 4) + (cg & 1) * 4 + k * 2,
                     dk + ((b * 2 + (cg >> 1)) * (kPfTok * 128) >> 4) + (cg & 1) * 4 + k * 2, idesc_s, k > 0);
        tc_commit(smem_u32(&sm.s_full));
      }
      __syncwarp();
    };
    if (steps > 0) scores(0);
    for (int i = 0; i < steps; ++i) {
      if (i + 1 < steps) scores(i + 1);
      const int b = i & 1;
      if (ok) ok = mbar_wait_park(smem_u32(&sm.p_full), i & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if ((sm.vs_kind[b][0] | sm.vs_kind[b][1]) & kPfWild) pf_unseen(sm, p.rb_qcount + rb0, p.rb_ctx + rb0, row_blocks - rb0, p.G, i, lane);
      tc_fence_after();
      if (ok && leader) {
#pragma unroll
        for (int cg = 0; cg < 4; ++cg)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_f16(tmem + kPfTmemO + cg * 32, dp + (cg * (kPfRows * 128) >> 4) + k * 2, dv + ((b * kD + cg * 32) * 128 >> 4) + k * 2, idesc_o, i > 0 || k > 0);
        tc_commit(smem_u32(&sm.kv_free[b]));
        tc_commit(smem_u32(&sm.pv_done));
      }
      __syncwarp();
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------ conversion
    const int ct = tid - 128;
    PfWalk ahead, at;
    // lanes 0..3 of warp 4 copy a page of a step each
    auto issue = [&](int i) {
      const PfRun& r = sm.run[ahead.run];
      const int n = min(kPfPages, r.pages - ahead.step * kPfPages), b = i & 1;
      if (lane == 0) mbar_expect_tx(smem_u32(&sm.raw_full[b]), n * p.lay.blob_bytes);
      __syncwarp();
      if (lane < n) {
        const int page = p.page_table[static_cast<size_t>(r.req) * p.max_pages + ahead.step * kPfPages + lane];
        bulk_g2s(smem_u32(raw + (b * kPfPages + lane) * stride), p.cache + (static_cast<size_t>(page) * p.Hkv + kvh) * p.lay.blob_bytes, p.lay.blob_bytes,
                 smem_u32(&sm.raw_full[b]));
      }
      ahead.advance(sm);
    };
    int issued = 0;
    if (warp == 4)
      for (; issued < 2 && issued < steps; ++issued) issue(issued);
    for (int i = 0; i < steps; ++i) {
      const int b = i & 1;
      const PfRun& r = sm.run[at.run];
      if (ok) ok = mbar_wait_park(smem_u32(&sm.raw_full[b]), (i >> 1) & 1, abort_flag);
      if (ok && i >= 2) ok = mbar_wait_park(smem_u32(&sm.kv_free[b]), ((i >> 1) - 1) & 1, abort_flag);
      pf_convert<KBITS, VBITS>(sm, b, raw + b * kPfPages * stride, stride, p.lay, min(kPfPages, r.pages - at.step * kPfPages), r.total - at.step * kPfTok, ct);
      at.advance(sm);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sm.kv_full[b]));
      asm volatile("bar.sync 2, 128;" ::: "memory");     // the raw pages have been read by all four warps
      if (warp == 4 && i + 2 < steps && __all_sync(0xffffffffu, ok)) {
        issue(i + 2);
        ++issued;
      }
    }
    if (warp == 4 && *abort_flag) {                      // copies in flight land (for a bounded time) before the CTA goes
      const long long t0 = clock64();
      for (int i = max(0, issued - 2); i < issued; ++i)
        while (!mbar_try_wait(smem_u32(&sm.raw_full[i & 1]), (i >> 1) & 1) && clock64() - t0 < kWaitBudgetCycles / 8) {
        }
    }
  } else {
    // --------------------------------------------------------------- softmax
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    float m = -INFINITY, l = 0.f;
    PfWalk at;
    for (int i = 0; i < steps; ++i) {
      const int b = i & 1, tok0 = at.step * kPfTok;
      const PfRun& r = sm.run[at.run];
      const int sees = (blk >= r.first && blk < r.end) ? limit - tok0 : 0;       // tokens of the step that this row sees
      at.advance(sm);
      if (ok) ok = mbar_wait_park(smem_u32(&sm.kv_full[b]), (i >> 1) & 1, abort_flag);      // the scales
      if (ok) ok = mbar_wait_park(smem_u32(&sm.s_full), i & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      tc_fence_after();
      float2 s[kPfTok / 2];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t a[4][16];
#pragma unroll
        for (int cg = 0; cg < 4; ++cg) tmem_ld_32x16(tmem + lane_base + cg * kPfTok + c * 16, a[cg]);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int cg = 0; cg < 4; ++cg) {
            const float4 k = *reinterpret_cast<const float4*>(sm.ks[b] + cg * kPfTok + c * 16 + j * 4);
            const float2 x = make_float2(__uint_as_float(a[cg][4 * j]), __uint_as_float(a[cg][4 * j + 1])), y = make_float2(__uint_as_float(a[cg][4 * j + 2]), __uint_as_float(a[cg][4 * j + 3]));
            float2& s0 = s[c * 8 + 2 * j];
            float2& s1 = s[c * 8 + 2 * j + 1];
            s0 = cg == 0 ? __fmul2_rn(x, make_float2(k.x, k.y)) : __ffma2_rn(x, make_float2(k.x, k.y), s0);
            s1 = cg == 0 ? __fmul2_rn(y, make_float2(k.z, k.w)) : __ffma2_rn(y, make_float2(k.z, k.w), s1);
          }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sm.s_free));
      if (sees < kPfTok) {
#pragma unroll
        for (int j = 0; j < kPfTok / 2; ++j) {
          if (2 * j >= sees) s[j].x = -INFINITY;
          if (2 * j + 1 >= sees) s[j].y = -INFINITY;
        }
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int j = 0; j < kPfTok / 2; ++j) mx[j & 3] = fmaxf(mx[j & 3], fmaxf(s[j].x, s[j].y));
      const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      float alpha = 1.f;
      const bool grew = top > m + ((sm.vs_kind[b][0] | sm.vs_kind[b][1]) & kPfLarge ? 0.f : kPfGrowth) || (m == -INFINITY && top > m);
      if (grew) {
        alpha = fast_exp2(m - top);
        m = top;
        l *= alpha;
      }
      const float use = m == -INFINITY ? 0.f : m;
      const float2 less = make_float2(-use, -use);
      float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int j = 0; j < kPfTok / 2; ++j) {
        const float2 d = __fadd2_rn(s[j], less);
        s[j] = make_float2(fast_exp2(d.x), fast_exp2(d.y));
        sum[j & 1] = __fadd2_rn(sum[j & 1], s[j]);
      }
      l += (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
      // the previous product has read the probabilities and written the output
      if (ok && i > 0) ok = mbar_wait_park(smem_u32(&sm.pv_done), (i - 1) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (i > 0 && __any_sync(0xffffffffu, grew)) {
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t o[32];
          tmem_ld_32x32(tmem + lane_base + kPfTmemO + c * 32, o);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
          tmem_st_32x32(tmem + lane_base + kPfTmemO + c * 32, o);
        }
        tmem_st_wait();
      }
#pragma unroll
      for (int cg = 0; cg < 4; ++cg)
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float4 v0 = *reinterpret_cast<const float4*>(sm.vs[b] + cg * kPfTok + c * 8), v1 = *reinterpret_cast<const float4*>(sm.vs[b] + cg * kPfTok + c * 8 + 4);
          const float2 w0 = __fmul2_rn(s[4 * c], make_float2(v0.x, v0.y)), w1 = __fmul2_rn(s[4 * c + 1], make_float2(v0.z, v0.w));
          const float2 w2 = __fmul2_rn(s[4 * c + 2], make_float2(v1.x, v1.y)), w3 = __fmul2_rn(s[4 * c + 3], make_float2(v1.z, v1.w));
          *reinterpret_cast<uint4*>(sm.p[cg] + tid * 128 + ((c ^ (tid & 7)) << 4)) =
              make_uint4(pack_f16x2(w0.x, w0.y), pack_f16x2(w1.x, w1.y), pack_f16x2(w2.x, w2.y), pack_f16x2(w3.x, w3.y));
        }
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sm.p_full));
    }
    if (steps == 0) {                                    // no row sees a token
      if (out_row != nullptr) {
#pragma unroll
        for (int j = 0; j < 16; ++j) reinterpret_cast<uint4*>(out_row)[j] = make_uint4(0u, 0u, 0u, 0u);
      }
    } else {
      if (ok) ok = mbar_wait_park(smem_u32(&sm.pv_done), (steps - 1) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      tc_fence_after();
      const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t o[32];
        tmem_ld_32x32(tmem + lane_base + kPfTmemO + c * 32, o);
        tmem_ld_wait();
        if (out_row != nullptr) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) w[k] = pack_bf16x2(__uint_as_float(o[8 * j + 2 * k]) * inv, __uint_as_float(o[8 * j + 2 * k + 1]) * inv);
            *reinterpret_cast<uint4*>(out_row + c * 32 + j * 8) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) tmem_dealloc(tmem, kPfTmemCols);
  if (tid == 0 && sm.abort_word) atomicExch(p.status, static_cast<uint32_t>(kErrBarrierTimeout));
}

template <int KB, int VB>
static int launch_prefill(const AttnParams& p, int row_blocks, cudaStream_t st) {
  const int stride = (p.lay.blob_bytes + 127) & ~127;
  const size_t smem = sizeof(PfSmem) + 1024 + static_cast<size_t>(2) * kPfPages * stride;
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -18;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(paged_prefill_kernel<KB, VB>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    configured[dev] = true;
  }
  return static_cast<int>(launch(paged_prefill_kernel<KB, VB>, dim3(p.Hkv, (row_blocks + kPfBlocks - 1) / kPfBlocks), dim3(kPfThreads), smem, st, p, row_blocks));
}

}  // namespace cb

extern "C" {

// Arguments as cb_paged_attn without splits; meant for row blocks that mostly follow one another in one request.
int cb_paged_prefill(const void* q, void* out, const void* cache, const void* page_table, const void* rb_req, const void* rb_qstart, const void* rb_qcount,
                     const void* rb_ctx, int row_blocks, int Hq, int Hkv, int D, int max_pages, int k_bits, int v_bits, float scale, int splits, void* partial,
                     void* counters, void* status, void* stream) {
  using namespace cb;
  if (row_blocks <= 0) return 0;
  if (splits > 1) return -14;
  AttnParams p;
  const int bad = make_attn_params(p, q, out, cache, page_table, rb_req, rb_qstart, rb_qcount, rb_ctx, Hq, Hkv, D, max_pages, k_bits, v_bits, scale, 1, partial, counters,
                                   status);
  if (bad) return bad;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return with_kv_bits(k_bits, v_bits, [&](auto kb, auto vb) { return launch_prefill<decltype(kb)::value, decltype(vb)::value>(p, row_blocks, st); });
}

}  // extern "C"
