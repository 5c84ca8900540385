// Paged GQA attention over the quantized KV cache, decode and chunked-prefill rows.
//
// Counterpart of the reference's paged_decode_native.cu:282 (one CTA per row /
// kv-head tile / KV split, fused INT8/INT4 dequant, split-KV with in-kernel
// last-arriver merge).  Differences that matter on B200:
//   * whole (page, kv-head) blobs (codes + scales of K and V) arrive with ONE
//     bulk async copy each into a per-warp multi-stage ring, completion on an
//     mbarrier -- the kernel is a pure HBM stream;
//   * the cache is stored pre-permuted (kv_layout.cuh) so MMA fragments are
//     plain 32/64-bit shared loads; int8 -> f16 conversion is one byte-permute
//     plus one packed subtract; group scales are applied to the 4 fp32
//     accumulators of a channel group (K) or folded into P (V), never per code;
//   * a row block is 16 MMA rows = (16 / G) consecutive query positions x G
//     query heads of one kv head, so one general kernel serves speculative
//     review rows, short portions of prompts and decode rows beside them.
//
// Steps of decode rows alone, up to eight rows a block, take the decode form below (paged_decode_kernel); longer portions of prompts
// take paged_prefill.cu where the caller estimates that it is the faster one.
//
// Waits are bounded; on a timeout the CTA records Status and exits cleanly.
#include "paged_attn.cuh"

namespace cb {

static constexpr int kAttnWarps = 4;
#ifdef CB_ATTN_OCC4
static constexpr int kAttnStages = 3;
static constexpr int kAttnMinCtas = 4;
#else
static constexpr int kAttnStages = 4;
static constexpr int kAttnMinCtas = 1;
#endif
// UPPER = false: MMA rows 8..15 of the block hold no query (decode: one position x G <= 8 heads), so their scores,
// softmax state and output rescaling are skipped; the tensor-core instructions still compute them, at no cost.
template <int KBITS, int VBITS, bool UPPER>
__device__ __forceinline__ void process_page(const uint8_t* blob, const KvLayout& lay, const uint32_t (&qf)[8][4],
                                             WarpState& st, int page_tok0, int limit_lo, int limit_hi, int g,
                                             int t4) {
  // limit_lo / limit_hi: number of visible tokens for row g / row g+8
  const float* ksc = reinterpret_cast<const float*>(blob + lay.k_scale_off);
  const float* vsc = reinterpret_cast<const float*>(blob + lay.v_scale_off);
  const uint8_t* vcodes = blob + lay.v_code_off;
  float s[2][4];
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int c = 0; c < 4; ++c) s[nt][c] = 0.f;

  // ---- S = Q K^T, one channel group (2 k-steps) at a time, scaled per (token, group)
#pragma unroll
  for (int cg = 0; cg < 4; ++cg) {
    float acc[2][4];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[nt][c] = 0.f;
    if (KBITS == 8) {
#pragma unroll
      for (int jh = 0; jh < 2; ++jh) {
        const int j = cg * 2 + jh;
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const uint32_t w = *reinterpret_cast<const uint32_t*>(blob + j * 256 + (nt * 8 + g) * 16 + t4 * 4);
          const uint32_t b0 = u8x2_to_f16x2(w, 0x5140u, 0x64806480u);
          const uint32_t b1 = u8x2_to_f16x2(w, 0x5342u, 0x64806480u);
          mma_f16(acc[nt], qf[j], b0, b1);
        }
      }
    } else if (KBITS == 6) {
      // nibble plane as for 4 bits; one 32-bit word of high bits serves both tokens (g and g + 8) of this lane,
      // every 2-bit field already at the byte of its code (kv_layout.cuh)
      const uint32_t hb = *reinterpret_cast<const uint32_t*>(blob + kPageTokens * kD / 2 + cg * 128 + g * 16 + t4 * 4);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const uint32_t w = *reinterpret_cast<const uint32_t*>(blob + cg * 256 + (nt * 8 + g) * 16 + t4 * 4);
        const uint32_t h1 = nt == 0 ? hb : (hb << 4);
        const uint32_t h2 = nt == 0 ? (hb >> 2) : (hb << 2);
        const uint32_t lo = (w & 0x0F0F0F0Fu) | (h1 & 0x30303030u);
        const uint32_t hi = ((w >> 4) & 0x0F0F0F0Fu) | (h2 & 0x30303030u);
        mma_f16(acc[nt], qf[cg * 2], u8x2_to_f16x2(lo, 0x5140u, 0x64206420u), u8x2_to_f16x2(lo, 0x5342u, 0x64206420u));
        mma_f16(acc[nt], qf[cg * 2 + 1], u8x2_to_f16x2(hi, 0x5140u, 0x64206420u),
                u8x2_to_f16x2(hi, 0x5342u, 0x64206420u));
      }
    } else {
      // 4-bit: one 32-bit word = this lane's 4 channels of both k-steps of the group
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const uint32_t w = *reinterpret_cast<const uint32_t*>(blob + cg * 256 + (nt * 8 + g) * 16 + t4 * 4);
        const uint32_t lo = w & 0x0F0F0F0Fu, hi = (w >> 4) & 0x0F0F0F0Fu;
        mma_f16(acc[nt], qf[cg * 2], u8x2_to_f16x2(lo, 0x5140u, 0x64086408u), u8x2_to_f16x2(lo, 0x5342u, 0x64086408u));
        mma_f16(acc[nt], qf[cg * 2 + 1], u8x2_to_f16x2(hi, 0x5140u, 0x64086408u),
                u8x2_to_f16x2(hi, 0x5342u, 0x64086408u));
      }
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const float k0 = ksc[(nt * 8 + 2 * t4) * 4 + cg], k1 = ksc[(nt * 8 + 2 * t4 + 1) * 4 + cg];
      s[nt][0] = fmaf(acc[nt][0], k0, s[nt][0]);
      s[nt][1] = fmaf(acc[nt][1], k1, s[nt][1]);
      if (UPPER) {
        s[nt][2] = fmaf(acc[nt][2], k0, s[nt][2]);
        s[nt][3] = fmaf(acc[nt][3], k1, s[nt][3]);
      }
    }
  }
  // ---- causal / length mask and online softmax (log2 domain; Q carries the scale)
  float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int c = 0; c < (UPPER ? 4 : 2); ++c) {
      const int tok = page_tok0 + nt * 8 + 2 * t4 + (c & 1);
      const int lim = (c < 2) ? limit_lo : limit_hi;
      if (tok >= lim) s[nt][c] = -INFINITY;
      mx[c >> 1] = fmaxf(mx[c >> 1], s[nt][c]);
    }
  float alpha[2] = {1.f, 1.f}, muse[2] = {0.f, 0.f};
#pragma unroll
  for (int r = 0; r < (UPPER ? 2 : 1); ++r) {
    mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
    mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
    const float mnew = fmaxf(st.m[r], mx[r]);
    muse[r] = (mnew == -INFINITY) ? 0.f : mnew;
    alpha[r] = fast_exp2(st.m[r] - muse[r]);  // exp2(-inf) = 0 on the first page
    st.m[r] = mnew;
    st.l[r] *= alpha[r];
  }
  float pr[2][4];
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (UPPER || c < 2) {
        pr[nt][c] = fast_exp2(s[nt][c] - muse[c >> 1]);
        st.l[c >> 1] += pr[nt][c];
      } else {
        pr[nt][c] = 0.f;
      }
    }
  // the running maximum settles after the first pages: skip the 64 multiplies when no row's maximum moved
  if (__any_sync(0xffffffffu, alpha[0] != 1.f || (UPPER && alpha[1] != 1.f))) {
#pragma unroll
    for (int n = 0; n < 16; ++n) {
      st.o[n][0] *= alpha[0];
      st.o[n][1] *= alpha[0];
      if (UPPER) {
        st.o[n][2] *= alpha[1];
        st.o[n][3] *= alpha[1];
      }
    }
  }
  // ---- O += P V, V group scales folded into P per channel group
#pragma unroll
  for (int cg = 0; cg < 4; ++cg) {
    // slots past the longest visible length may hold stale bytes (even NaN bit
    // patterns): their scale is forced to zero so that 0 * scale stays 0
    const int vis = max(limit_lo, limit_hi) - page_tok0;
    const float v00 = (2 * t4 < vis) ? vsc[(2 * t4) * 4 + cg] : 0.f;
    const float v01 = (2 * t4 + 1 < vis) ? vsc[(2 * t4 + 1) * 4 + cg] : 0.f;
    const float v10 = (8 + 2 * t4 < vis) ? vsc[(8 + 2 * t4) * 4 + cg] : 0.f;
    const float v11 = (9 + 2 * t4 < vis) ? vsc[(8 + 2 * t4 + 1) * 4 + cg] : 0.f;
    uint32_t a[4];
    a[0] = pack_f16x2(pr[0][0] * v00, pr[0][1] * v01);
    a[1] = UPPER ? pack_f16x2(pr[0][2] * v00, pr[0][3] * v01) : 0u;
    a[2] = pack_f16x2(pr[1][0] * v10, pr[1][1] * v11);
    a[3] = UPPER ? pack_f16x2(pr[1][2] * v10, pr[1][3] * v11) : 0u;
    const int chunk = (cg * 8 + g) ^ ((t4 & 3) << 2);
    if (VBITS == 8) {
      const uint2 lo = *reinterpret_cast<const uint2*>(vcodes + t4 * 256 + chunk * 8);
      const uint2 hi = *reinterpret_cast<const uint2*>(vcodes + (t4 + 4) * 256 + chunk * 8);
      mma_f16(st.o[cg * 4 + 0], a, u8x2_to_f16x2(lo.x, 0x5140u, 0x64806480u), u8x2_to_f16x2(hi.x, 0x5140u, 0x64806480u));
      mma_f16(st.o[cg * 4 + 1], a, u8x2_to_f16x2(lo.x, 0x5342u, 0x64806480u), u8x2_to_f16x2(hi.x, 0x5342u, 0x64806480u));
      mma_f16(st.o[cg * 4 + 2], a, u8x2_to_f16x2(lo.y, 0x5140u, 0x64806480u), u8x2_to_f16x2(hi.y, 0x5140u, 0x64806480u));
      mma_f16(st.o[cg * 4 + 3], a, u8x2_to_f16x2(lo.y, 0x5342u, 0x64806480u), u8x2_to_f16x2(hi.y, 0x5342u, 0x64806480u));
    } else {
      // byte = channel sub, low nibble = even token, high nibble = odd token
      const uint32_t lo = *reinterpret_cast<const uint32_t*>(vcodes + t4 * 128 + chunk * 4);
      const uint32_t hi = *reinterpret_cast<const uint32_t*>(vcodes + (t4 + 4) * 128 + chunk * 4);
      // spread nibbles: even tokens -> bytes (sub), odd tokens -> bytes (sub) of a second word
      uint32_t le = lo & 0x0F0F0F0Fu, lod = (lo >> 4) & 0x0F0F0F0Fu;
      uint32_t he = hi & 0x0F0F0F0Fu, hod = (hi >> 4) & 0x0F0F0F0Fu;
      if (VBITS == 6) {
        // high bits: one 32-bit word for both token pairs (t4 and t4 + 4) of this lane, fields in place
        const uint32_t hw = *reinterpret_cast<const uint32_t*>(vcodes + kPageTokens * kD / 2 + t4 * 128 + chunk * 4);
        le |= hw & 0x30303030u;
        lod |= (hw >> 2) & 0x30303030u;
        he |= (hw << 4) & 0x30303030u;
        hod |= (hw << 2) & 0x30303030u;
      }
      const uint32_t vbias = VBITS == 6 ? 0x64206420u : 0x64086408u;
#pragma unroll
      for (int sub = 0; sub < 4; ++sub) {
        // f16x2 (even tok, odd tok) of channel `sub`: byte `sub` of le and of lod
        const uint32_t pl = prmt(le, lod, sub | ((4u + sub) << 4));          // bytes: [e_sub, o_sub, x, x]
        const uint32_t ph = prmt(he, hod, sub | ((4u + sub) << 4));
        const uint32_t b0 = u8x2_to_f16x2(pl, 0x5140u, vbias);
        const uint32_t b1 = u8x2_to_f16x2(ph, 0x5140u, vbias);
        mma_f16(st.o[cg * 4 + sub], a, b0, b1);
      }
    }
  }
}

template <int KBITS, int VBITS>
__global__ void __launch_bounds__(kAttnWarps * 32, kAttnMinCtas)
paged_attn_kernel(const AttnParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t4 = lane & 3;
  const int kvh = blockIdx.x, rb = blockIdx.y, split = blockIdx.z;
  pdl_wait();
  pdl_launch_dependents();
  const int qcount = p.rb_qcount[rb];
  if (qcount <= 0) return;  // padding block (uniform across the CTA)
  const int req = p.rb_req[rb], qstart = p.rb_qstart[rb], ctx = p.rb_ctx[rb];
  const int G = p.G;
  const int blob_bytes = p.lay.blob_bytes;
  const int stage_stride = (blob_bytes + 127) & ~127;

  uint8_t* my_stages = smem + static_cast<size_t>(warp) * kAttnStages * stage_stride;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + static_cast<size_t>(kAttnWarps) * kAttnStages * stage_stride);
  uint64_t* my_bars = bars + warp * kAttnStages;
  __shared__ uint32_t abort_word;
  __shared__ uint32_t is_last;
  if (threadIdx.x == 0) { abort_word = 0; is_last = 0; }
  if (lane == 0) {
    for (int s = 0; s < kAttnStages; ++s) mbar_init(smem_u32(&my_bars[s]), 1);
    mbar_fence_init();
  }
  __syncthreads();
  volatile uint32_t* abort_flag = &abort_word;

  // rows of this lane: row g and row g+8; row r -> (query position r / G, head r % G)
  const int total_tokens = ctx + qcount - 1;
  const int total_pages = (total_tokens + kPageTokens - 1) / kPageTokens;
  const int pps = (total_pages + p.splits - 1) / p.splits;
  const int pg_lo = split * pps;
  const int pg_hi = min(total_pages, pg_lo + pps);

  // The first copies of this warp's page stream are issued before anything else: their DRAM latency then overlaps
  // the query load and conversion below instead of following them (every CTA pays this start-up once).
  const int* ptab = p.page_table + static_cast<size_t>(req) * p.max_pages;
  const int first = pg_lo + warp;
  const int my_pages = first < pg_hi ? (pg_hi - first + kAttnWarps - 1) / kAttnWarps : 0;
  auto issue = [&](int i, int page) {
    const int s = i % kAttnStages;
    const uint8_t* src = p.cache + (static_cast<size_t>(page) * p.Hkv + kvh) * blob_bytes;
    const uint32_t bar = smem_u32(&my_bars[s]);
    mbar_expect_tx(bar, blob_bytes);
    bulk_g2s(smem_u32(my_stages + s * stage_stride), src, blob_bytes, bar);
  };
  if (lane == 0) {
    int pg[kAttnStages];
#pragma unroll
    for (int i = 0; i < kAttnStages; ++i) pg[i] = i < my_pages ? ptab[first + i * kAttnWarps] : 0;   // loads first ...
#pragma unroll
    for (int i = 0; i < kAttnStages; ++i)
      if (i < my_pages) issue(i, pg[i]);                                                               // ... then copies
  }

  const bool upper_rows = qcount * G > 8;     // uniform over the CTA: do MMA rows 8..15 hold a query?
  int limit[2];
  uint32_t qf[8][4];
#pragma unroll
  for (int rr = 0; rr < 2; ++rr) {
    const int row = g + 8 * rr;
    const int qp = row / G, hh = row - qp * G;
    const bool valid = qp < qcount;
    limit[rr] = valid ? ctx + qp : 0;
    const __nv_bfloat16* qrow = p.q + (static_cast<size_t>(qstart + qp) * p.Hq + kvh * G + hh) * kD;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float f[4] = {0.f, 0.f, 0.f, 0.f};
      if (valid) {
        const uint2 raw = *reinterpret_cast<const uint2*>(qrow + j * 16 + t4 * 4);
        const __nv_bfloat162* bp = reinterpret_cast<const __nv_bfloat162*>(&raw);
        const float2 x = __bfloat1622float2(bp[0]), y = __bfloat1622float2(bp[1]);
        f[0] = x.x * p.scale_log2; f[1] = x.y * p.scale_log2;
        f[2] = y.x * p.scale_log2; f[3] = y.y * p.scale_log2;
      }
      qf[j][rr] = pack_f16x2(f[0], f[1]);       // a0 / a1 : k = 2*t4 .. (first half of the k-step)
      qf[j][2 + rr] = pack_f16x2(f[2], f[3]);   // a2 / a3 : k = 2*t4 + 8 ..
    }
  }

  WarpState st;
  st.m[0] = st.m[1] = -INFINITY;
  st.l[0] = st.l[1] = 0.f;
#pragma unroll
  for (int n = 0; n < 16; ++n)
#pragma unroll
    for (int c = 0; c < 4; ++c) st.o[n][c] = 0.f;

  // ---- per-warp page stream (set up before the query load, see above): pages pg_lo + warp, + 4, ...
  // The page id of the copy issued at the end of iteration i is loaded at the START of iteration i - 1, so that lane 0
  // never sits on a page-table load between two pages.
  int page_next = (lane == 0 && kAttnStages < my_pages) ? ptab[first + kAttnStages * kAttnWarps] : 0;
  bool ok = true;
  for (int i = 0; i < my_pages && ok; ++i) {
    const int s = i % kAttnStages;
    ok = mbar_wait_t<20>(smem_u32(&my_bars[s]), static_cast<uint32_t>(i / kAttnStages) & 1u, abort_flag);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) break;
    const int page_after = (lane == 0 && i + 1 + kAttnStages < my_pages) ? ptab[first + (i + 1 + kAttnStages) * kAttnWarps] : 0;
    if (upper_rows)
      process_page<KBITS, VBITS, true>(my_stages + s * stage_stride, p.lay, qf, st,
                                       (first + i * kAttnWarps) * kPageTokens, limit[0], limit[1], g, t4);
    else
      process_page<KBITS, VBITS, false>(my_stages + s * stage_stride, p.lay, qf, st,
                                        (first + i * kAttnWarps) * kPageTokens, limit[0], limit[1], g, t4);
    __syncwarp();
    if (lane == 0 && i + kAttnStages < my_pages) issue(i + kAttnStages, page_next);
    page_next = page_after;
  }
  // if a wait gave up, copies may still be in flight: give them a bounded time to land
  if (!ok && lane == 0) {
    for (int s = 0; s < kAttnStages; ++s) {
      const long long t0 = clock64();
      while (!mbar_try_wait(smem_u32(&my_bars[s]), 0) && !mbar_try_wait(smem_u32(&my_bars[s]), 1) &&
             clock64() - t0 < kWaitBudgetCycles / 8) {
      }
    }
  }
  // finish row sums across the 4 lanes sharing a row
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    st.l[r] += __shfl_xor_sync(0xffffffffu, st.l[r], 1);
    st.l[r] += __shfl_xor_sync(0xffffffffu, st.l[r], 2);
  }
  __syncthreads();  // all warps are done with their stage memory

  // ---- merge the 4 warps through shared memory: [warp][16 rows][D + 2]
  float* mg = reinterpret_cast<float*>(smem);
  constexpr int RS = kD + 2;
  {
    float* mine = mg + warp * 16 * RS;
#pragma unroll
    for (int n = 0; n < 16; ++n) {
      const int cgi = n >> 2, sub = n & 3;
      const int c0 = cgi * 32 + (2 * t4) * 4 + sub, c1 = cgi * 32 + (2 * t4 + 1) * 4 + sub;
      mine[g * RS + c0] = st.o[n][0];
      mine[g * RS + c1] = st.o[n][1];
      mine[(g + 8) * RS + c0] = st.o[n][2];
      mine[(g + 8) * RS + c1] = st.o[n][3];
    }
    if (t4 == 0) {
      mine[g * RS + kD] = st.m[0];
      mine[g * RS + kD + 1] = st.l[0];
      mine[(g + 8) * RS + kD] = st.m[1];
      mine[(g + 8) * RS + kD + 1] = st.l[1];
    }
  }
  __syncthreads();
  // thread -> (row = tid / 8, 16 channels starting at (tid % 8) * 16)
  const int row = threadIdx.x >> 3, cbase = (threadIdx.x & 7) * 16;
  float mstar = -INFINITY;
#pragma unroll
  for (int w = 0; w < kAttnWarps; ++w) mstar = fmaxf(mstar, mg[(w * 16 + row) * RS + kD]);
  float lsum = 0.f, ov[16];
#pragma unroll
  for (int c = 0; c < 16; ++c) ov[c] = 0.f;
#pragma unroll
  for (int w = 0; w < kAttnWarps; ++w) {
    const float mw = mg[(w * 16 + row) * RS + kD];
    const float f = (mw == -INFINITY) ? 0.f : fast_exp2(mw - mstar);
    lsum += f * mg[(w * 16 + row) * RS + kD + 1];
#pragma unroll
    for (int c = 0; c < 16; ++c) ov[c] += f * mg[(w * 16 + row) * RS + cbase + c];
  }
  const int qp = row / G, hh = row - qp * G;
  const bool row_valid = qp < qcount;
  __nv_bfloat16* orow = p.out + (static_cast<size_t>(qstart + qp) * p.Hq + kvh * G + hh) * kD + cbase;

  if (p.splits == 1) {
    if (row_valid) {
      const float inv = lsum > 0.f ? 1.f / lsum : 0.f;
      uint32_t pk[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) pk[c] = pack_bf16x2(ov[2 * c] * inv, ov[2 * c + 1] * inv);
      reinterpret_cast<uint4*>(orow)[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
      reinterpret_cast<uint4*>(orow)[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
    }
  } else {
    float* part = p.partial + ((static_cast<size_t>(rb) * p.Hkv + kvh) * p.splits + split) * 16 * RS;
#pragma unroll
    for (int c = 0; c < 16; ++c) part[row * RS + cbase + c] = ov[c];
    if ((threadIdx.x & 7) == 0) {
      part[row * RS + kD] = mstar;
      part[row * RS + kD + 1] = lsum;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      const uint32_t idx = rb * p.Hkv + kvh;
      const uint32_t prev = atomicAdd(&p.counters[idx], 1u);
      const uint32_t last = (prev == static_cast<uint32_t>(p.splits) - 1u) ? 1u : 0u;
      if (last) p.counters[idx] = 0;
      is_last = last;
    }
    __syncthreads();
    if (is_last) {
      __threadfence();
      const float* base = p.partial + (static_cast<size_t>(rb) * p.Hkv + kvh) * p.splits * 16 * RS;
      float ms = -INFINITY;
      for (int sp = 0; sp < p.splits; ++sp) ms = fmaxf(ms, __ldcg(base + (sp * 16 + row) * RS + kD));
      float ls = 0.f;
#pragma unroll
      for (int c = 0; c < 16; ++c) ov[c] = 0.f;
      for (int sp = 0; sp < p.splits; ++sp) {
        const float mw = __ldcg(base + (sp * 16 + row) * RS + kD);
        const float f = (mw == -INFINITY) ? 0.f : fast_exp2(mw - ms);
        ls += f * __ldcg(base + (sp * 16 + row) * RS + kD + 1);
#pragma unroll
        for (int c = 0; c < 16; ++c) ov[c] += f * __ldcg(base + (sp * 16 + row) * RS + cbase + c);
      }
      if (row_valid) {
        const float inv = ls > 0.f ? 1.f / ls : 0.f;
        uint32_t pk[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) pk[c] = pack_bf16x2(ov[2 * c] * inv, ov[2 * c + 1] * inv);
        reinterpret_cast<uint4*>(orow)[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        reinterpret_cast<uint4*>(orow)[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
      }
    }
  }
  if (threadIdx.x == 0 && abort_word) atomicExch(p.status, static_cast<uint32_t>(kErrBarrierTimeout));
}

// Decode form: row blocks of at most eight rows (one position of up to eight query heads per key / value head, or a few positions of
// fewer).  The cache is the MMA's 16-row operand -- S^T = K Q^T, O^T = V^T P^T -- so a page takes 16 MMAs where the general kernel
// takes 32 of which half the rows are empty, the output needs 32 registers a lane instead of 64, and four CTAs run on an SM
// instead of two; that is what the time hangs on, since a warp spends most of a page's life waiting for its own loads.  The
// code words are the same: what is a column pair's B operand there is a row's A operand here.  Probabilities change
// lanes by a matrix transpose after the V scale and the rounding to f16, the point where the general kernel rounds them.
// KV splits that would give a warp less than two pages are not used: one row over 700 tokens took 46 us in 32 splits, 7 in 6.
//
// Measured, INT8 K and V, 32 / 8 heads (general kernel -> this one): 256 rows of 1280 tokens 164 -> 124 us (753 MB: 6.1 TB/s), 48
// rows of 560 to 1500 33.5 -> 30.7, 7 of 900 to 2100 25.8 -> 13, 1 of 700 46 -> 7.
static constexpr int kDecStages = 3;
static constexpr int kDecRows = 8;
static constexpr int kDecMinPages = 2 * kAttnWarps;

__device__ __forceinline__ uint32_t transpose8(uint32_t a) {
  uint32_t r;
  asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(a));
  return r;
}

struct DecState {
  float m[2], l[2];          // rows 2 t and 2 t + 1: running max (log2 domain), this lane's part of the sum
  float o[8][4];             // [32-channel group * 2 + h]: channels 32 cg + 4 g + 2 h and the next one x the two rows
};

template <int KBITS, int VBITS>
__device__ __forceinline__ void decode_page(const uint8_t* blob, const KvLayout& lay, const uint32_t (&qf)[8][2], DecState& st, int tok0, const int (&limit)[2], int visible,
                                            int g, int t) {
  const uint8_t* vcodes = blob + lay.v_code_off;
  float s[4] = {0.f, 0.f, 0.f, 0.f};                     // tokens g and g + 8 x rows 2 t, 2 t + 1
  const float4 kl = *reinterpret_cast<const float4*>(blob + lay.k_scale_off + g * 16), kh = *reinterpret_cast<const float4*>(blob + lay.k_scale_off + (g + 8) * 16);
#pragma unroll
  for (int cg = 0; cg < 4; ++cg) {
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    if constexpr (KBITS == 8) {
#pragma unroll
      for (int jh = 0; jh < 2; ++jh) {
        const int j = cg * 2 + jh;
        const uint32_t w0 = *reinterpret_cast<const uint32_t*>(blob + j * 256 + g * 16 + t * 4), w1 = *reinterpret_cast<const uint32_t*>(blob + j * 256 + (g + 8) * 16 + t * 4);
        const uint32_t a[4] = {u8x2_to_f16x2(w0, 0x5140u, 0x64806480u), u8x2_to_f16x2(w1, 0x5140u, 0x64806480u), u8x2_to_f16x2(w0, 0x5342u, 0x64806480u),
                               u8x2_to_f16x2(w1, 0x5342u, 0x64806480u)};
        mma_f16(acc, a, qf[j][0], qf[j][1]);
      }
    } else {
      constexpr uint32_t bias = KBITS == 6 ? 0x64206420u : 0x64086408u;
      const uint32_t w0 = *reinterpret_cast<const uint32_t*>(blob + cg * 256 + g * 16 + t * 4), w1 = *reinterpret_cast<const uint32_t*>(blob + cg * 256 + (g + 8) * 16 + t * 4);
      uint32_t l0 = w0 & 0x0F0F0F0Fu, h0 = (w0 >> 4) & 0x0F0F0F0Fu, l1 = w1 & 0x0F0F0F0Fu, h1 = (w1 >> 4) & 0x0F0F0F0Fu;
      if constexpr (KBITS == 6) {
        const uint32_t hb = *reinterpret_cast<const uint32_t*>(blob + kPageTokens * kD / 2 + cg * 128 + g * 16 + t * 4);
        l0 |= hb & 0x30303030u;
        h0 |= (hb >> 2) & 0x30303030u;
        l1 |= (hb << 4) & 0x30303030u;
        h1 |= (hb << 2) & 0x30303030u;
      }
      const uint32_t a[4] = {u8x2_to_f16x2(l0, 0x5140u, bias), u8x2_to_f16x2(l1, 0x5140u, bias), u8x2_to_f16x2(l0, 0x5342u, bias), u8x2_to_f16x2(l1, 0x5342u, bias)};
      const uint32_t b[4] = {u8x2_to_f16x2(h0, 0x5140u, bias), u8x2_to_f16x2(h1, 0x5140u, bias), u8x2_to_f16x2(h0, 0x5342u, bias), u8x2_to_f16x2(h1, 0x5342u, bias)};
      mma_f16(acc, a, qf[cg * 2][0], qf[cg * 2][1]);
      mma_f16(acc, b, qf[cg * 2 + 1][0], qf[cg * 2 + 1][1]);
    }
    const float k0 = (&kl.x)[cg], k1 = (&kh.x)[cg];
    s[0] = fmaf(acc[0], k0, s[0]); s[1] = fmaf(acc[1], k0, s[1]);
    s[2] = fmaf(acc[2], k1, s[2]); s[3] = fmaf(acc[3], k1, s[3]);
  }
  float alpha[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    if (tok0 + g >= limit[r]) s[r] = -INFINITY;
    if (tok0 + g + 8 >= limit[r]) s[2 + r] = -INFINITY;
    float mx = fmaxf(s[r], s[2 + r]);
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
    const float m = fmaxf(st.m[r], mx), use = m == -INFINITY ? 0.f : m;
    alpha[r] = fast_exp2(st.m[r] - use);
    st.m[r] = m;
    s[r] = fast_exp2(s[r] - use);
    s[2 + r] = fast_exp2(s[2 + r] - use);
    st.l[r] = fmaf(st.l[r], alpha[r], s[r] + s[2 + r]);
  }
  if (__any_sync(0xffffffffu, alpha[0] != 1.f || alpha[1] != 1.f)) {
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int c = 0; c < 4; ++c) st.o[n][c] *= alpha[c & 1];
  }
  // slots past the longest visible length may hold stale bytes (even NaN bit patterns): their scale counts as zero
  float4 vl = make_float4(0.f, 0.f, 0.f, 0.f), vh = vl;
  if (tok0 + g < visible) vl = *reinterpret_cast<const float4*>(blob + lay.v_scale_off + g * 16);
  if (tok0 + g + 8 < visible) vh = *reinterpret_cast<const float4*>(blob + lay.v_scale_off + (g + 8) * 16);
#pragma unroll
  for (int cg = 0; cg < 4; ++cg) {
    const float v0 = (&vl.x)[cg], v1 = (&vh.x)[cg];
    const uint32_t b0 = transpose8(pack_f16x2(s[0] * v0, s[1] * v0)), b1 = transpose8(pack_f16x2(s[2] * v1, s[3] * v1));
    const int chunk = (cg * 8 + g) ^ (t << 2);
    uint32_t lo[4], hi[4];                                // token pairs t and t + 4 of four channels
    if constexpr (VBITS == 8) {
      const uint2 l = *reinterpret_cast<const uint2*>(vcodes + t * 256 + chunk * 8), h = *reinterpret_cast<const uint2*>(vcodes + (t + 4) * 256 + chunk * 8);
      lo[0] = u8x2_to_f16x2(l.x, 0x5140u, 0x64806480u); lo[1] = u8x2_to_f16x2(l.x, 0x5342u, 0x64806480u);
      lo[2] = u8x2_to_f16x2(l.y, 0x5140u, 0x64806480u); lo[3] = u8x2_to_f16x2(l.y, 0x5342u, 0x64806480u);
      hi[0] = u8x2_to_f16x2(h.x, 0x5140u, 0x64806480u); hi[1] = u8x2_to_f16x2(h.x, 0x5342u, 0x64806480u);
      hi[2] = u8x2_to_f16x2(h.y, 0x5140u, 0x64806480u); hi[3] = u8x2_to_f16x2(h.y, 0x5342u, 0x64806480u);
    } else {
      constexpr uint32_t bias = VBITS == 6 ? 0x64206420u : 0x64086408u;
      const uint32_t l = *reinterpret_cast<const uint32_t*>(vcodes + t * 128 + chunk * 4), h = *reinterpret_cast<const uint32_t*>(vcodes + (t + 4) * 128 + chunk * 4);
      uint32_t le = l & 0x0F0F0F0Fu, lod = (l >> 4) & 0x0F0F0F0Fu, he = h & 0x0F0F0F0Fu, hod = (h >> 4) & 0x0F0F0F0Fu;
      if constexpr (VBITS == 6) {
        const uint32_t hw = *reinterpret_cast<const uint32_t*>(vcodes + kPageTokens * kD / 2 + t * 128 + chunk * 4);
        le |= hw & 0x30303030u;
        lod |= (hw >> 2) & 0x30303030u;
        he |= (hw << 4) & 0x30303030u;
        hod |= (hw << 2) & 0x30303030u;
      }
      const uint32_t l01 = prmt(le, lod, 0x5140u), l23 = prmt(le, lod, 0x7362u), h01 = prmt(he, hod, 0x5140u), h23 = prmt(he, hod, 0x7362u);
      lo[0] = u8x2_to_f16x2(l01, 0x5140u, bias); lo[1] = u8x2_to_f16x2(l01, 0x5342u, bias);
      lo[2] = u8x2_to_f16x2(l23, 0x5140u, bias); lo[3] = u8x2_to_f16x2(l23, 0x5342u, bias);
      hi[0] = u8x2_to_f16x2(h01, 0x5140u, bias); hi[1] = u8x2_to_f16x2(h01, 0x5342u, bias);
      hi[2] = u8x2_to_f16x2(h23, 0x5140u, bias); hi[3] = u8x2_to_f16x2(h23, 0x5342u, bias);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t a[4] = {lo[2 * h], lo[2 * h + 1], hi[2 * h], hi[2 * h + 1]};
      mma_f16(st.o[cg * 2 + h], a, b0, b1);
    }
  }
}

template <int KBITS, int VBITS>
__global__ void __launch_bounds__(kAttnWarps * 32, 4)
paged_decode_kernel(const AttnParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  constexpr int RS = kD + 2;
  __shared__ __align__(8) uint64_t bars[kAttnWarps * kDecStages];
  __shared__ uint32_t abort_word, is_last;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int kvh = blockIdx.x, rb = blockIdx.y, split = blockIdx.z;
  pdl_wait();
  pdl_launch_dependents();
  const int qcount = p.rb_qcount[rb];
  if (qcount <= 0) return;                                // padding block (uniform across the CTA)
  const int req = p.rb_req[rb], qstart = p.rb_qstart[rb], ctx = p.rb_ctx[rb];
  const int G = p.G;
  const int total = ctx + qcount - 1, pages = (total + kPageTokens - 1) / kPageTokens;
  const int splits = max(1, min(p.splits, (pages + kDecMinPages - 1) / kDecMinPages));
  const int per = max(1, (pages + splits - 1) / splits);
  const int used = max(1, (pages + per - 1) / per);       // splits that have pages; rows that see no token are written, as zeros
  if (split >= used) return;
  if (qcount * G > kDecRows) {                            // the caller's promise does not hold: said, not computed wrongly
    if (tid == 0) atomicExch(p.status, static_cast<uint32_t>(kErrBadArgument));
    return;
  }
  const int stride = (p.lay.blob_bytes + 127) & ~127;
  uint8_t* stages = smem + static_cast<size_t>(warp) * kDecStages * stride;
  uint64_t* my = bars + warp * kDecStages;
  volatile uint32_t* abort_flag = &abort_word;
  if (tid == 0) abort_word = 0;
  if (lane == 0) {
    for (int s = 0; s < kDecStages; ++s) mbar_init(smem_u32(&my[s]), 1);
    mbar_fence_init();
  }
  __syncthreads();
  const int lo = split * per, hi = min(pages, lo + per), first = lo + warp;
  const int n = first < hi ? (hi - first + kAttnWarps - 1) / kAttnWarps : 0;
  const int* ptab = p.page_table + static_cast<size_t>(req) * p.max_pages;
  auto issue = [&](int i, int page) {
    const int s = i % kDecStages;
    const uint32_t bar = smem_u32(&my[s]);
    mbar_expect_tx(bar, p.lay.blob_bytes);
    bulk_g2s(smem_u32(stages + s * stride), p.cache + (static_cast<size_t>(page) * p.Hkv + kvh) * p.lay.blob_bytes, p.lay.blob_bytes, bar);
  };
  if (lane == 0) {
    int pg[kDecStages];
#pragma unroll
    for (int i = 0; i < kDecStages; ++i) pg[i] = i < n ? ptab[first + i * kAttnWarps] : 0;
#pragma unroll
    for (int i = 0; i < kDecStages; ++i)
      if (i < n) issue(i, pg[i]);
  }
  int limit[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int qp = (2 * t + r) / G;
    limit[r] = qp < qcount ? ctx + qp : 0;
  }
  uint32_t qf[8][2];
  {
    const int qp = g / G, hh = g - qp * G;
    const bool valid = qp < qcount;
    const __nv_bfloat16* q = p.q + (static_cast<size_t>(qstart + qp) * p.Hq + kvh * G + hh) * kD;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      uint2 w = make_uint2(0u, 0u);
      if (valid) w = *reinterpret_cast<const uint2*>(q + j * 16 + t * 4);
      const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w.x)), y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w.y));
      qf[j][0] = pack_f16x2(x.x * p.scale_log2, x.y * p.scale_log2);
      qf[j][1] = pack_f16x2(y.x * p.scale_log2, y.y * p.scale_log2);
    }
  }
  DecState st;
  st.m[0] = st.m[1] = -INFINITY;
  st.l[0] = st.l[1] = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) st.o[i][c] = 0.f;
  int page_next = (lane == 0 && kDecStages < n) ? ptab[first + kDecStages * kAttnWarps] : 0;
  bool ok = true;
  int slot = 0;
  uint32_t phase = 0;
  for (int i = 0; i < n; ++i) {
    ok = __all_sync(0xffffffffu, mbar_wait_t<20>(smem_u32(&my[slot]), phase, abort_flag));
    if (!ok) break;
    const int page_after = (lane == 0 && i + 1 + kDecStages < n) ? ptab[first + (i + 1 + kDecStages) * kAttnWarps] : 0;
    decode_page<KBITS, VBITS>(stages + slot * stride, p.lay, qf, st, (first + i * kAttnWarps) * kPageTokens, limit, total, g, t);
    __syncwarp();
    if (lane == 0 && i + kDecStages < n) issue(i + kDecStages, page_next);
    page_next = page_after;
    if (++slot == kDecStages) { slot = 0; phase ^= 1u; }
  }
  if (!ok && lane == 0) {
    // a wait gave up: copies may still be in flight, they get a bounded time to land
    for (int s = 0; s < kDecStages; ++s) {
      const long long t0 = clock64();
      while (!mbar_try_wait(smem_u32(&my[s]), 0) && !mbar_try_wait(smem_u32(&my[s]), 1) && clock64() - t0 < kWaitBudgetCycles / 8) {
      }
    }
    atomicExch(p.status, static_cast<uint32_t>(kErrBarrierTimeout));
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    st.l[r] += __shfl_xor_sync(0xffffffffu, st.l[r], 4);
    st.l[r] += __shfl_xor_sync(0xffffffffu, st.l[r], 8);
    st.l[r] += __shfl_xor_sync(0xffffffffu, st.l[r], 16);
  }
  __syncthreads();                                        // all warps are done with their stages
  // the warps meet in shared memory: [warp][8 rows][D | max, sum]
  float* mg = reinterpret_cast<float*>(smem);
  float* mine = mg + warp * kDecRows * RS;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int c = 0; c < 2; ++c)
      *reinterpret_cast<float2*>(mine + (2 * t + c) * RS + (i >> 1) * 32 + 4 * g + 2 * (i & 1)) = make_float2(st.o[i][c], st.o[i][2 + c]);
  if (g == 0) {
#pragma unroll
    for (int r = 0; r < 2; ++r) *reinterpret_cast<float2*>(mine + (2 * t + r) * RS + kD) = make_float2(st.m[r], st.l[r]);
  }
  __syncthreads();
  const int row = tid >> 4, cb = (tid & 15) * 8;          // eight channels of a row
  float m = -INFINITY, l = 0.f, o[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) o[c] = 0.f;
#pragma unroll
  for (int w = 0; w < kAttnWarps; ++w) m = fmaxf(m, mg[(w * kDecRows + row) * RS + kD]);
#pragma unroll
  for (int w = 0; w < kAttnWarps; ++w) {
    const float* x = mg + (w * kDecRows + row) * RS;
    const float f = x[kD] == -INFINITY ? 0.f : fast_exp2(x[kD] - m);
    l = fmaf(f, x[kD + 1], l);
#pragma unroll
    for (int c = 0; c < 8; ++c) o[c] = fmaf(f, x[cb + c], o[c]);
  }
  if (used > 1) {
    // parts of the row block: [split][8 rows][D], then [split][8 rows]{max, sum}; the last split to arrive merges them in order
    const size_t idx = static_cast<size_t>(rb) * p.Hkv + kvh;
    float* part = p.partial + idx * p.splits * 16 * RS;
    float* ml = part + static_cast<size_t>(used) * kDecRows * kD;
    float* to = part + (static_cast<size_t>(split) * kDecRows + row) * kD + cb;
    __stcg(reinterpret_cast<float4*>(to), make_float4(o[0], o[1], o[2], o[3]));
    __stcg(reinterpret_cast<float4*>(to + 4), make_float4(o[4], o[5], o[6], o[7]));
    if (cb == 0) __stcg(reinterpret_cast<float2*>(ml + (split * kDecRows + row) * 2), make_float2(m, l));
    __syncthreads();
    if (tid == 0) {
      const uint32_t prev = atom_add_acq_rel_gpu(p.counters + idx, 1u);
      is_last = prev == static_cast<uint32_t>(used) - 1u;
      if (is_last) p.counters[idx] = 0;
    }
    __syncthreads();
    if (!is_last) return;
    float2* sml = reinterpret_cast<float2*>(mg);
    for (int i = tid; i < used * kDecRows; i += kAttnWarps * 32) sml[i] = __ldcg(reinterpret_cast<const float2*>(ml) + i);
    __syncthreads();
    m = -INFINITY; l = 0.f;
    for (int s = 0; s < used; ++s) m = fmaxf(m, sml[s * kDecRows + row].x);
#pragma unroll
    for (int c = 0; c < 8; ++c) o[c] = 0.f;
#pragma unroll 4
    for (int s = 0; s < used; ++s) {
      const float* x = part + (static_cast<size_t>(s) * kDecRows + row) * kD + cb;
      const float4 a = __ldcg(reinterpret_cast<const float4*>(x)), b = __ldcg(reinterpret_cast<const float4*>(x + 4));
      const float2 e = sml[s * kDecRows + row];
      const float f = e.x == -INFINITY ? 0.f : fast_exp2(e.x - m);
      l = fmaf(f, e.y, l);
      o[0] = fmaf(f, a.x, o[0]); o[1] = fmaf(f, a.y, o[1]); o[2] = fmaf(f, a.z, o[2]); o[3] = fmaf(f, a.w, o[3]);
      o[4] = fmaf(f, b.x, o[4]); o[5] = fmaf(f, b.y, o[5]); o[6] = fmaf(f, b.z, o[6]); o[7] = fmaf(f, b.w, o[7]);
    }
  }
  const int qp = row / G, hh = row - qp * G;
  if (qp >= qcount) return;
  const float inv = l > 0.f ? 1.f / l : 0.f;
  *reinterpret_cast<uint4*>(p.out + (static_cast<size_t>(qstart + qp) * p.Hq + kvh * G + hh) * kD + cb) =
      make_uint4(pack_bf16x2(o[0] * inv, o[1] * inv), pack_bf16x2(o[2] * inv, o[3] * inv), pack_bf16x2(o[4] * inv, o[5] * inv), pack_bf16x2(o[6] * inv, o[7] * inv));
}

template <int KB, int VB>
static int launch_decode(const AttnParams& p, int row_blocks, cudaStream_t st) {
  const int stride = (p.lay.blob_bytes + 127) & ~127;
  size_t smem = static_cast<size_t>(kAttnWarps) * kDecStages * stride;
  const size_t merge = static_cast<size_t>(kAttnWarps) * kDecRows * (kD + 2) * 4;      // also holds {max, sum} of 64 splits
  if (smem < merge) smem = merge;
  static bool configured[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -18;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(paged_decode_kernel<KB, VB>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    configured[dev] = true;
  }
  return static_cast<int>(launch(paged_decode_kernel<KB, VB>, dim3(p.Hkv, row_blocks, p.splits), dim3(kAttnWarps * 32), smem, st, p));
}

template <int KB, int VB>
static int launch_attn(const AttnParams& p, dim3 grid, size_t smem, cudaStream_t st) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(paged_attn_kernel<KB, VB>, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
    if (e != cudaSuccess) return static_cast<int>(e);
    configured = true;
  }
  return static_cast<int>(launch(paged_attn_kernel<KB, VB>, grid, dim3(kAttnWarps * 32), smem, st, p));
}

}  // namespace cb

extern "C" {

// fp32 scratch elements needed for `splits` > 1
long long cb_paged_attn_partial_floats(int row_blocks, int Hkv, int splits) {
  return splits > 1 ? static_cast<long long>(row_blocks) * Hkv * splits * 16 * (cb::kD + 2) : 0;
}

int cb_paged_attn(const void* q, void* out, const void* cache, const void* page_table, const void* rb_req,
                  const void* rb_qstart, const void* rb_qcount, const void* rb_ctx, int row_blocks, int Hq, int Hkv,
                  int D, int max_pages, int k_bits, int v_bits, float scale, int splits, void* partial,
                  void* counters, void* status, void* stream) {
  using namespace cb;
  if (row_blocks <= 0) return 0;
  AttnParams p;
  const int bad = make_attn_params(p, q, out, cache, page_table, rb_req, rb_qstart, rb_qcount, rb_ctx, Hq, Hkv, D, max_pages, k_bits, v_bits, scale, splits, partial, counters,
                                   status);
  if (bad) return bad;
  const int stage_stride = (p.lay.blob_bytes + 127) & ~127;
  size_t smem = static_cast<size_t>(kAttnWarps) * kAttnStages * stage_stride + kAttnWarps * kAttnStages * 8;
  const size_t merge = static_cast<size_t>(kAttnWarps) * 16 * (kD + 2) * 4;
  if (smem < merge) smem = merge;
  dim3 grid(Hkv, row_blocks, p.splits);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return with_kv_bits(k_bits, v_bits, [&](auto kb, auto vb) { return launch_attn<decltype(kb)::value, decltype(vb)::value>(p, grid, smem, st); });
}

// Arguments as cb_paged_attn; every row block holds at most eight rows (positions x query heads per key / value head), splits <= 64.
int cb_paged_decode(const void* q, void* out, const void* cache, const void* page_table, const void* rb_req, const void* rb_qstart, const void* rb_qcount,
                    const void* rb_ctx, int row_blocks, int Hq, int Hkv, int D, int max_pages, int k_bits, int v_bits, float scale, int splits, void* partial,
                    void* counters, void* status, void* stream) {
  using namespace cb;
  if (row_blocks <= 0) return 0;
  AttnParams p;
  const int bad = make_attn_params(p, q, out, cache, page_table, rb_req, rb_qstart, rb_qcount, rb_ctx, Hq, Hkv, D, max_pages, k_bits, v_bits, scale, splits, partial, counters,
                                   status);
  if (bad) return bad;
  if (p.G > kDecRows || p.splits > 64) return -14;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return with_kv_bits(k_bits, v_bits, [&](auto kb, auto vb) { return launch_decode<decltype(kb)::value, decltype(vb)::value>(p, row_blocks, st); });
}

}  // extern "C"
