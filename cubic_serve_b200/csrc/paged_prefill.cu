// Paged GQA attention over the quantized KV cache for portions of prompts, on the tensor cores of tcgen05 (page layout: kv_layout.cuh;
// row blocks: paged_attn.cu).
//
// What bounds it: shared memory, then the MMAs.  An item is sixteen consecutive row blocks -- 256 rows, two tiles of one tcgen05 MMA each --
// of a key / value head; a CTA takes items one after the other and converts a step of 64 tokens once for both tiles.
// A cached value is a code of at most 8 bits times an fp32 scale, one per token and 32 channels.  The conversion writes it as a sum of two f16
// (hi + lo), so that a step's scores and its output are one chain of MMAs each.  Scales inside the softmax would take
// four score tiles and four copies of the probabilities, one per channel group (what this kernel did before: 256 multiply-adds, 256 multiplications
// and 128 packings a row and step instead of 64, 0 and 32; 5800 cycles a step of 128 rows).
// Powers of two keep hi and lo in the range of f16: one a step for K, undone in the softmax' multiply-add; one for V that grows with the
// largest scale of a run of steps, falls back towards one, and is undone with the output (a row keeps that of its own request's steps).
// What is 2^-k of the largest scale keeps 22 bits up to k = 6 to 8, then 28 - k; probabilities have 11.  A product's error stays below 2^-18 (V) and 2^-20 (K) as long
// as the largest scale is below 16 (values of 2000), as far as f16 products of probabilities and scales would go.  Beyond that the rows
// that see such tokens are computed once more, in fp32 from the pages (pf_row); what values with scales that are not finite contribute is added (pf_odd).
// MMAs of a step take 640 + 512 cycles a tile (measured in a loop of their own); with their operands, raw pages and the conversion's stores shared memory
// moves about 280 KB a step: 4000 cycles a step of 256 rows where 2 x 5800 were spent.  General kernel -> before -> now, one B200, cold L2, 32 heads
// over 8, 8 bits: 8 x 1024 tokens 702 -> 520 -> 213 us, 4 x 256 behind 2048 276 -> 233 -> 100, one prompt of 8192 3734 -> 2775 -> 1165, 40 x 20 behind 300
// 63 -> 103 -> 56, 8 x 64 26 -> 15 -> 17; 32 over 4, 4 / 8 bits, 2 x 2048 571 -> 421 -> 192; 64 over 4, 6 bits, 3 x 500 190 -> 131 -> 79.
//
// Roles: warps 0-7 own a row a thread (softmax needs no exchange: tensor-memory lane = row); warps 8-11 convert raw pages of K to the swizzled operand
// (hi and lo, [token][channel]), warps 12-15 those of V; warps 16 and 18 issue the MMAs; warp 17 lists the items' requests and copies their
// pages three steps ahead.  Tensor memory of a tile: scores, probabilities (the A operand of their product), output and the first half of Q's
// channels; the other half of Q is in shared memory, where an MMA of 64 columns takes 48 cycles instead of 32.
// The scores of step i + 1 are computed while the softmax of step i runs.  Row blocks of several requests may meet in an item: it walks
// their steps one request after the other, rows of another request taking part with probability zero.  The output accumulator stays
// in tensor memory and is rescaled only when a row's maximum has grown by more than a factor of four (2 in the log2 domain): until
// then probabilities relative to the older maximum are at most 4.
// Every wait is bounded; on a timeout the roles leave, the status word is set and tensor memory is freed.
#include "paged_attn.cuh"
#include <limits.h>

namespace cb {

static constexpr int kPfTiles = 2;
static constexpr int kPfRows = 128;                      // of a tile
static constexpr int kPfBlocks = kPfTiles * kPfRows / 16;
static constexpr int kPfPages = 4;                       // pages of a step
static constexpr int kPfTok = kPfPages * kPageTokens;    // 64
static constexpr int kPfThreads = 640;
// registers a thread: at launch, and of the softmax', the conversion's and the other warps after they have shared them out anew
static constexpr int kPfRegs = 96, kPfRegsSoftmax = 136, kPfRegsConvert = 72, kPfRegsOther = 64;
static_assert(2 * kPfRegsSoftmax + 2 * kPfRegsConvert + kPfRegsOther <= 5 * kPfRegs, "five warpgroups");
static constexpr int kPfLists = 4;
static constexpr int kPfRaw = 3;                         // steps of raw pages
// Steps whose powers of two are kept.  Nothing else orders the note of step g + kPfNotes behind the reads of step g's: a tile that sees nothing of the
// steps behind g holds back neither their scores nor k_free.  It holds back v_free of step g alone, whose product waits for the tile's probabilities,
// and that reaches the conversion of K by way of the raw pages: note of K (s) <- raw_full (s) <- raw_free (s - kPfRaw) <- V of s - kPfRaw
// converted <- v_free (s - kPfRaw - 2) <- p_full of every tile that takes part in it.
static constexpr int kPfNotes = kPfRaw + 2;
static constexpr int kPfSorted = 512;                    // groups of row blocks that are dealt by their length
static constexpr float kPfGrowth = 2.f;
static constexpr int kPfLarge = 3;                       // exponent of scales from which on small ones beside them are looked at
static constexpr int kPfVFall = 80;                      // most by which v_exp falls in a run: outputs in its units stay below 2^(37 + 80)
// tensor memory, columns of a tile: scores, probabilities (two f16 a column), channels 0..63 of Q (likewise), output
static constexpr uint32_t kPfTmemCols = 512, kPfTmemTile = 256, kPfTmemP = 64, kPfTmemQ = 96, kPfTmemO = 128;
static constexpr int kPfHalf = kPfTok * 128;             // bytes of 64 channels of a step

struct PfRun {
  int first, end, req, total, pages, steps;              // row blocks [first, end) of the item, tokens that they see, ...
  int tile_steps[kPfTiles];                              // ... steps that the rows of each tile see something of
};
struct PfList {
  int kvh, runs, steps, tiles;                           // kvh < 0: no more items; tiles: bit mask of those with steps
  int qstart[kPfBlocks], qcount[kPfBlocks], ctx[kPfBlocks];
  PfRun run[kPfBlocks];
};
struct __align__(1024) PfSmem {
  uint8_t q[kPfTiles][kPfRows * 128];                    // f16, channels 64..127: [row][128 B], 16-byte chunk ^ (row & 7)
  uint8_t k[2][2][2 * kPfHalf];                          // f16 [stage][hi, lo][64-channel half][token][128 B]
  uint8_t v[2][2][2 * kPfHalf];                          // likewise
  float k_mul[kPfNotes];                                 // scores are this times what the MMAs give
  int v_exp[kPfNotes];                                   // output is 2^v_exp times ...
  // tokens of a run: rows that see more are computed once more [0], have values with scales that are not finite added [1]; the least of all
  int redo[kPfLists][2][kPfBlocks], redo_least[kPfLists];
  uint64_t raw_full[kPfRaw], raw_free[kPfRaw], k_full[2], k_free[2], v_full[2], v_free[2], k_note[kPfNotes], v_note[kPfNotes];
  uint64_t list_full[kPfLists], list_free[kPfLists], q_full[kPfTiles], s_full[kPfTiles], s_free[kPfTiles], p_full[kPfTiles], pv_done[kPfTiles];
  PfList list[kPfLists];
  uint16_t order[kPfSorted];                             // groups of row blocks, those that see most first
  uint32_t tmem, abort_word;
};

// Shared-memory descriptor of an operand whose rows of 128 bytes run along N (or M), 128-byte swizzle: 8 rows of K are 1024 bytes, blocks of 64 columns
// `block` bytes apart.
__device__ __forceinline__ uint64_t umma_desc_sw128_n(uint32_t smem_addr, uint32_t block) {
  return (umma_desc_sw128(smem_addr) & ~(static_cast<uint64_t>(0x3FFF) << 16)) | static_cast<uint64_t>(block >> 4) << 16;
}
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((min(max(e, -126), 127) + 127) << 23); }

// Where a role stands in an item's list of steps: runs one after the other.
struct PfWalk {
  int run = 0, step = 0;
  __device__ __forceinline__ void advance(const PfList& l) {
    if (++step == l.run[run].steps) { step = 0; ++run; }
  }
};

__device__ __forceinline__ uint4 conv8(uint2 w, uint32_t bias) {        // eight codes in order -> eight f16
  return make_uint4(u8x2_to_f16x2(w.x, 0x5140u, bias), u8x2_to_f16x2(w.x, 0x5342u, bias), u8x2_to_f16x2(w.y, 0x5140u, bias), u8x2_to_f16x2(w.y, 0x5342u, bias));
}

// Two codes times their scales sh + sl: the rounded product with sh, and what it left over with the product with sl.  The residual is exact (a code
// has 8 bits, sh 11), so hi + lo is off by the rounding of sl and of lo: 2^-22 of the value.
__device__ __forceinline__ void pf_scaled(uint32_t code, uint32_t sh, uint32_t sl, uint32_t& hi, uint32_t& lo) {
  uint32_t n, r;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(hi) : "r"(code), "r"(sh));
  asm("neg.f16x2 %0, %1;" : "=r"(n) : "r"(hi));
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(code), "r"(sh), "r"(n));
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(lo) : "r"(code), "r"(sl), "r"(r));
}
__device__ __forceinline__ void pf_scaled8(const uint4& c, uint32_t sh, uint32_t sl, uint4& hi, uint4& lo) {
  pf_scaled(c.x, sh, sl, hi.x, lo.x);
  pf_scaled(c.y, sh, sl, hi.y, lo.y);
  pf_scaled(c.z, sh, sl, hi.z, lo.z);
  pf_scaled(c.w, sh, sl, hi.w, lo.w);
}
// an fp32 scale as a pair of f16, each twice
__device__ __forceinline__ void pf_split(float s, uint32_t& sh, uint32_t& sl) {
  sh = pack_f16x2(s, s);
  const float r = s - __low2float(*reinterpret_cast<const __half2*>(&sh));
  sl = pack_f16x2(r, r);
}

// The largest magnitude of a token's scales, as bits; FINITE: of those that are
template <bool FINITE>
__device__ __forceinline__ uint32_t pf_most(const float4& s) {
  auto magnitude = [](float x) {
    const uint32_t b = __float_as_uint(x) & 0x7FFFFFFFu;
    return !FINITE || b < 0x7F800000u ? b : 0u;
  };
  return max(max(magnitude(s.x), magnitude(s.y)), max(magnitude(s.z), magnitude(s.w)));
}
__device__ __forceinline__ int pf_exponent(uint32_t magnitude) { return max(static_cast<int>(magnitude >> 23) - 127, -100); }

// The scales of a step's tokens `lane` and `lane` + 32, zeros from `visible` on
__device__ __forceinline__ void pf_scales(const uint8_t* scales, int stride, int visible, int lane, float4 (&of)[2]) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int tok = lane + 32 * h;
    of[h] = *reinterpret_cast<const float4*>(scales + (tok >> 4) * stride + (tok & 15) * 16);
    if (tok >= visible) of[h] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// One step's codes into operands: all of a thread's loads, then its arithmetic (few warps hide nothing).
// What K holds of tokens that no row sees is masked with their scores.
template <int KBITS>
__device__ __forceinline__ void pf_convert_k(uint8_t (&k)[2][2 * kPfHalf], const uint8_t* raw, int stride, const KvLayout& lay, float mul, int tid) {
  constexpr uint32_t kb = KBITS == 8 ? 0x64806480u : KBITS == 6 ? 0x64206420u : 0x64086408u;
  // an item is 16 channels (8 bit) or 32 (4 and 6 bit) of a token
  constexpr int kItems = KBITS == 8 ? kPageTokens * 8 : kPageTokens * 4, kMine = kPfPages * kItems / 128;
  uint4 x[kMine], xh[kMine];
  float s[kMine];
#pragma unroll
  for (int j = 0; j < kMine; ++j) {
    const int i = tid + j * 128, r = i % kItems, tok = r & 15, blk = r >> 4;
    const uint8_t* src = raw + i / kItems * stride;
    x[j] = *reinterpret_cast<const uint4*>(src + blk * 256 + tok * 16);
    if constexpr (KBITS == 6) xh[j] = *reinterpret_cast<const uint4*>(src + kPageTokens * kD / 2 + blk * 128 + (tok & 7) * 16);
    s[j] = *reinterpret_cast<const float*>(src + lay.k_scale_off + tok * 16 + (KBITS == 8 ? blk >> 1 : blk) * 4);
  }
#pragma unroll
  for (int j = 0; j < kMine; ++j) {
    const int i = tid + j * 128, r = i % kItems, tok = r & 15, blk = r >> 4, sw = tok & 7;
    const int at = (KBITS == 8 ? blk >> 2 : blk >> 1) * kPfHalf + (i / kItems * 16 + tok) * 128;
    uint4* row_hi = reinterpret_cast<uint4*>(k[0] + at);
    uint4* row_lo = reinterpret_cast<uint4*>(k[1] + at);
    const int c = KBITS == 8 ? (blk & 3) * 2 : (blk & 1) * 4;
    uint32_t sh, sl;
    pf_split(s[j] * mul, sh, sl);
    auto put = [&](int chunk, uint2 codes) {
      uint4 hi, lo;
      pf_scaled8(conv8(codes, kb), sh, sl, hi, lo);
      row_hi[chunk ^ sw] = hi;
      row_lo[chunk ^ sw] = lo;
    };
    if constexpr (KBITS == 8) {
      put(c, make_uint2(x[j].x, x[j].y));
      put(c + 1, make_uint2(x[j].z, x[j].w));
    } else {
      const uint32_t n[4] = {x[j].x, x[j].y, x[j].z, x[j].w};
      uint32_t lo[4], hi[4];
      const uint32_t hw[4] = {xh[j].x, xh[j].y, xh[j].z, xh[j].w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        lo[q] = n[q] & 0x0F0F0F0Fu;
        hi[q] = (n[q] >> 4) & 0x0F0F0F0Fu;
        if constexpr (KBITS == 6) {
          lo[q] |= (tok < 8 ? hw[q] : hw[q] << 4) & 0x30303030u;
          hi[q] |= (tok < 8 ? hw[q] >> 2 : hw[q] << 2) & 0x30303030u;
        }
      }
      put(c, make_uint2(lo[0], lo[1]));
      put(c + 1, make_uint2(lo[2], lo[3]));
      put(c + 2, make_uint2(hi[0], hi[1]));
      put(c + 3, make_uint2(hi[2], hi[3]));
    }
  }
}
// V from `visible` on becomes zeros: those slots may hold anything, and a probability of zero has to stay zero.  Likewise where a scale is not finite.
template <int VBITS>
__device__ __forceinline__ void pf_convert_v(uint8_t (&v)[2][2 * kPfHalf], const uint8_t* raw, int stride, const KvLayout& lay, int visible, float mul, int tid) {
  constexpr uint32_t vb = VBITS == 8 ? 0x64806480u : VBITS == 6 ? 0x64206420u : 0x64086408u;
  // an item is 8 channels of a token pair of a page
  const int c = tid & 15, pair = tid >> 4, at = (2 * c) ^ ((pair & 3) << 2);
  uint4 x[kPfPages];                                     // 8 bit: the codes; else low nibbles, high bits
  float s[kPfPages][2];
#pragma unroll
  for (int j = 0; j < kPfPages; ++j) {
    const uint8_t* page = raw + j * stride;
    const uint8_t* src = page + lay.v_code_off;
    if constexpr (VBITS == 8) {
      x[j] = *reinterpret_cast<const uint4*>(src + pair * 256 + at * 8);
    } else {
      const uint2 n = *reinterpret_cast<const uint2*>(src + pair * 128 + at * 4);
      uint2 hw = make_uint2(0u, 0u);
      if constexpr (VBITS == 6) hw = *reinterpret_cast<const uint2*>(src + kPageTokens * kD / 2 + (pair & 3) * 128 + at * 4);
      x[j] = make_uint4(n.x, n.y, hw.x, hw.y);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) s[j][h] = *reinterpret_cast<const float*>(page + lay.v_scale_off + (2 * pair + h) * 16 + (c >> 2) * 4);
  }
#pragma unroll
  for (int j = 0; j < kPfPages; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int tok = (j * 8 + pair) * 2 + h;
      uint4 codes;
      if constexpr (VBITS == 8) {
        const uint32_t sel = h ? 0x5341u : 0x5240u;
        codes = make_uint4(u8x2_to_f16x2(x[j].x, sel, vb), u8x2_to_f16x2(x[j].y, sel, vb), u8x2_to_f16x2(x[j].z, sel, vb), u8x2_to_f16x2(x[j].w, sel, vb));
      } else {
        uint2 n = h ? make_uint2((x[j].x >> 4) & 0x0F0F0F0Fu, (x[j].y >> 4) & 0x0F0F0F0Fu) : make_uint2(x[j].x & 0x0F0F0F0Fu, x[j].y & 0x0F0F0F0Fu);
        if constexpr (VBITS == 6) {
          auto high = [&](uint32_t w) { return (pair < 4 ? (h ? w >> 2 : w) : (h ? w << 2 : w << 4)) & 0x30303030u; };
          n.x |= high(x[j].z);
          n.y |= high(x[j].w);
        }
        codes = conv8(n, vb);
      }
      float f = s[j][h] * mul;
      if (tok >= visible || !(fabsf(f) < INFINITY)) f = 0.f;
      uint32_t sh, sl;
      uint4 hi, lo;
      pf_split(f, sh, sl);
      pf_scaled8(codes, sh, sl, hi, lo);
      const int to = (c >> 3) * kPfHalf + tok * 128 + (((c & 7) ^ (tok & 7)) << 4);
      *reinterpret_cast<uint4*>(v[0] + to) = hi;
      *reinterpret_cast<uint4*>(v[1] + to) = lo;
    }
}

// Codes of the channels 4 lane .. 4 lane + 3 of a token of a page, a byte each, with their bias
template <int BITS>
__device__ __forceinline__ uint32_t pf_codes_k(const uint8_t* k, int tok, int lane) {
  if constexpr (BITS == 8) return *reinterpret_cast<const uint32_t*>(k + (lane >> 2) * 256 + tok * 16 + (lane & 3) * 4);
  const int blk = lane >> 3, high = lane >> 2 & 1, t = lane & 3;
  uint32_t x = *reinterpret_cast<const uint32_t*>(k + blk * 256 + tok * 16 + t * 4) >> (4 * high) & 0x0F0F0F0Fu;
  if constexpr (BITS == 6) {
    const uint32_t w = *reinterpret_cast<const uint32_t*>(k + kPageTokens * kD / 2 + blk * 128 + (tok & 7) * 16 + t * 4);
    x |= (tok < 8 ? (high ? w >> 2 : w) : (high ? w << 2 : w << 4)) & 0x30303030u;
  }
  return x;
}
template <int BITS>
__device__ __forceinline__ uint32_t pf_codes_v(const uint8_t* v, int tok, int lane) {
  const int pair = tok >> 1, odd = tok & 1, at = lane ^ ((pair & 3) << 2);
  if constexpr (BITS == 8) {
    const uint2 w = *reinterpret_cast<const uint2*>(v + pair * 256 + at * 8);
    return prmt(w.x, w.y, odd ? 0x7531u : 0x6420u);
  }
  uint32_t x = *reinterpret_cast<const uint32_t*>(v + pair * 128 + at * 4) >> (4 * odd) & 0x0F0F0F0Fu;
  if constexpr (BITS == 6) {
    const uint32_t w = *reinterpret_cast<const uint32_t*>(v + kPageTokens * kD / 2 + (pair & 3) * 128 + at * 4);
    x |= (pair < 4 ? (odd ? w >> 2 : w) : (odd ? w << 2 : w << 4)) & 0x30303030u;
  }
  return x;
}

// A row in fp32, by a warp whose lanes have four channels each: `limit` tokens of request `req`, the query at `q` (result likewise in `out`).
// A hundred times as long as the MMAs (8 x 1024 tokens 23 ms): for caches whose scales are as large and as far apart as no model's.
template <int KBITS, int VBITS>
__device__ __forceinline__ void pf_row(const AttnParams& p, int req, int kvh, int limit, const __nv_bfloat16* q, __nv_bfloat16* out, int lane) {
  constexpr int kTok = 4;                                // tokens at a time, of one page
  constexpr float kBias = 1 << (KBITS - 1), vBias = 1 << (VBITS - 1);
  const uint2 qw = reinterpret_cast<const uint2*>(q)[lane];
  const float2 q01 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&qw.x)), q23 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&qw.y));
  const float qf[4] = {q01.x * p.scale_log2, q01.y * p.scale_log2, q23.x * p.scale_log2, q23.y * p.scale_log2};
  float m = -INFINITY, sum = 0.f, o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
  for (int t0 = 0; t0 < limit; t0 += kTok) {
    const int page = p.page_table[static_cast<size_t>(req) * p.max_pages + t0 / kPageTokens], tok0 = t0 % kPageTokens;
    const uint8_t* blob = p.cache + (static_cast<size_t>(page) * p.Hkv + kvh) * p.lay.blob_bytes;
    uint32_t kc[kTok], vc[kTok];
    float ks[kTok], vs[kTok], z[kTok];
#pragma unroll
    for (int j = 0; j < kTok; ++j) {
      kc[j] = pf_codes_k<KBITS>(blob, tok0 + j, lane);
      vc[j] = pf_codes_v<VBITS>(blob + p.lay.v_code_off, tok0 + j, lane);
      ks[j] = *reinterpret_cast<const float*>(blob + p.lay.k_scale_off + (tok0 + j) * 16 + (lane >> 3) * 4);
      vs[j] = *reinterpret_cast<const float*>(blob + p.lay.v_scale_off + (tok0 + j) * 16 + (lane >> 3) * 4);
    }
    float top = -INFINITY;
#pragma unroll
    for (int j = 0; j < kTok; ++j) {
      float d = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) d = fmaf(qf[c], static_cast<float>(kc[j] >> (8 * c) & 255u) - kBias, d);
      d *= ks[j];
#pragma unroll
      for (int o2 = 16; o2 > 0; o2 >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o2);
      z[j] = t0 + j < limit ? d : -INFINITY;
      top = fmaxf(top, z[j]);
    }
    if (top > m) {
      const float alpha = fast_exp2(m - top);
      m = top;
      sum *= alpha;
#pragma unroll
      for (int c = 0; c < 4; ++c) o[c] *= alpha;
    }
    const float use = m == -INFINITY ? 0.f : m;
#pragma unroll
    for (int j = 0; j < kTok; ++j) {
      if (t0 + j >= limit) break;
      const float pr = fast_exp2(z[j] - use);
      sum += pr;
#pragma unroll
      for (int c = 0; c < 4; ++c) o[c] = fmaf(pr, (static_cast<float>(vc[j] >> (8 * c) & 255u) - vBias) * vs[j], o[c]);
    }
  }
  const float inv = sum > 0.f ? 1.f / sum : sum == 0.f ? 0.f : sum;
  reinterpret_cast<uint2*>(out)[lane] = make_uint2(pack_bf16x2(o[0] * inv, o[1] * inv), pack_bf16x2(o[2] * inv, o[3] * inv));
}

// Adds to the rows of a warp (a lane has one: its request, how many tokens it sees, where its query and result are, its maximum and the reciprocal of its
// sum) what tokens from `from` on whose V scales are not finite contribute; the operands have left them out.  Rows of a request look for them together.
template <int KBITS, int VBITS>
__device__ __forceinline__ void pf_odd(const AttnParams& p, int kvh, int req, int from, int limit, long long at, float m, float inv, int lane) {
  constexpr float kBias = 1 << (KBITS - 1), vBias = 1 << (VBITS - 1);
  constexpr int kScan = 4;
#pragma unroll 1
  for (uint32_t left = __ballot_sync(0xffffffffu, limit > from); left;) {
    const int rq = __shfl_sync(0xffffffffu, req, __ffs(left) - 1);
    const bool mine = (left >> lane & 1) != 0 && req == rq;
    uint32_t rows = __ballot_sync(0xffffffffu, mine);
    left &= ~rows;
    const int most = __reduce_max_sync(0xffffffffu, mine ? limit : 0), least = __reduce_min_sync(0xffffffffu, mine ? from : INT_MAX);
    auto blob_of = [&](int tok) {
      return p.cache + (static_cast<size_t>(p.page_table[static_cast<size_t>(rq) * p.max_pages + tok / kPageTokens]) * p.Hkv + kvh) * p.lay.blob_bytes;
    };
    auto next = [&](int t) {                               // the first of them from t on, or `most`
#pragma unroll 1
      for (int t0 = t & ~31; t0 < most; t0 += 32 * kScan) {
        bool odd[kScan];                                   // the lane's token of every 32
#pragma unroll
        for (int j = 0; j < kScan; ++j) {
          const int tok = t0 + 32 * j + lane;
          float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
          if (tok >= t && tok < most) f = *reinterpret_cast<const float4*>(blob_of(tok) + p.lay.v_scale_off + tok % kPageTokens * 16);
          odd[j] = !(fabsf(f.x) < INFINITY && fabsf(f.y) < INFINITY && fabsf(f.z) < INFINITY && fabsf(f.w) < INFINITY);
        }
#pragma unroll
        for (int j = 0; j < kScan; ++j) {
          const uint32_t toks = __ballot_sync(0xffffffffu, odd[j]);
          if (toks) return t0 + 32 * j + __ffs(toks) - 1;
        }
      }
      return most;
    };
#pragma unroll 1
    for (int t = next(least); t < most && rows != 0; t = next(t + 1)) {
      const int tok = t % kPageTokens;
      const uint8_t* blob = blob_of(t);
      const uint32_t kc = pf_codes_k<KBITS>(blob, tok, lane), vc = pf_codes_v<VBITS>(blob + p.lay.v_code_off, tok, lane);
      const float ks = *reinterpret_cast<const float*>(blob + p.lay.k_scale_off + tok * 16 + (lane >> 3) * 4) * p.scale_log2;
      const float vs = *reinterpret_cast<const float*>(blob + p.lay.v_scale_off + tok * 16 + (lane >> 3) * 4);
      const bool add = !(fabsf(vs) < INFINITY);
#pragma unroll 1
      for (uint32_t see = rows & __ballot_sync(0xffffffffu, limit > t); see; see &= see - 1) {
        const int of = __ffs(see) - 1;
        const long long to = __shfl_sync(0xffffffffu, at, of);
        const float top = __shfl_sync(0xffffffffu, m, of), scale = __shfl_sync(0xffffffffu, inv, of);
        const uint2 qw = reinterpret_cast<const uint2*>(p.q + to)[lane];
        uint2* out = reinterpret_cast<uint2*>(p.out + to) + lane;
        const uint2 w = *out;
        auto two = [](uint32_t x) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x)); };
        const float2 q01 = two(qw.x), q23 = two(qw.y), o01 = two(w.x), o23 = two(w.y);
        const float qf[4] = {q01.x, q01.y, q23.x, q23.y};
        float o[4] = {o01.x, o01.y, o23.x, o23.y}, z = 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c) z = fmaf(qf[c], static_cast<float>(kc >> (8 * c) & 255u) - kBias, z);
        z *= ks;
#pragma unroll
        for (int o2 = 16; o2 > 0; o2 >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o2);
        if (add) {
          const float pr = fast_exp2(z - (top == -INFINITY ? 0.f : top)) * scale;
#pragma unroll
          for (int c = 0; c < 4; ++c) o[c] = fmaf(pr, (static_cast<float>(vc >> (8 * c) & 255u) - vBias) * vs, o[c]);
          *out = make_uint2(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]));
        }
        // (NaN stays: behind it there is nothing to add)
        if (__all_sync(0xffffffffu, o[0] != o[0] && o[1] != o[1] && o[2] != o[2] && o[3] != o[3])) rows &= ~(1u << of);
      }
    }
  }
}

template <int KBITS, int VBITS>
__global__ void __launch_bounds__(kPfThreads, 1)
paged_prefill_kernel(const AttnParams p, const int row_blocks) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  PfSmem& sm = *reinterpret_cast<PfSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* raw = reinterpret_cast<uint8_t*>(&sm + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int stride = (p.lay.blob_bytes + 127) & ~127;
  const int groups = (row_blocks + kPfBlocks - 1) / kPfBlocks, ctas = gridDim.x;
  const long long items = static_cast<long long>(groups) * p.Hkv;
  const bool sorted = items > ctas && groups <= kPfSorted;
  volatile uint32_t* abort_flag = &sm.abort_word;
  if (tid == 0) {
    for (int b = 0; b < kPfRaw; ++b) {
      mbar_init(smem_u32(&sm.raw_full[b]), 1);
      mbar_init(smem_u32(&sm.raw_free[b]), 8);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&sm.k_full[b]), 4);
      mbar_init(smem_u32(&sm.k_free[b]), 1);
      mbar_init(smem_u32(&sm.v_full[b]), 4);
      mbar_init(smem_u32(&sm.v_free[b]), 1);
    }
    for (int b = 0; b < kPfNotes; ++b) {
      mbar_init(smem_u32(&sm.k_note[b]), 1);
      mbar_init(smem_u32(&sm.v_note[b]), 1);
    }
    for (int b = 0; b < kPfLists; ++b) {
      mbar_init(smem_u32(&sm.list_full[b]), 1);
      mbar_init(smem_u32(&sm.list_free[b]), 18);         // all warps but 17 and 19
    }
    for (int t = 0; t < kPfTiles; ++t) {
      mbar_init(smem_u32(&sm.q_full[t]), 4);
      mbar_init(smem_u32(&sm.s_full[t]), 1);
      mbar_init(smem_u32(&sm.s_free[t]), 4);
      mbar_init(smem_u32(&sm.p_full[t]), 4);
      mbar_init(smem_u32(&sm.pv_done[t]), 1);
    }
    sm.abort_word = 0;
    mbar_fence_init();
  }
  if (warp == 16) {
    tmem_alloc(smem_u32(&sm.tmem), kPfTmemCols);
    tmem_relinquish();
  }
  pdl_wait();
  pdl_launch_dependents();
  if (sorted) {
    // With more items than CTAs the groups are dealt by what their last block sees, to and fro: every CTA finds the same order for itself
    uint16_t* seen = reinterpret_cast<uint16_t*>(sm.v[0][0]);
    for (int g = tid; g < groups; g += kPfThreads) {
      const int last = min(g * kPfBlocks + kPfBlocks, row_blocks) - 1;
      seen[g] = static_cast<uint16_t>(min((max(p.rb_ctx[last] + p.rb_qcount[last], 0) + kPfTok - 2) / kPfTok, 65535));
    }
    __syncthreads();
    for (int g = tid; g < groups; g += kPfThreads) {
      const int mine = seen[g];
      int rank = 0;
      for (int o = 0; o < groups; ++o) rank += seen[o] > mine || (seen[o] == mine && o > g);
      sm.order[rank] = static_cast<uint16_t>(g);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem;
  bool ok = true;

  if (warp >= 16) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kPfRegsOther));
    if (warp == 17) {
      // ------------------------------------------------------- items and pages
      int gs = 0;
      auto publish = [&](int n) {                        // the CTA's n-th item; false: there is none
        const long long at = static_cast<long long>(n) * ctas + (n & 1 ? ctas - 1 - static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x));
        PfList& l = sm.list[n % kPfLists];
        if (ok && n >= kPfLists) ok = mbar_wait_park(smem_u32(&sm.list_free[n % kPfLists]), (n / kPfLists - 1) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) return false;
        sm.redo[n % kPfLists][lane / kPfBlocks][lane % kPfBlocks] = INT_MAX;
        if (lane == 0) sm.redo_least[n % kPfLists] = INT_MAX;
        if (at >= items) {                               // no item in this round: there is no further round
          if (lane == 0) l.kvh = -1;
        } else {
          const int rank = static_cast<int>(at / p.Hkv);
          const int rb0 = (sorted ? sm.order[rank] : groups - 1 - rank) * kPfBlocks;      // the blocks that see most first
          int cnt = 0, req = -1, sees = 0, ctx = 0;
          if (lane < kPfBlocks) {
            if (rb0 + lane < row_blocks) {
              cnt = max(p.rb_qcount[rb0 + lane], 0);
              req = p.rb_req[rb0 + lane];
              ctx = p.rb_ctx[rb0 + lane];
              l.qstart[lane] = p.rb_qstart[rb0 + lane];
            }
            l.qcount[lane] = cnt;
            l.ctx[lane] = ctx;
            if (cnt > 0) sees = max(ctx + cnt - 1, 0);
          }
          const int req_before = __shfl_up_sync(0xffffffffu, req, 1), cnt_before = __shfl_up_sync(0xffffffffu, cnt, 1);
          const bool on = lane > 0 && cnt > 0 && cnt_before > 0 && req_before == req;     // goes on with the run of the block before it
          uint32_t starts = __ballot_sync(0xffffffffu, cnt > 0 && !on);
          const uint32_t goes_on = __ballot_sync(0xffffffffu, on);
          int runs = 0, steps = 0, tiles = 0;
          while (starts) {
            const int s = __ffs(starts) - 1;
            starts &= starts - 1;
            const int end = s + __ffs(~(goes_on >> (s + 1)));
            const bool in = lane >= s && lane < end;
            PfRun r;
            r.first = s;
            r.end = end;
            r.req = __shfl_sync(0xffffffffu, req, s);
            r.total = 0;
#pragma unroll
            for (int t = 0; t < kPfTiles; ++t) {
              const int most = static_cast<int>(__reduce_max_sync(0xffffffffu, in && lane / 8 == t ? static_cast<uint32_t>(sees) : 0u));
              r.tile_steps[t] = (most + kPfTok - 1) / kPfTok;
              if (most > 0) tiles |= 1 << t;
              r.total = max(r.total, most);
            }
            r.pages = (r.total + kPageTokens - 1) / kPageTokens;
            r.steps = (r.pages + kPfPages - 1) / kPfPages;
            if (r.steps > 0) {
              if (lane == 0) l.run[runs] = r;
              ++runs;
              steps += r.steps;
            }
          }
          if (lane == 0) {
            l.kvh = static_cast<int>(at % p.Hkv);
            l.runs = runs;
            l.steps = steps;
            l.tiles = tiles;
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm.list_full[n % kPfLists]));
        return at < items;
      };
      bool more = publish(0);
      for (int it = 0; more && ok; ++it) {
        const PfList& l = sm.list[it % kPfLists];
        const int steps = l.steps, kvh = l.kvh;
        bool next = false;
        PfWalk w;
        for (int i = 0; i < steps; ++i, ++gs) {
          const int b = gs % kPfRaw;
          if (ok && gs >= kPfRaw) ok = mbar_wait_park(smem_u32(&sm.raw_free[b]), (gs / kPfRaw - 1) & 1, abort_flag);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          const PfRun& r = l.run[w.run];
          const int n = min(kPfPages, r.pages - w.step * kPfPages);
          if (lane == 0) mbar_expect_tx(smem_u32(&sm.raw_full[b]), n * p.lay.blob_bytes);
          __syncwarp();
          if (lane < n) {
            const int page = p.page_table[static_cast<size_t>(r.req) * p.max_pages + w.step * kPfPages + lane];
            bulk_g2s(smem_u32(raw + (b * kPfPages + lane) * stride), p.cache + (static_cast<size_t>(page) * p.Hkv + kvh) * p.lay.blob_bytes, p.lay.blob_bytes,
                     smem_u32(&sm.raw_full[b]));
          }
          w.advance(l);
          if (i == min(1, steps - 1)) next = publish(it + 1);
        }
        if (steps == 0) next = publish(it + 1);
        more = next;
      }
      if (*abort_flag) {                                 // copies in flight land (for a bounded time) before the CTA goes
        const long long t0 = clock64();
        for (int i = max(0, gs - kPfRaw); i < gs; ++i)
          while (!mbar_try_wait(smem_u32(&sm.raw_full[i % kPfRaw]), (i / kPfRaw) & 1) && clock64() - t0 < kWaitBudgetCycles / 8) {
          }
      }
    } else if (warp != 19) {
      // ---------------------------------------------------------------- MMAs
      // Warp 16 issues those of the scores, warp 18 those of the output: what one waits for does not hold up the other
      const bool leader = elect_one(), is_s = warp == 16;
      const uint32_t idesc_s = umma_idesc(kPfRows, kPfTok, 0u, 0u), idesc_o = umma_idesc(kPfRows, kD, 0u, 0u) | 1u << 16;      // V: channels are contiguous
      const uint64_t dq = umma_desc_sw128(smem_u32(sm.q[0])), dk = umma_desc_sw128(smem_u32(sm.k[0][0])), dv = umma_desc_sw128_n(smem_u32(sm.v[0][0]), kPfHalf);
      int gs = 0;                                        // steps of earlier items
      int n[kPfTiles] = {0, 0};                          // steps per tile
      uint32_t q_phase = 0;                              // bit = tile
      for (int it = 0;; ++it) {
        const PfList& l = sm.list[it % kPfLists];
        if (ok) ok = mbar_wait_park(smem_u32(&sm.list_full[it % kPfLists]), (it / kPfLists) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok || l.kvh < 0) break;
        const int steps = l.steps;
        uint32_t q_new = 3;                              // tiles whose Q of this item has not been waited for
        PfWalk w;
        for (int i = 0; i < steps; ++i, ++gs) {
          const int b = gs & 1;
          if (ok) ok = mbar_wait_park(smem_u32(is_s ? &sm.k_full[b] : &sm.v_full[b]), (gs >> 1) & 1, abort_flag);
#pragma unroll
          for (int t = 0; t < kPfTiles; ++t) {
            if (w.step >= l.run[w.run].tile_steps[t]) continue;
            const uint32_t tile = tmem + t * kPfTmemTile;
            if (is_s) {
              if (q_new >> t & 1) {
                if (ok) ok = mbar_wait_park(smem_u32(&sm.q_full[t]), q_phase >> t & 1, abort_flag);
                q_new ^= 1u << t;
                q_phase ^= 1u << t;
              }
              if (ok && n[t] > 0) ok = mbar_wait_park(smem_u32(&sm.s_free[t]), (n[t] - 1) & 1, abort_flag);
            } else {
              if (ok) ok = mbar_wait_park(smem_u32(&sm.p_full[t]), n[t] & 1, abort_flag);
            }
            ok = __all_sync(0xffffffffu, ok);
            ++n[t];
            tc_fence_after();
            if (ok && leader) {
              if (is_s) {
#pragma unroll
                for (int part = 0; part < 2; ++part) {
                  const uint64_t k0 = dk + ((b * 2 + part) * (2 * kPfHalf) >> 4);
#pragma unroll
                  for (int k = 0; k < 4; ++k) umma_f16_ts(tile, tile + kPfTmemQ + k * 8, k0 + k * 2, idesc_s, part > 0 || k > 0);
#pragma unroll
                  for (int k = 0; k < 4; ++k) umma_f16(tile, dq + (t * (kPfRows * 128) >> 4) + k * 2, k0 + (kPfHalf >> 4) + k * 2, idesc_s, 1);
                }
                tc_commit(smem_u32(&sm.s_full[t]));
              } else {
#pragma unroll
                for (int part = 0; part < 2; ++part)
#pragma unroll
                  for (int k = 0; k < 4; ++k)
                    umma_f16_ts(tile + kPfTmemO, tile + kPfTmemP + k * 8, dv + ((b * 2 + part) * (2 * kPfHalf) >> 4) + k * (16 * 128 >> 4), idesc_o, 1);
                tc_commit(smem_u32(&sm.pv_done[t]));
              }
            }
            __syncwarp();
          }
          if (ok && leader) tc_commit(smem_u32(is_s ? &sm.k_free[b] : &sm.v_free[b]));
          __syncwarp();
          w.advance(l);
        }
        if (lane == 0) mbar_arrive(smem_u32(&sm.list_free[it % kPfLists]));
      }
    }
  } else if (warp >= 8) {
    // ------------------------------------------------------------ conversion
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kPfRegsConvert));
    // warps 8-11 convert K, warps 12-15 V: scores run a step ahead of their softmax, and wait for no conversion of V
    const bool is_v = warp >= 12;
    const int ct = tid & 127;
    int gs = 0, v_exp = 0, v_top = 0;                    // v_top: largest of the run
    for (int it = 0;; ++it) {
      const PfList& l = sm.list[it % kPfLists];
      if (ok) ok = mbar_wait_park(smem_u32(&sm.list_full[it % kPfLists]), (it / kPfLists) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok || l.kvh < 0) break;
      const int steps = l.steps;
      PfWalk w;
      for (int i = 0; i < steps; ++i, ++gs) {
        const int b = gs & 1, slot = gs % kPfRaw, note = gs % kPfNotes, visible = l.run[w.run].total - w.step * kPfTok;
        const int run = w.run, tok0 = w.step * kPfTok;
        w.advance(l);
        if (ok) ok = mbar_wait_park(smem_u32(&sm.raw_full[slot]), (gs / kPfRaw) & 1, abort_flag);
        if (ok && gs >= 2) ok = mbar_wait_park(smem_u32(is_v ? &sm.v_free[b] : &sm.k_free[b]), ((gs >> 1) - 1) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const uint8_t* pages = raw + slot * kPfPages * stride;
        float4 scale[2];
        pf_scales(pages + (is_v ? p.lay.v_scale_off : p.lay.k_scale_off), stride, visible, lane, scale);
        uint32_t most = __reduce_max_sync(0xffffffffu, max(pf_most<false>(scale[0]), pf_most<false>(scale[1])));       // (every warp for itself)
        const bool odd = most >= 0x7F800000u;                            // some are not finite
        if (odd) most = __reduce_max_sync(0xffffffffu, max(pf_most<true>(scale[0]), pf_most<true>(scale[1])));
        const int e = pf_exponent(most);
        auto redo_from = [&](int what, int tok) {                        // rows that see more than `tok` tokens of the run
          atomicMin(&sm.redo[it % kPfLists][what][run], tok);
          atomicMin(&sm.redo_least[it % kPfLists], tok);
        };
        if (!is_v) {
          // codes times scales below 2^13
          if (warp == 8) {
            if (e > kPfLarge) {
              const uint32_t of[2] = {pf_most<true>(scale[0]), pf_most<true>(scale[1])};
              if (__any_sync(0xffffffffu, (of[0] != 0 && pf_exponent(of[0]) < e - 8) || (of[1] != 0 && pf_exponent(of[1]) < e - 8)) && lane == 0) redo_from(0, tok0);
            }
            if (lane == 0) {
              sm.k_mul[note] = pow2f(e - 5);
              mbar_arrive(smem_u32(&sm.k_note[note]));
            }
          }
          pf_convert_k<KBITS>(sm.k[b], pages, stride, p.lay, pow2f(5 - e), ct);
        } else {
          // below 2^11, to be changed when they pass 2^15, or when the scales fall below 2^v_exp and that is more than one
          if (tok0 == 0) {
            v_exp = v_top = e - 3;
          } else if (e - 7 > v_exp || (v_exp > kPfLarge - 3 && e < v_exp && most != 0)) {
            v_exp = max(e - 3, v_top - kPfVFall);
            v_top = max(v_top, v_exp);
          }
          if (warp == 12) {
            if (odd || v_exp > kPfLarge - 3) {
              const float least = v_exp > kPfLarge - 3 ? pow2f(v_exp - 8) : 0.f;
#pragma unroll 1
              for (int what = 0; what < 2; ++what) {                     // tokens with a scale below 2^-8 beside large ones, with one that is not finite
                bool out[2] = {false, false};
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                  const float f[4] = {scale[h].x, scale[h].y, scale[h].z, scale[h].w};
#pragma unroll
                  for (int j = 0; j < 4; ++j) out[h] |= what == 0 ? f[j] != 0.f && fabsf(f[j]) < least : !(fabsf(f[j]) < INFINITY);
                }
                const uint32_t lo = __ballot_sync(0xffffffffu, out[0]), hi = __ballot_sync(0xffffffffu, out[1]);
                if ((lo | hi) != 0 && lane == 0) redo_from(what, tok0 + (lo != 0 ? __ffs(lo) - 1 : 31 + __ffs(hi)));
              }
            }
            if (lane == 0) {
              sm.v_exp[note] = v_exp;
              mbar_arrive(smem_u32(&sm.v_note[note]));
            }
          }
          pf_convert_v<VBITS>(sm.v[b], pages, stride, p.lay, visible, pow2f(-v_exp), ct);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(smem_u32(is_v ? &sm.v_full[b] : &sm.k_full[b]));
          mbar_arrive(smem_u32(&sm.raw_free[slot]));
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sm.list_free[it % kPfLists]));
    }
  } else {
    // --------------------------------------------------------------- softmax
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kPfRegsSoftmax));
    const int t = warp >> 2, row = tid & 127, blk = tid >> 4;
    const uint32_t tile = tmem + t * kPfTmemTile + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const int qp = (tid & 15) / p.G, hh = (tid & 15) - qp * p.G;
    struct Row {
      __nv_bfloat16* out;                                // null: not a query
      int limit;                                         // tokens that it sees
    };
    // the row of the thread in item `it`, and Q of its tile; false: no more items
    auto begin = [&](int it, Row& r) {
      const PfList& l = sm.list[it % kPfLists];
      if (ok) ok = mbar_wait_park(smem_u32(&sm.list_full[it % kPfLists]), (it / kPfLists) & 1, abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      r.out = nullptr;
      r.limit = 0;
      if (!ok || l.kvh < 0) return false;
      const __nv_bfloat16* q = nullptr;
      if (qp < l.qcount[blk]) {
        r.limit = l.ctx[blk] + qp;
        const size_t at = (static_cast<size_t>(l.qstart[blk] + qp) * p.Hq + l.kvh * p.G + hh) * kD;
        q = p.q + at;
        r.out = p.out + at;
      }
      if (l.tiles >> t & 1) {
        uint32_t x[32];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            uint4 u = make_uint4(0u, 0u, 0u, 0u);
            if (q != nullptr) u = reinterpret_cast<const uint4*>(q)[h * 8 + c];
            const uint32_t in[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&in[j]));
              x[c * 4 + j] = pack_f16x2(f.x * p.scale_log2, f.y * p.scale_log2);
            }
          }
          if (h == 0) {
            tmem_st_32x32(tile + kPfTmemQ, x);
          } else {
#pragma unroll
            for (int c = 0; c < 8; ++c)
              *reinterpret_cast<uint4*>(sm.q[t] + row * 128 + ((c ^ (row & 7)) << 4)) = make_uint4(x[4 * c], x[4 * c + 1], x[4 * c + 2], x[4 * c + 3]);
          }
        }
        tmem_st_wait();
        fence_proxy_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm.q_full[t]));
      }
      return true;
    };
    int gs = 0, n = 0;                                   // steps of earlier items; steps that this tile took part in
    Row cur;
    bool more = begin(0, cur);
    for (int it = 0; more; ++it) {
      const PfList& l = sm.list[it % kPfLists];
      const int steps = l.steps;
      const bool part = l.tiles >> t & 1;
      float m = -INFINITY, sum = 0.f;
      int v_exp = 0;
      bool first = true;
      if (part) {                                        // output starts at zero
        uint32_t z[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) z[j] = 0u;
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_st_32x32(tile + kPfTmemO + c * 32, z);
        tmem_st_wait();
      }
      PfWalk w;
      for (int i = 0; i < steps; ++i, ++gs) {
        const PfRun& r = l.run[w.run];
        const int note = gs % kPfNotes, tok0 = w.step * kPfTok;
        const bool skip = w.step >= r.tile_steps[t];
        const int sees = (blk >= r.first && blk < r.end) ? cur.limit - tok0 : 0;       // tokens of the step that this row sees
        w.advance(l);
        if (skip) continue;
        if (ok) ok = mbar_wait_park(smem_u32(&sm.s_full[t]), n & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
        uint32_t a[2][32];
        tmem_ld_32x32(tile, a[0]);
        tmem_ld_32x32(tile + 32, a[1]);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm.s_free[t]));
        // (a note is written again after this step's product, which waits for what follows: kPfNotes)
        if (ok) ok = mbar_wait_park(smem_u32(&sm.k_note[note]), (gs / kPfNotes) & 1, abort_flag);
        if (ok) ok = mbar_wait_park(smem_u32(&sm.v_note[note]), (gs / kPfNotes) & 1, abort_flag);
        if (sees < kPfTok) {
#pragma unroll
          for (int j = 0; j < kPfTok; ++j)
            if (j >= sees) a[j >> 5][j & 31] = 0xFF800000u;                             // -inf
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int j = 0; j < kPfTok; ++j) mx[j & 3] = fmaxf(mx[j & 3], __uint_as_float(a[j >> 5][j & 31]));
        const float mul = sm.k_mul[note], top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * mul;
        float alpha = 1.f;
        bool grew = top > m + kPfGrowth || (m == -INFINITY && top > m);
        if (grew) {
          alpha = fast_exp2(m - top);
          m = top;
          sum *= alpha;
        }
        const int e = sm.v_exp[note];
        if (sees > 0 && e != v_exp) {                    // (rows of other requests keep theirs: nothing is added to their outputs)
          alpha = v_exp - e < -126 ? 0.f : alpha * pow2f(v_exp - e);
          v_exp = e;
          grew = true;
        }
        const float use = m == -INFINITY ? 0.f : m;
        const float2 less = make_float2(-use, -use), mul2 = make_float2(mul, mul);
        float2 part_sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        uint32_t pr[32];
#pragma unroll
        for (int j = 0; j < kPfTok / 2; ++j) {
          const float2 d = __ffma2_rn(make_float2(__uint_as_float(a[j >> 4][2 * j & 31]), __uint_as_float(a[j >> 4][(2 * j + 1) & 31])), mul2, less);
          const float2 x = make_float2(fast_exp2(d.x), fast_exp2(d.y));
          part_sum[j & 1] = __fadd2_rn(part_sum[j & 1], x);
          pr[j] = pack_f16x2(x.x, x.y);
        }
        sum += (part_sum[0].x + part_sum[0].y) + (part_sum[1].x + part_sum[1].y);
        // the previous product has read the probabilities and written the output
        if (ok && !first) ok = mbar_wait_park(smem_u32(&sm.pv_done[t]), (n - 1) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
        tmem_st_32x32(tile + kPfTmemP, pr);
        if (!first && __any_sync(0xffffffffu, grew)) {
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t o[32];
            tmem_ld_32x32(tile + kPfTmemO + c * 32, o);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
            tmem_st_32x32(tile + kPfTmemO + c * 32, o);
          }
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm.p_full[t]));
        first = false;
        ++n;
      }
      // the next item's Q while the last product runs (all of this item's scores are there)
      Row next;
      more = begin(it + 1, next);
      if (!part) {                                       // no row of the tile sees a token
        if (cur.out != nullptr) {
#pragma unroll
          for (int j = 0; j < 16; ++j) reinterpret_cast<uint4*>(cur.out)[j] = make_uint4(0u, 0u, 0u, 0u);
        }
      } else {
        if (ok) ok = mbar_wait_park(smem_u32(&sm.pv_done[t]), (n - 1) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
        const float inv = sum > 0.f ? 1.f / sum : sum == 0.f ? 0.f : sum;               // NaN stays
        const float up = pow2f(v_exp);
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t o[32];
          tmem_ld_32x32(tile + kPfTmemO + c * 32, o);
          tmem_ld_wait();
          if (cur.out != nullptr) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint32_t x[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) x[k] = pack_bf16x2(__uint_as_float(o[8 * j + 2 * k]) * inv * up, __uint_as_float(o[8 * j + 2 * k + 1]) * inv * up);
              *reinterpret_cast<uint4*>(cur.out + c * 32 + j * 8) = make_uint4(x[0], x[1], x[2], x[3]);
            }
          }
        }
        tc_fence_before();
        if (*const_cast<volatile int*>(&sm.redo_least[it % kPfLists]) != INT_MAX && ok) {
          // (what later steps still add to `redo` is beyond what the rows of this tile see)
          __syncwarp();                                  // a row's result is written again by other lanes
          int req = 0, from[2] = {INT_MAX, INT_MAX};
          for (int i = 0; i < l.runs; ++i)
            if (blk >= l.run[i].first && blk < l.run[i].end) {
              req = l.run[i].req;
              for (int what = 0; what < 2; ++what) from[what] = *const_cast<volatile int*>(&sm.redo[it % kPfLists][what][i]);
            }
          const bool again = cur.out != nullptr && cur.limit > from[0];
          const long long at = cur.out != nullptr ? cur.out - p.out : 0;
#pragma unroll 1
          for (uint32_t rows = __ballot_sync(0xffffffffu, again); rows; rows &= rows - 1) {
            const int of = __ffs(rows) - 1;
            const long long to = __shfl_sync(0xffffffffu, at, of);
            pf_row<KBITS, VBITS>(p, __shfl_sync(0xffffffffu, req, of), l.kvh, __shfl_sync(0xffffffffu, cur.limit, of), p.q + to, p.out + to, lane);
          }
          pf_odd<KBITS, VBITS>(p, l.kvh, req, from[1], again || cur.out == nullptr ? 0 : cur.limit, at, m, inv, lane);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sm.list_free[it % kPfLists]));
      cur = next;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 16) tmem_dealloc(tmem, kPfTmemCols);
  if (tid == 0 && sm.abort_word) atomicExch(p.status, static_cast<uint32_t>(kErrBarrierTimeout));
}

template <int KB, int VB>
static int launch_prefill(const AttnParams& p, int row_blocks, cudaStream_t st) {
  const int stride = (p.lay.blob_bytes + 127) & ~127;
  const size_t smem = sizeof(PfSmem) + 1024 + static_cast<size_t>(kPfRaw) * kPfPages * stride;
  static int sms[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -18;
  if (!sms[dev]) {
    cudaError_t e = cudaFuncSetAttribute(paged_prefill_kernel<KB, VB>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    int n = 0;
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return static_cast<int>(e);
    // the warps' new shares come out of the registers that the block was launched with
    cudaFuncAttributes at;
    e = cudaFuncGetAttributes(&at, paged_prefill_kernel<KB, VB>);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (at.numRegs < kPfRegs) return -19;
    sms[dev] = n;
  }
  const long long items = static_cast<long long>((row_blocks + kPfBlocks - 1) / kPfBlocks) * p.Hkv;
  return static_cast<int>(launch(paged_prefill_kernel<KB, VB>, dim3(static_cast<unsigned>(items < sms[dev] ? items : sms[dev])), dim3(kPfThreads), smem, st, p, row_blocks));
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
