// Fused per-head RMSNorm (optional) + RoPE + KV quantize-on-write.
//
// One launch after the QKV GEMM replaces the reference's separate q/k norm,
// M-RoPE (position/qwen_mrope.py:25) and cache quantization kernels
// (cache_quantization_native.cu:49).  One warp handles one (token, head) at a
// time; lane l holds channels 4 l .. 4 l + 3: one 8-byte load and store for q, the
// eight lanes of a 32-channel quantization group are neighbours (three exchanges
// for its maximum), a rotate-half pair (c, c + 64) is lanes l and l ^ 16, and the
// four codes are one word of the K planes and one chunk of the V planes.
//
// What bounds it: with a channel of every 32 per lane (2-byte accesses, byte and
// per-code atomic stores) it was instruction issue: 4096 tokens of 32 + 8 + 8 heads 55 us, 41 us so.
#include "ptx.cuh"
#include "kv_layout.cuh"
#include "launch.cuh"

namespace cb {

static constexpr int kHeadDim = 128;

struct KvWriteParams {
  const __nv_bfloat16* qkv;    // [T, (Hq + 2*Hkv) * D]
  __nv_bfloat16* q_out;        // [T, Hq * D]
  uint8_t* cache;              // [pages][Hkv][blob]
  const int* positions;        // [T] rotary position (the temporal axis when pos_h / pos_w are given)
  const int* pos_h;            // [T] or null: row-axis positions of the three-axis rotary form
  const int* pos_w;            // [T] or null: column-axis positions
  int mrope_h, mrope_w;        // frequency slots 1, 4, 7, .. (< 3 mrope_h) follow pos_h, slots 2, 5, 8, .. (< 3 mrope_w) pos_w
  const __nv_bfloat16* qkv_bias;  // [(Hq + 2 Hkv) D] or null: bias of the q / k / v projections, added before the norm
  const int* slots;            // [T] page * 16 + offset, < 0: do not write (padding row)
  const __nv_bfloat16* q_norm; // [D] or null
  const __nv_bfloat16* k_norm; // [D] or null
  const float* inv_freq;       // [D/2]
  int T, Hq, Hkv;
  int rotary_dim;              // <= D, multiple of 2; pairs (c, c + rotary_dim/2)
  float eps;
  int rotate;                  // normalised Walsh-Hadamard transform of every q / k / v head vector (after RoPE)
  KvLayout lay;
};

// Four neighbouring channels; eight bytes at once where every row starts on a multiple of eight (WIDE).
template <bool WIDE>
__device__ __forceinline__ void load4(const __nv_bfloat16* at, float (&v)[4]) {
  if constexpr (WIDE) {
    const uint2 raw = *reinterpret_cast<const uint2*>(at);
    const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x)), hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    v[0] = lo.x; v[1] = lo.y; v[2] = hi.x; v[3] = hi.y;
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = __bfloat162float(at[k]);
  }
}
template <bool WIDE>
__device__ __forceinline__ void store4(__nv_bfloat16* at, uint2 v) {
  if constexpr (WIDE) {
    *reinterpret_cast<uint2*>(at) = v;
  } else {
    const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&v.x), hi = *reinterpret_cast<const __nv_bfloat162*>(&v.y);
    at[0] = lo.x; at[1] = lo.y; at[2] = hi.x; at[3] = hi.y;
  }
}
static inline bool on8(const void* a, const void* b) { return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 7) == 0; }

// Normalised Walsh-Hadamard transform of a 128-vector held as v[a] = x[4 lane + a] (the transform treats all index bits alike,
// so any four of them may be the registers).  fp32 stages, the caller rounds once (reference:
// ops/cuda/cache_rotation_native.cu:12).  The transform is its own inverse, and q . k is unchanged when both are
// transformed, so attention over a rotated cache needs only the transform of its output (V's rotation undone).
__device__ __forceinline__ void hadamard128(float (&v)[4], int lane) {
  float a = v[0] + v[1], b = v[0] - v[1], c = v[2] + v[3], d = v[2] - v[3];
  v[0] = a + c; v[1] = b + d; v[2] = a - c; v[3] = b - d;
#pragma unroll
  for (int m = 1; m < 32; m <<= 1) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float o = __shfl_xor_sync(0xffffffffu, v[k], m);
      v[k] = (lane & m) ? o - v[k] : v[k] + o;
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) v[k] *= 0.08838834764831845f;     // 1 / sqrt(128)
}

// four bytes, or four nibble fields at the bytes' bit `shift`, of a word that other tokens' writers share
__device__ __forceinline__ void merge_word(uint8_t* at, uint32_t mask, uint32_t bits) {
  atomicAnd(reinterpret_cast<uint32_t*>(at), ~mask);
  atomicOr(reinterpret_cast<uint32_t*>(at), bits);
}

// `v`: channels 4 lane .. 4 lane + 3 of a K or V head vector of token slot `tok` (layout: kv_layout.cuh).
__device__ __forceinline__ void quantize_store(const float (&v)[4], int bits, bool is_v, uint8_t* blob,
                                               const KvLayout& lay, int tok, int lane) {
  const float qmax = bits == 8 ? 127.f : (bits == 6 ? 31.f : 7.f);
  const int bias = bits == 8 ? 128 : (bits == 6 ? 32 : 8);
  uint8_t* codes = blob + (is_v ? lay.v_code_off : 0);
  float* scales = reinterpret_cast<float*>(blob + (is_v ? lay.v_scale_off : lay.k_scale_off));
  float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
  amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
  const float scale = amax > 0.f ? amax / qmax : 1.f;
  uint32_t word = 0;                                     // the four codes, a byte each
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float c = fminf(fmaxf(rintf(v[k] / scale), -qmax), qmax);
    word |= static_cast<uint32_t>(static_cast<int>(c) + bias) << (8 * k);
  }
  const int blk = lane >> 3, t = lane & 3;
  if ((lane & 7) == 0) scales[tok * (kHeadDim / kKvGroup) + blk] = scale;
  if (!is_v) {
    if (bits == 8) {
      *reinterpret_cast<uint32_t*>(codes + (lane >> 2) * 256 + tok * 16 + t * 4) = word;
      return;
    }
    // lanes t and t + 4 of a block: channels c and c + 16 share bytes
    const uint32_t other = __shfl_xor_sync(0xffffffffu, word, 4);
    if (lane & 4) return;
    *reinterpret_cast<uint32_t*>(codes + blk * 256 + tok * 16 + t * 4) = (word & 0x0F0F0F0Fu) | ((other & 0x0F0F0F0Fu) << 4);
    if (bits == 6) {
      const uint32_t hi = (word & 0x30303030u) | ((other & 0x30303030u) << 2);        // bits 4..7 of every byte
      merge_word(codes + kPageTokens * kHeadDim / 2 + blk * 128 + (tok & 7) * 16 + t * 4, tok < 8 ? 0xF0F0F0F0u : 0x0F0F0F0Fu, tok < 8 ? hi : hi >> 4);
    }
    return;
  }
  const int pair = tok >> 1, chunk = lane ^ ((pair & 3) << 2);
  if (bits == 8) {
    uint8_t* at = codes + pair * (kHeadDim * 2) + chunk * 8 + (tok & 1);
#pragma unroll
    for (int k = 0; k < 4; ++k) at[2 * k] = static_cast<uint8_t>(word >> (8 * k));
    return;
  }
  // even and odd tokens share bytes
  const int odd = tok & 1;
  merge_word(codes + pair * kHeadDim + chunk * 4, odd ? 0xF0F0F0F0u : 0x0F0F0F0Fu, odd ? (word & 0x0F0F0F0Fu) << 4 : word & 0x0F0F0F0Fu);
  if (bits == 6) {
    const int shift = (pair < 4 ? 0 : 4) - 2 * odd;      // bits 4, 5 of a code to bit 4 or 0, two further for odd tokens
    const uint32_t hi = word & 0x30303030u;
    merge_word(codes + kPageTokens * kHeadDim / 2 + (pair & 3) * kHeadDim + chunk * 4, shift >= 0 ? 0x30303030u >> shift : 0x30303030u << -shift,
               shift >= 0 ? hi >> shift : hi << -shift);
  }
}

static constexpr int kRopeWarps = 8;

// One CTA per token; its eight warps share the token's heads (warp w takes heads w, w + 8, ...).  The rotary
// angles depend on (position, channel) only, so the CTA computes its sin / cos pairs ONCE, a thread each, and reuses them
// for every head of the token: full-precision sincosf on arguments of thousands of radians is expensive.
template <bool WIDE>
__global__ void __launch_bounds__(kRopeWarps * 32)
rope_kv_write_kernel(const KvWriteParams p) {
  __shared__ __align__(16) float sn_s[64], cs_s[64];
  pdl_wait();
  pdl_launch_dependents();
  const int t = blockIdx.x;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int heads = p.Hq + 2 * p.Hkv;
  const int half = p.rotary_dim >> 1;
  if (threadIdx.x < half) {
    // three-axis form: frequency slot j turns by the position on its axis (interleaved layout: temporal by default, the
    // row axis on slots 1, 4, 7, .., the column axis on 2, 5, 8, .. as far as their counts reach)
    const int j = threadIdx.x, r = j % 3;
    int pos = p.positions[t];
    if (p.pos_h != nullptr) {
      if (r == 1 && j < 3 * p.mrope_h) pos = p.pos_h[t];
      if (r == 2 && j < 3 * p.mrope_w) pos = p.pos_w[t];
    }
    sincosf(static_cast<float>(pos) * p.inv_freq[j], &sn_s[j], &cs_s[j]);
  }
  const int slot = p.slots[t];
  __syncthreads();
  // lane's frequency slots: its channels modulo the rotated half
  const bool turns = 4 * lane < p.rotary_dim, upper = 4 * lane >= half;
  float4 sn = make_float4(0.f, 0.f, 0.f, 0.f), cs = make_float4(1.f, 1.f, 1.f, 1.f);
  if (turns) {
    sn = *reinterpret_cast<const float4*>(sn_s + (4 * lane - (upper ? half : 0)));
    cs = *reinterpret_cast<const float4*>(cs_s + (4 * lane - (upper ? half : 0)));
    if (!upper) sn = make_float4(-sn.x, -sn.y, -sn.z, -sn.w);      // a cos - b sin below, b cos + a sin above
  }
  const int pair_lane = half >> 2;                                 // lanes between the two channels of a pair
#pragma unroll 2
  for (int h = warp; h < heads; h += kRopeWarps) {
    float v[4];
    load4<WIDE>(p.qkv + (static_cast<size_t>(t) * heads + h) * kHeadDim + 4 * lane, v);
    if (p.qkv_bias != nullptr) {
      // the projection's output was rounded to bf16 by the GEMM; the sum is rounded again, as an unfused add would
#pragma unroll
      for (int k = 0; k < 4; ++k)
        v[k] = __bfloat162float(__float2bfloat16(v[k] + __bfloat162float(p.qkv_bias[h * kHeadDim + 4 * lane + k])));
    }
    const bool is_q = h < p.Hq;
    const bool is_k = !is_q && h < p.Hq + p.Hkv;
    if (is_q || is_k) {
      const __nv_bfloat16* nw = is_q ? p.q_norm : p.k_norm;
      if (nw) {
        float ss = v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3];
        ss = warp_sum(ss);
        const float inv = rsqrtf(ss / static_cast<float>(kHeadDim) + p.eps);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          // round to bf16 after the norm, as an unfused norm kernel would
          v[k] = __bfloat162float(__float2bfloat16(v[k] * inv * __bfloat162float(nw[4 * lane + k])));
        }
      }
      if (half) {
        float o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) o[k] = __shfl_xor_sync(0xffffffffu, v[k], pair_lane);
        if (turns) {
          v[0] = v[0] * cs.x + o[0] * sn.x; v[1] = v[1] * cs.y + o[1] * sn.y;
          v[2] = v[2] * cs.z + o[2] * sn.z; v[3] = v[3] * cs.w + o[3] * sn.w;
        }
      }
    }
    if (p.rotate) hadamard128(v, lane);
    const uint2 bf = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
    if (is_q) {
      store4<WIDE>(p.q_out + (static_cast<size_t>(t) * p.Hq + h) * kHeadDim + 4 * lane, bf);
      continue;
    }
    if (slot < 0) continue;
    const int kvh = is_k ? h - p.Hq : h - p.Hq - p.Hkv;
    const int page = slot >> 4, tok = slot & 15;
    uint8_t* blob = p.cache + (static_cast<size_t>(page) * p.Hkv + kvh) * p.lay.blob_bytes;
    // the cache stores what attention will see: bf16-rounded values
    const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&bf.x)), hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&bf.y));
    const float r[4] = {lo.x, lo.y, hi.x, hi.y};
    quantize_store(r, is_k ? p.lay.k_bits : p.lay.v_bits, !is_k, blob, p.lay, tok, lane);
  }
}

// Walsh-Hadamard transform of `vectors` consecutive 128-vectors per row (in place allowed): undoes the rotation of
// V on the attention output.  One warp per vector.
template <bool WIDE>
__global__ void __launch_bounds__(256)
hadamard_kernel(const __nv_bfloat16* __restrict__ x, int ldx, __nv_bfloat16* __restrict__ y, int ldy, int vectors,
                int rows) {
  pdl_wait();
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31;
  const long long w = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (w >= static_cast<long long>(rows) * vectors) return;
  const int r = static_cast<int>(w / vectors), h = static_cast<int>(w - static_cast<long long>(r) * vectors);
  const __nv_bfloat16* src = x + static_cast<size_t>(r) * ldx + h * 128;
  __nv_bfloat16* dst = y + static_cast<size_t>(r) * ldy + h * 128;
  float v[4];
  load4<WIDE>(src + 4 * lane, v);
  hadamard128(v, lane);
  store4<WIDE>(dst + 4 * lane, make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3])));
}

// Copy whole pages (all kv heads) src -> dst: copy-on-write of a shared page.
__global__ void __launch_bounds__(256)
copy_pages_kernel(uint8_t* cache, const int* src_pages, const int* dst_pages, int page_bytes_vec) {
  const int s = src_pages[blockIdx.x], d = dst_pages[blockIdx.x];
  if (s < 0 || d < 0 || s == d) return;
  const uint4* sp = reinterpret_cast<const uint4*>(cache + static_cast<size_t>(s) * page_bytes_vec * 16);
  uint4* dp = reinterpret_cast<uint4*>(cache + static_cast<size_t>(d) * page_bytes_vec * 16);
  // blockIdx.y strides over the page, so that rows of megabytes (recurrent-state rows) use more than one SM
  for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < page_bytes_vec; i += blockDim.x * gridDim.y) dp[i] = sp[i];
}

}  // namespace cb

extern "C" {

int cb_kv_blob_bytes(int head_dim, int k_bits, int v_bits) {
  return cb::make_kv_layout(head_dim, k_bits, v_bits).blob_bytes;
}

// Three-axis rotary positions: ``positions`` is the temporal axis, ``pos_h`` / ``pos_w`` the row and column axes (both
// null: one axis); ``mrope_h`` / ``mrope_w`` are the frequency-slot counts of those two axes.  ``qkv_bias`` (or null) is
// added to every q / k / v row as it is read.
int cb_rope_kv_write_axes(const void* qkv, void* q_out, void* cache, const void* positions, const void* pos_h,
                          const void* pos_w, int mrope_h, int mrope_w, const void* qkv_bias, const void* slots,
                          const void* q_norm, const void* k_norm, const void* inv_freq, int T, int Hq, int Hkv, int D,
                          int rotary_dim, float eps, int k_bits, int v_bits, int rotate, void* stream);

int cb_rope_kv_write(const void* qkv, void* q_out, void* cache, const void* positions, const void* slots,
                     const void* q_norm, const void* k_norm, const void* inv_freq, int T, int Hq, int Hkv, int D,
                     int rotary_dim, float eps, int k_bits, int v_bits, int rotate, void* stream) {
  return cb_rope_kv_write_axes(qkv, q_out, cache, positions, nullptr, nullptr, 0, 0, nullptr, slots, q_norm, k_norm,
                               inv_freq, T, Hq, Hkv, D, rotary_dim, eps, k_bits, v_bits, rotate, stream);
}

int cb_rope_kv_write_axes(const void* qkv, void* q_out, void* cache, const void* positions, const void* pos_h,
                          const void* pos_w, int mrope_h, int mrope_w, const void* qkv_bias, const void* slots,
                          const void* q_norm, const void* k_norm, const void* inv_freq, int T, int Hq, int Hkv, int D,
                          int rotary_dim, float eps, int k_bits, int v_bits, int rotate, void* stream) {
  using namespace cb;
  if (T <= 0) return 0;
  if (D != 128) return -10;
  if (!(k_bits == 8 || k_bits == 6 || k_bits == 4) || !(v_bits == 8 || v_bits == 6 || v_bits == 4)) return -11;
  if (!(rotary_dim == 128 || rotary_dim == 64 || rotary_dim == 0)) return -12;
  if ((pos_h == nullptr) != (pos_w == nullptr)) return -13;
  if (pos_h != nullptr) {
    const int half = rotary_dim / 2;   // the last slot of either axis has to exist: 3 h - 2 and 3 w - 1 below half
    if (mrope_h <= 0 || mrope_w <= 0 || 3 * mrope_h - 2 >= half || 3 * mrope_w - 1 >= half) return -14;
  }
  KvWriteParams p;
  p.pos_h = static_cast<const int*>(pos_h);
  p.pos_w = static_cast<const int*>(pos_w);
  p.mrope_h = mrope_h;
  p.mrope_w = mrope_w;
  p.qkv_bias = static_cast<const __nv_bfloat16*>(qkv_bias);
  p.qkv = static_cast<const __nv_bfloat16*>(qkv);
  p.q_out = static_cast<__nv_bfloat16*>(q_out);
  p.cache = static_cast<uint8_t*>(cache);
  p.positions = static_cast<const int*>(positions);
  p.slots = static_cast<const int*>(slots);
  p.q_norm = static_cast<const __nv_bfloat16*>(q_norm);
  p.k_norm = static_cast<const __nv_bfloat16*>(k_norm);
  p.inv_freq = static_cast<const float*>(inv_freq);
  p.T = T; p.Hq = Hq; p.Hkv = Hkv; p.rotary_dim = rotary_dim; p.eps = eps; p.rotate = rotate;
  p.lay = make_kv_layout(D, k_bits, v_bits);
  // rows are multiples of 256 bytes, so the first decides for all
  return static_cast<int>(launch(on8(qkv, q_out) ? rope_kv_write_kernel<true> : rope_kv_write_kernel<false>, dim3(static_cast<unsigned>(T)), dim3(kRopeWarps * 32), 0,
                                 static_cast<cudaStream_t>(stream), p));
}

// y[r, 128 h .. 128 h + 127] = normalised Walsh-Hadamard transform of x[r, same], h < vectors (bf16, in place allowed).
int cb_hadamard(const void* x, int ldx, void* y, int ldy, int vectors, int rows, void* stream) {
  if (rows <= 0 || vectors <= 0) return 0;
  const long long warps = static_cast<long long>(rows) * vectors;
  const bool wide = cb::on8(x, y) && (rows == 1 || ((ldx | ldy) & 3) == 0);
  return static_cast<int>(cb::launch(wide ? cb::hadamard_kernel<true> : cb::hadamard_kernel<false>, dim3(static_cast<unsigned>((warps + 7) / 8)), dim3(256), 0,
                                     static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(x), ldx,
                                     static_cast<__nv_bfloat16*>(y), ldy, vectors, rows));
}

int cb_copy_pages(void* cache, const void* src_pages, const void* dst_pages, int n, long long page_bytes,
                  void* stream) {
  if (n <= 0) return 0;
  if (page_bytes % 16 != 0) return -10;
  const long long vecs = page_bytes / 16;
  const unsigned chunks = static_cast<unsigned>(vecs > 256 * 16 ? (vecs / (256 * 16) > 64 ? 64 : vecs / (256 * 16)) : 1);
  cb::copy_pages_kernel<<<dim3(static_cast<unsigned>(n), chunks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<uint8_t*>(cache), static_cast<const int*>(src_pages), static_cast<const int*>(dst_pages),
      static_cast<int>(page_bytes / 16));
  return static_cast<int>(cudaGetLastError());
}

}  // extern "C"
