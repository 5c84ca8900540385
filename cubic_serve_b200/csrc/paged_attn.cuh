// Shared by the paged attention kernels (paged_attn.cu: decode and short row blocks, paged_prefill.cu: portions of prompts):
// parameters, fragments, and the host side's argument checks.
#pragma once
#include "ptx.cuh"
#include "launch.cuh"
#include "kv_layout.cuh"
#include <type_traits>

namespace cb {

static constexpr int kD = 128;

struct AttnParams {
  const __nv_bfloat16* q;   // [T, Hq, D]
  __nv_bfloat16* out;       // [T, Hq, D]
  const uint8_t* cache;     // [pages][Hkv][blob]
  const int* page_table;    // [requests, max_pages]
  const int* rb_req;        // [row_blocks] request (page-table row)
  const int* rb_qstart;     // [row_blocks] index of first query token in q/out
  const int* rb_qcount;     // [row_blocks] query positions in this block (<= 16/G); 0 = padding block
  const int* rb_ctx;        // [row_blocks] tokens visible to the FIRST query position (its own included)
  float* partial;           // [row_blocks][Hkv][splits][16][D + 2] fp32 (splits > 1)
  uint32_t* counters;       // [row_blocks * Hkv] zero on entry, zero on exit
  uint32_t* status;
  int Hq, Hkv, G;
  int max_pages;
  int splits;
  float scale_log2;         // softmax scale * log2(e)
  KvLayout lay;
};

__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}
// two offset-binary bytes (selected by `sel` against the 0x64 magic) -> f16x2 of the signed codes
__device__ __forceinline__ uint32_t u8x2_to_f16x2(uint32_t word, uint32_t sel, uint32_t bias_f16x2) {
  uint32_t v = prmt(word, 0x64646464u, sel);
  uint32_t r;
  asm("sub.f16x2 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(bias_f16x2));
  return r;
}
__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float fast_exp2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

struct WarpState {
  float m[2];       // running max (log2 domain) for rows g and g+8
  float l[2];       // running partial sum (this lane's columns only)
  float o[16][4];   // O accumulators: n-tile (cg*4 + sub) x {row g: 2 cols, row g+8: 2 cols}
};

// Fills `p` from the arguments of the C entries; 0 or a negative argument error.
static inline int make_attn_params(AttnParams& p, const void* q, void* out, const void* cache, const void* page_table, const void* rb_req, const void* rb_qstart,
                                   const void* rb_qcount, const void* rb_ctx, int Hq, int Hkv, int D, int max_pages, int k_bits, int v_bits, float scale, int splits,
                                   void* partial, void* counters, void* status) {
  if (D != kD || Hkv <= 0 || Hq % Hkv != 0) return -10;
  const int G = Hq / Hkv;
  if (G > 16 || (16 % G) != 0) return -11;
  if (splits < 1) splits = 1;
  if (splits > 1 && (!partial || !counters)) return -12;
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.out = static_cast<__nv_bfloat16*>(out);
  p.cache = static_cast<const uint8_t*>(cache);
  p.page_table = static_cast<const int*>(page_table);
  p.rb_req = static_cast<const int*>(rb_req);
  p.rb_qstart = static_cast<const int*>(rb_qstart);
  p.rb_qcount = static_cast<const int*>(rb_qcount);
  p.rb_ctx = static_cast<const int*>(rb_ctx);
  p.partial = static_cast<float*>(partial);
  p.counters = static_cast<uint32_t*>(counters);
  p.status = static_cast<uint32_t*>(status);
  p.Hq = Hq; p.Hkv = Hkv; p.G = G; p.max_pages = max_pages; p.splits = splits;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.lay = make_kv_layout(D, k_bits, v_bits);
  return 0;
}

// Calls `f` with the bits of K and V as constants; -13 for widths that the cache does not have.
template <typename F>
static inline int with_kv_bits(int k_bits, int v_bits, F&& f) {
  auto with_v = [&](auto kb) {
    switch (v_bits) {
      case 8: return f(kb, std::integral_constant<int, 8>());
      case 6: return f(kb, std::integral_constant<int, 6>());
      case 4: return f(kb, std::integral_constant<int, 4>());
      default: return -13;
    }
  };
  switch (k_bits) {
    case 8: return with_v(std::integral_constant<int, 8>());
    case 6: return with_v(std::integral_constant<int, 6>());
    case 4: return with_v(std::integral_constant<int, 4>());
    default: return -13;
  }
}

}  // namespace cb
