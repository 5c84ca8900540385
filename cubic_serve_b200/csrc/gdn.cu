// Gated DeltaNet (linear attention) layer kernels of the hybrid decoder family.
//
// A step's tokens arrive as SEGMENTS: the contiguous rows [row0, row0 + count) of one request, whose first row has
// absolute position pos0; `slot` is the request's row of the persistent state tensors.  A request that starts at
// position 0 starts from zero state (slots are reused without clearing).
//
//   gdn_conv_kernel    depthwise causal conv1d (kernel 4) + SiLU over the mixed q/k/v channels, history in registers,
//                      per-request conv state (the last three inputs of every channel)
//   gdn_delta_kernel   per (segment, value head): L2-normalised q / k, beta = sigmoid(b),
//                      decay = exp(-exp(A_log) * softplus(a + dt_bias)), the gated delta rule
//                          S <- S * decay;  delta = (v - S k) * beta;  S <- S + delta k^T;  o = S q
//                      with the 128 x 128 fp32 state of the head held in registers for the whole segment, then the
//                      gated RMSNorm of the head (o * rsqrt(mean o^2 + eps) * w * silu(z))
//
// Speculative review passes run both kernels with commit = 0: outputs are produced for every row, the persistent
// state is left as it was.  Once the accepted prefix is known (on the device), the SAME kernels run again over the
// recorded inputs of the review rows with segments whose count is the accepted length and commit = 1: that fold
// brings conv and delta state to the accepted position without a host round trip (the reference's separate fold
// kernel: ops/cuda/linear_attention/gated_delta_fold.cu:22).
//
// Reference counterparts: ops/cuda/linear_attention/causal_conv_native.cu:13, gated_delta_native.cu:36,
// gated_delta_coefficients_native.cu:17 and the oracle ops/eager/hybrid.py:255-548 (fp32 recurrence branch).
#include "launch.cuh"
#include "mma.cuh"
#include "ptx.cuh"
#include "segments.cuh"
#include <limits.h>
#include <type_traits>

namespace cb {

static constexpr int kGdnDim = 128;            // key and value head width (d_k = d_v = 128)

struct GdnSegments {
  const int* row0;      // [S] first row of the segment in the step's token order
  const int* count;     // [S] rows of the segment (0 = padding)
  const int* slot;      // [S] state slot of the request
  const int* pos0;      // [S] absolute position of the first row (0 = fresh state)
};

// Tiles of kConvRows rows of a segment x 128 threads of V neighbouring channels.  The convolution has no chain: a tile takes the
// three inputs before its first row from the rows themselves.  (One thread walking a channel's whole segment left 3000 rows of
// 8192 channels to 320 blocks with four loads in flight each: 290 us where the bytes take 15.)  Only the first tile of a segment
// touches the request's state: it has read the old inputs before it writes the new ones.  Rows that are written over the rows that
// are read (`x` and `y` are not __restrict__) take tiles as long as the step: one thread then walks its channels of a whole segment, every row
// read before it is written.
static constexpr int kConvRows = 32;

struct ConvTile {
  int row0, count, slot, pos0, off;                     // the tile's segment, and the tile's first row inside it
};

// find_tile (segments.cuh) with all that is known of a segment loaded at once: in short steps the chain of loads is the time.
__device__ __forceinline__ bool conv_tile(const Segments& sg, int rows, int tile, ConvTile& t) {
  if (sg.single) {
    t = ConvTile{sg.row0[tile], sg.count[tile], sg.slot[tile], sg.pos0[tile], 0};
    return t.count > 0;
  }
  const int lane = threadIdx.x & 31;
  int base = 0;
  for (int s0 = 0; s0 < sg.num; s0 += 32) {
    const int s = min(s0 + lane, sg.num - 1);
    ConvTile v{sg.row0[s], sg.count[s], sg.slot[s], sg.pos0[s], 0};
    const int nb = s0 + lane < sg.num ? (v.count + rows - 1) / rows : 0;
    int inc = nb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int w = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += w;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, base + inc > tile);
    if (hit) {
      const int l = __ffs(hit) - 1;
      t.row0 = __shfl_sync(0xffffffffu, v.row0, l);
      t.count = __shfl_sync(0xffffffffu, v.count, l);
      t.slot = __shfl_sync(0xffffffffu, v.slot, l);
      t.pos0 = __shfl_sync(0xffffffffu, v.pos0, l);
      t.off = (tile - (base + __shfl_sync(0xffffffffu, inc - nb, l))) * rows;
      return true;
    }
    base += __shfl_sync(0xffffffffu, inc, 31);
  }
  return false;
}

template <int V>
__global__ void __launch_bounds__(128, 10)
gdn_conv_kernel(const __nv_bfloat16* x, int ldx, __nv_bfloat16* y, int ldy,
                const float* __restrict__ w,            // [C, 4], tap 3 multiplies the current input
                const float* __restrict__ bias,         // [C] or null
                __nv_bfloat16* __restrict__ state,      // [slots, 3, C]
                Segments seg, int tile_rows, int C, int commit) {
  ConvTile tile;
  if (!conv_tile(seg, tile_rows, blockIdx.y, tile)) return;
  const int c = (blockIdx.x * 128 + threadIdx.x) * V;
  if (c >= C) return;
  const int n = tile.count, off = tile.off;
  const __nv_bfloat16* xp = x + static_cast<size_t>(tile.row0) * ldx + c;
  __nv_bfloat16* yp = y + static_cast<size_t>(tile.row0) * ldy + c;
  __nv_bfloat16* st = state + static_cast<size_t>(tile.slot) * 3 * C + c;
  struct Chan { float v[V]; };
  using Raw = std::conditional_t<V == 2, __nv_bfloat162, __nv_bfloat16>;      // rows in flight stay packed: registers are what bounds a decode step
  auto fetch = [](const __nv_bfloat16* at) { return *reinterpret_cast<const Raw*>(at); };
  auto widen = [](Raw x) {
    Chan r;
    if constexpr (V == 2) {
      const float2 f = __bfloat1622float2(x);
      r.v[0] = f.x; r.v[1] = f.y;
    } else {
      r.v[0] = __bfloat162float(x);
    }
    return r;
  };
  auto load = [&](const __nv_bfloat16* at) { return widen(fetch(at)); };
  auto store = [](__nv_bfloat16* at, const Chan& r) {
    if constexpr (V == 2) *reinterpret_cast<__nv_bfloat162*>(at) = __floats2bfloat162_rn(r.v[0], r.v[1]);
    else *at = __float2bfloat16(r.v[0]);
  };
  float4 wv[V];
  float b[V];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    wv[i] = *reinterpret_cast<const float4*>(w + static_cast<size_t>(c + i) * 4);
    b[i] = bias ? bias[c + i] : 0.f;
  }
  Chan h[3] = {};                                       // inputs at t - 3, t - 2, t - 1
  if (off > 0) {
#pragma unroll
    for (int j = 0; j < 3; ++j) h[j] = load(xp + static_cast<size_t>(off - 3 + j) * ldx);
  } else if (tile.pos0 > 0) {
#pragma unroll
    for (int j = 0; j < 3; ++j) h[j] = load(st + static_cast<size_t>(j) * C);
  }
  // the segment's last three inputs: of a longer segment from its rows, else they are in registers at the end (to fetch them here made
  // a step of four rows wait for memory twice, 11 us instead of 9)
  commit &= off == 0;
  if (commit && n > tile_rows) {
#pragma unroll
    for (int j = 0; j < 3; ++j) store(st + static_cast<size_t>(j) * C, load(xp + static_cast<size_t>(n - 3 + j) * ldx));
  }
  const int end = off + min(n - off, tile_rows);
  // N rows at a time: the loads do not depend on the arithmetic, so they are issued together.  A decode step runs the code of one row only:
  // its instructions come from memory too.
  int t = off;
  auto rows = [&](auto count) {
    constexpr int N = decltype(count)::value;
    Raw v[N];
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = fetch(xp + static_cast<size_t>(t + j) * ldx);
#pragma unroll
    for (int j = 0; j < N; ++j) {
      Chan o;
      const Chan x0 = widen(v[j]);
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const float a = b[i] + wv[i].x * h[0].v[i] + wv[i].y * h[1].v[i] + wv[i].z * h[2].v[i] + wv[i].w * x0.v[i];
        o.v[i] = silu_fast(a);
      }
      store(yp + static_cast<size_t>(t + j) * ldy, o);
      h[0] = h[1]; h[1] = h[2]; h[2] = x0;
    }
    t += N;
  };
  while (t + 8 <= end) rows(std::integral_constant<int, 8>());
  if (t + 4 <= end) rows(std::integral_constant<int, 4>());
  if (t + 2 <= end) rows(std::integral_constant<int, 2>());
  if (t < end) rows(std::integral_constant<int, 1>());
  if (commit && n <= tile_rows) {
#pragma unroll
    for (int j = 0; j < 3; ++j) store(st + static_cast<size_t>(j) * C, h[j]);
  }
}

struct GdnDeltaParams {
  const __nv_bfloat16* qkv;   // [T, ldqkv] after the convolution: q [Hk * 128] | k [Hk * 128] | v [Hv * 128]
  int ldqkv;
  const __nv_bfloat16* z;     // [T, ldz] gate of the output norm, [Hv * 128]
  int ldz;
  const __nv_bfloat16* ba;    // [T, ldba]: b [Hv] | a [Hv]
  int ldba;
  const float* a_log;         // [Hv]
  const float* dt_bias;       // [Hv]
  const float* norm_w;        // [128]
  float* state;               // [slots, Hv, 128 (v), 128 (k)] fp32
  __nv_bfloat16* out;         // [T, ldo]: [Hv * 128]
  int ldo;
  int Hk, Hv;
  float eps_norm;             // RMSNorm epsilon
  float eps_l2;               // L2-normalisation epsilon
  int commit;                 // 0: the state is read but not written back (speculative review pass)
  int most;                   // segments of more rows are left out (gdn_delta_chunk_kernel takes them)
  GdnSegments seg;
};

// grid (Hv, segments), 256 threads.  Eight lanes share a state row: lane l8 = lane & 7 owns the float4 chunks
// l8, l8 + 8, l8 + 16, l8 + 24 of the row's 128 key columns, so one load instruction of a warp covers four whole
// 512-byte rows (fully coalesced; the state is the only large operand: 64 KiB per CTA read and written once per
// step).  A thread holds four rows: warp * 16 + (lane >> 3) + 4 i.  Row sums (S k and S q) are reduced over the
// eight lanes by shuffles.  Two CTAs per SM (128 registers per thread): one CTA's state load / store overlaps the
// other's arithmetic.
//
// A segment is walked in blocks of 16 tokens, three phases per block:
//   A (parallel, three warp tasks per token)  L2-normalised q / k, v, z, beta and decay of the block's tokens into shared memory
//   B (the recurrence, no CTA barrier inside)  per token: decay, S k, delta, rank-one update, S q; outputs to shared memory
//   C (parallel, a warp per token)  gated RMSNorm of the block's outputs, coalesced stores
// so the token-serial part is only the arithmetic that really depends on the state.
static constexpr int kGdnBlock = 16;

__global__ void __launch_bounds__(256, 2)
gdn_delta_kernel(const GdnDeltaParams p) {
  const int head = blockIdx.x;
  const int s = blockIdx.y;
  const int n = p.seg.count[s];
  if (n <= 0 || n > p.most) return;
  const int row0 = p.seg.row0[s];
  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int l8 = lane & 7;
  const int vrow = warp * 16 + (lane >> 3);              // + 4 i
  const int khead = head / (p.Hv / p.Hk);
  __shared__ __align__(16) float qs[kGdnBlock][kGdnDim];
  __shared__ __align__(16) float ks[kGdnBlock][kGdnDim];
  __shared__ float vs[kGdnBlock][kGdnDim];
  __shared__ float os[kGdnBlock][kGdnDim];
  __shared__ float zs[kGdnBlock][kGdnDim];
  __shared__ float4 coef[kGdnBlock];                      // {beta, decay, k . q}

  float* sp = p.state + ((static_cast<size_t>(p.seg.slot[s]) * p.Hv + head) * kGdnDim + vrow) * kGdnDim + l8 * 4;
  float2 S[4][4][2];                                     // [row i][chunk c]: columns 4 (l8 + 8 c) .. + 3
  if (p.seg.pos0[s] > 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float4 e = *reinterpret_cast<const float4*>(sp + (4 * i) * kGdnDim + 32 * c);
        S[i][c][0] = make_float2(e.x, e.y);
        S[i][c][1] = make_float2(e.z, e.w);
      }
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) S[i][c][0] = S[i][c][1] = make_float2(0.f, 0.f);
  }
  const float neg_exp_a = -__expf(p.a_log[head]);
  const float dtb = p.dt_bias[head];
  const int q_off = khead * kGdnDim, k_off = (p.Hk + khead) * kGdnDim, v_off = (2 * p.Hk + head) * kGdnDim;
  float nw[4];
#pragma unroll
  for (int a = 0; a < 4; ++a) nw[a] = p.norm_w[lane + 32 * a];

  for (int t0 = 0; t0 < n; t0 += kGdnBlock) {
    const int nb = min(kGdnBlock, n - t0);
    // ---- A: operands of the block's tokens.  Three independent tasks per token (q and k, v and z, coefficients) dealt
    // to the eight warps, so that a one-token decode step still uses three warps at once
    for (int task = warp; task < nb * 3; task += 8) {
      const int j = task / 3, part = task - j * 3;
      const size_t r = static_cast<size_t>(row0 + t0 + j);
      const __nv_bfloat16* row = p.qkv + r * p.ldqkv;
      if (part == 0) {
        // stored boundary of the oracle: normalised q / k are rounded to bf16; q carries the 1 / sqrt(d_k) scale
        float q[4], k[4], qq = 0.f, kk = 0.f, kq = 0.f;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          q[a] = __bfloat162float(row[q_off + lane + 32 * a]);
          k[a] = __bfloat162float(row[k_off + lane + 32 * a]);
          qq = fmaf(q[a], q[a], qq);
          kk = fmaf(k[a], k[a], kk);
        }
        const float qi = rsqrtf(warp_sum(qq) + p.eps_l2), ki = rsqrtf(warp_sum(kk) + p.eps_l2);
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const float qn = __bfloat162float(__float2bfloat16(q[a] * qi)) * 0.08838834764831845f, kn = __bfloat162float(__float2bfloat16(k[a] * ki));
          qs[j][lane + 32 * a] = qn;
          ks[j][lane + 32 * a] = kn;
          kq = fmaf(kn, qn, kq);
        }
        kq = warp_sum(kq);
        if (lane == 0) coef[j].z = kq;
      } else if (part == 1) {
        const __nv_bfloat16* zrow = p.z + r * p.ldz + head * kGdnDim;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          vs[j][lane + 32 * a] = __bfloat162float(row[v_off + lane + 32 * a]);
          zs[j][lane + 32 * a] = __bfloat162float(zrow[lane + 32 * a]);
        }
      } else if (lane == 0) {
        const float bb = __bfloat162float(p.ba[r * p.ldba + head]);
        const float x = __bfloat162float(p.ba[r * p.ldba + p.Hv + head]) + dtb;
        const float softplus = x > 20.f ? x : log1pf(__expf(x));
        coef[j].x = 1.f / (1.f + __expf(-bb));
        coef[j].y = __expf(neg_exp_a * softplus);
      }
    }
    __syncthreads();
    // ---- B: the recurrence.  The read-out is taken from the decayed state, S q = S' q + (k . q) delta, so that a token has one
    // reduction over the eight lanes instead of two; fp32 arithmetic two at a time
    for (int j = 0; j < nb; ++j) {
      const float4 co = coef[j];
      const float2 decay = make_float2(co.y, co.y);
      float4 kv[4], qv[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        kv[c] = *reinterpret_cast<const float4*>(&ks[j][4 * (l8 + 8 * c)]);
        qv[c] = *reinterpret_cast<const float4*>(&qs[j][4 * (l8 + 8 * c)]);
      }
      float mem[4], o[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float2 m = make_float2(0.f, 0.f), a = m;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          S[i][c][0] = __fmul2_rn(S[i][c][0], decay);
          S[i][c][1] = __fmul2_rn(S[i][c][1], decay);
          m = __ffma2_rn(S[i][c][0], make_float2(kv[c].x, kv[c].y), m);
          a = __ffma2_rn(S[i][c][0], make_float2(qv[c].x, qv[c].y), a);
          m = __ffma2_rn(S[i][c][1], make_float2(kv[c].z, kv[c].w), m);
          a = __ffma2_rn(S[i][c][1], make_float2(qv[c].z, qv[c].w), a);
        }
        mem[i] = m.x + m.y;
        o[i] = a.x + a.y;
      }
#pragma unroll
      for (int sh = 1; sh < 8; sh <<= 1)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          mem[i] += __shfl_xor_sync(0xffffffffu, mem[i], sh);
          o[i] += __shfl_xor_sync(0xffffffffu, o[i], sh);
        }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float delta = (vs[j][vrow + 4 * i] - mem[i]) * co.x;
        const float2 d = make_float2(delta, delta);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          S[i][c][0] = __ffma2_rn(d, make_float2(kv[c].x, kv[c].y), S[i][c][0]);
          S[i][c][1] = __ffma2_rn(d, make_float2(kv[c].z, kv[c].w), S[i][c][1]);
        }
        if (l8 == 0) os[j][vrow + 4 * i] = __bfloat162float(__float2bfloat16(fmaf(delta, co.z, o[i])));   // stored in bf16
      }
    }
    __syncthreads();
    // ---- C: gated RMSNorm over each token's 128 outputs
    for (int j = warp; j < nb; j += 8) {
      const size_t r = static_cast<size_t>(row0 + t0 + j);
      float ob[4];
      float ss = 0.f;
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        ob[a] = os[j][lane + 32 * a];
        ss = fmaf(ob[a], ob[a], ss);
      }
      const float inv = rsqrtf(warp_sum(ss) * (1.f / kGdnDim) + p.eps_norm);
      __nv_bfloat16* orow = p.out + r * p.ldo + head * kGdnDim;
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const float normed = __bfloat162float(__float2bfloat16(ob[a] * inv));
        orow[lane + 32 * a] = __float2bfloat16(normed * nw[a] * silu_fast(zs[j][lane + 32 * a]));
      }
    }
    // (the next block's phase A writes q / k / v / z: z of this block is still being read here, hence the barrier)
    if (t0 + kGdnBlock < n) __syncthreads();
  }
  if (!p.commit) return;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) 
      *reinterpret_cast<float4*>(sp + (4 * i) * kGdnDim + 32 * c) = make_float4(S[i][c][0].x, S[i][c][0].y, S[i][c][1].x, S[i][c][1].y);
}

// ------------------------------------------------------------------------------------------------- chunks of long segments
// The recurrence above has one token after the other: about 1900 cycles each, whatever the machine has idle.  Segments of kGdnChunk tokens and
// more are taken in chunks of 32 on the tensor cores.  With G the running product of the decays of a chunk and S its state at the start,
//     Delta = (I + L)^-1 beta (V - G K S^T),   L[t][s] = beta_t G_t / G_s (k_t . k_s) for s < t
//     o_t = G_t S q_t + sum over s <= t of G_t / G_s (q_t . k_s) Delta_s,      S <- G_end S + sum of G_end / G_s Delta_s k_s^T
// so that a chunk's chain is a dozen dependent products instead of 32 reductions.  (I + L)^-1 is taken by blocks of 16 tokens: the two blocks on the
// diagonal are inverted, the one below them is applied between.
//
// A value row (a row of S, a column of V, Delta and o) never meets another before the output norm: a warp holds 16 rows of S in registers and
// walks the chunk alone, everything transposed ([value row][token]), so that a product's accumulators are the next one's A operand
// without a shuffle.  Operands are f16: normalised k and q, bf16 of at most one, behind 2^15 (all bits down to 2^-32); what is computed in fp32 (S, Delta, L, the inverses, q . k) is
// split in two f16 behind a power of two that puts the largest of its value row at 2^13 (22 bits); Delta as it enters the state in three.  Sums with what is
// larger than the product (inverse less one, decayed state) are fp32 multiply-adds outside the tensor cores, which cut their sums off.
// Decay ratios are products of their factors, as in the recurrence: no logarithm, no quotient; they, and Delta on its way into the state, carry what a
// rounding leaves over.
// Against 64 bits, the recurrence -> this (relative error of the state; outputs, rounded to bf16, 2.9e-3 either way): random decays 0.74 -> 0.60e-7 (32 rows), 0.72 -> 0.63e-7
// (331), slow ones 13.1 -> 12.0e-7 (1000; the decays themselves), none 2.9 -> 1.4e-7 (640) and with values 2^-24 to 1 of each other 2.7 -> 1.3e-7 (320).  It grows faster with the
// likeness of a chunk's keys, as Delta is the product with an inverse: a mean cosine of 0.84 without decay 4.0 -> 2.9e-7, with random decays 0.77 -> 0.79e-7, of 0.99 without
// decay 3.9 -> 5.2e-7 (keys of random projections behind the convolution: 0.11).
//
// A CTA is a head of a segment: warps 0-7 walk the chunks, warps 8-15 prepare the next chunk's operands and norm and store the last one's outputs
// meanwhile.
// What bounds it: the chain of a chunk (6.9 us at 1.9 GHz, about 13000 cycles, of which its MMAs take 3500) and its preparation, which takes as long beside it.
// One row after the other -> in chunks, 32 heads, one B200: segments of 1000, 536, 823, 359 and 646 rows 1013 -> 254 us, one of 1750 924 -> 382, one of 331
// 307 -> 93, one of 32 34 -> 28, 16 of 256 1040 -> 254.
// A chunk with a key, query, value or coefficient that is not finite is walked token by token: zero times it, in a row before it, is not zero.  Likewise, by
// a warp for itself, one whose state or Delta is not.
static constexpr int kGdnChunk = 32;
static constexpr int kGdnChunkThreads = 512, kGdnPrepareThreads = 256;
// registers a thread: at launch, and of the walking and the preparing warps after they have shared them out anew
static constexpr int kGdnRegs = 128, kGdnRegsWalk = 184, kGdnRegsPrepare = 72;
static_assert(2 * kGdnRegsWalk + 2 * kGdnRegsPrepare <= 4 * kGdnRegs, "four warpgroups");
struct GdnOperands {
  uint8_t q[kGdnChunk * 256], k[kGdnChunk * 256];        // f16 [token][128], 16-byte chunk ^ (token & 7)
  __half inv[2][2][16 * 16];                             // [block][hi, lo] inverses of the blocks on the diagonal, less one
  __half l10[2][16 * 16];                                // [hi, lo] block of L below the diagonal
  __half a[3][2][16 * 16];                               // [block 00, 10, 11][hi, lo] q . k with ratios
  float4 coef[kGdnChunk];                                // beta_t, G_t, G_end / G_t, decay
  __nv_bfloat16 o[kGdnChunk][kGdnDim];
  float squares[8][kGdnChunk];                           // [warp][token]
  int wild;
};
struct __align__(128) GdnChunkSmem {
  GdnOperands op[2];                                     // [parity of the chunk]
  __nv_bfloat16 raw[2][kGdnChunk * kGdnDim];             // next chunk: q, k
  __nv_bfloat16 v[3][kGdnChunk * kGdnDim];               // chunk modulo 3
  float ratio[kGdnChunk][kGdnChunk];                     // [t][s] G_t / G_s, s <= t
  float low[2][16][16];                                  // blocks on the diagonal of L
};
static constexpr float kGdnUp = 4096.f;                  // of L, the inverses and q . k: entries of at most about one
static constexpr float kGdnKeyUp = 32768.f;              // of normalised q and k: elements of at most one, with all bits of bf16 down to 2^-32
static constexpr float kGdnKeyDown = 1.f / kGdnKeyUp;

template <int kThreads>
__device__ __forceinline__ void gdn_bar_sync(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(kThreads) : "memory"); }
template <int kThreads>
__device__ __forceinline__ void gdn_bar_arrive(int id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(kThreads) : "memory"); }

// Two rows of 16 f16 a 16-byte chunk apart would meet in a bank: chunk ^ (row >> 2 & 1).
__device__ __forceinline__ int gdn_at16(int row, int col) { return row * 16 + ((((col >> 3) ^ (row >> 2)) & 1) << 3) + (col & 7); }

__device__ __forceinline__ void gdn_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t gdn_pack(float x, float y) {
  const __half2 h = __floats2half2_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ void gdn_split(float x, float y, uint32_t& hi, uint32_t& lo) {
  hi = gdn_pack(x, y);
  const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&hi));
  lo = gdn_pack(x - h.x, y - h.y);
}
__device__ __forceinline__ float gdn_pow2(int e) { return __int_as_float((e + 127) << 23); }
__device__ __forceinline__ uint32_t gdn_bits(float x) { return __float_as_uint(x) & 0x7FFFFFFFu; }
// The largest magnitudes, as bits, of the value rows g and g + 8 of the warp's fragments (`most`: what the thread has of them): the four lanes of a row
__device__ __forceinline__ void gdn_row_max(uint32_t (&most)[2]) {
#pragma unroll
  for (int o = 1; o < 4; o <<= 1)
#pragma unroll
    for (int r = 0; r < 2; ++r) most[r] = max(most[r], __shfl_xor_sync(0xffffffffu, most[r], o));
}
// Its exponent; 0 and small ones count as 2^-85
__device__ __forceinline__ int gdn_exponent(uint32_t magnitude) { return max(static_cast<int>(magnitude >> 23) - 127, -85); }
// Accumulators of 16 value rows x 16 tokens (two n-tiles) -> the A operand over those tokens, each row times its 2^(13 - e); down: 2^(e - 13) of the rows
__device__ __forceinline__ void gdn_operand(const float (&x)[2][4], uint32_t (&hi)[4], uint32_t (&lo)[4], float (&down)[2]) {
  uint32_t most[2];
  float up[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) most[r] = max(max(gdn_bits(x[0][2 * r]), gdn_bits(x[0][2 * r + 1])), max(gdn_bits(x[1][2 * r]), gdn_bits(x[1][2 * r + 1])));
  gdn_row_max(most);
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int e = gdn_exponent(most[r]);
    up[r] = gdn_pow2(13 - e);
    down[r] = gdn_pow2(e - 13);
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int r = 0; r < 2; ++r) gdn_split(x[j][2 * r] * up[r], x[j][2 * r + 1] * up[r], hi[2 * j + r], lo[2 * j + r]);
}
// d[n-tile] = x (hi, lo) times a block of 16 x 16 (hi, lo), [column token][row token]
__device__ __forceinline__ void gdn_block(float (&d)[2][4], const uint32_t (&hi)[4], const uint32_t (&lo)[4], const __half (&m)[2][16 * 16], int lane) {
  uint32_t bh[4], bl[4];
  const int row = (lane & 7) + ((lane >> 4) << 3), col = ((lane >> 3) & 1) << 3;      // matrices: (n 0, k 0) (n 0, k 8) (n 8, k 0) (n 8, k 8)
  ldsm4(bh, smem_u32(&m[0][gdn_at16(row, col)]));
  ldsm4(bl, smem_u32(&m[1][gdn_at16(row, col)]));
#pragma unroll
  for (int j = 0; j < 2; ++j) {
#pragma unroll
    for (int i = 0; i < 4; ++i) d[j][i] = 0.f;
    gdn_mma(d[j], lo, bh[2 * j], bh[2 * j + 1]);
    gdn_mma(d[j], hi, bl[2 * j], bl[2 * j + 1]);
    gdn_mma(d[j], hi, bh[2 * j], bh[2 * j + 1]);
  }
}

// grid (Hv, segments).  Named barriers: 1 + parity: a chunk's operands are there; 3 + parity: it has been walked; 5: among the preparing warps.
__global__ void __launch_bounds__(kGdnChunkThreads, 1)
gdn_delta_chunk_kernel(const GdnDeltaParams p) {
  pdl_wait();
  pdl_launch_dependents();
  extern __shared__ __align__(128) uint8_t gdn_smem[];
  GdnChunkSmem& sm = *reinterpret_cast<GdnChunkSmem*>(gdn_smem);
  const int head = blockIdx.x, s = blockIdx.y;
  const int n = p.seg.count[s];
  if (n < kGdnChunk) return;
  const int row0 = p.seg.row0[s], chunks = (n + kGdnChunk - 1) / kGdnChunk;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kGdnRegsPrepare));
    constexpr int kTokens = kGdnChunk / 8;               // tokens of a warp
    const int tid = threadIdx.x & 255, w = warp - 8;
    const int khead = head / (p.Hv / p.Hk);
    const __nv_bfloat16* qg = p.qkv + khead * kGdnDim;
    const __nv_bfloat16* kg = p.qkv + (p.Hk + khead) * kGdnDim;
    const __nv_bfloat16* vg = p.qkv + (2 * p.Hk + head) * kGdnDim;
    const float neg_exp_a = -__expf(p.a_log[head]), dtb = p.dt_bias[head];
    const float4 nw = make_float4(p.norm_w[4 * lane], p.norm_w[4 * lane + 1], p.norm_w[4 * lane + 2], p.norm_w[4 * lane + 3]);
    __nv_bfloat16 bb = __float2bfloat16(0.f), aa = bb;   // b and a of token `lane` of the chunk to be prepared
    auto fetch = [&](int i) {                            // rows past the segment's become zeros
      const int t0 = i * kGdnChunk;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int t = j * 16 + (tid >> 4), col = (tid & 15) * 8;
        const bool in = t0 + t < n;
        const size_t r = static_cast<size_t>(row0 + (in ? t0 + t : 0)) * p.ldqkv + col;
        cp_async16(smem_u32(&sm.raw[0][t * kGdnDim + col]), qg + r, in);
        cp_async16(smem_u32(&sm.raw[1][t * kGdnDim + col]), kg + r, in);
        cp_async16(smem_u32(&sm.v[i % 3][t * kGdnDim + col]), vg + r, in);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      if (t0 + lane < n) {
        const size_t r = static_cast<size_t>(row0 + t0 + lane) * p.ldba + head;
        bb = p.ba[r];
        aa = p.ba[r + p.Hv];
      }
    };
    fetch(0);
    for (int i = 0; i < chunks + 2; ++i) {
      GdnOperands& op = sm.op[i & 1];
      if (i >= 2) {
        // ---- gated RMSNorm of chunk i - 2: a lane has four value rows
        const int t0 = (i - 2) * kGdnChunk + w * kTokens, here = min(n - t0, kTokens);
        uint2 z[kTokens];
#pragma unroll
        for (int j = 0; j < kTokens; ++j) {
          z[j] = make_uint2(0u, 0u);
          if (j < here) z[j] = *reinterpret_cast<const uint2*>(p.z + static_cast<size_t>(row0 + t0 + j) * p.ldz + head * kGdnDim + 4 * lane);
        }
        gdn_bar_sync<kGdnChunkThreads>(3 + (i & 1));
        float ss = op.squares[lane >> 2][w * kTokens + (lane & 3)];                       // lane = warp, token
#pragma unroll
        for (int sh = 4; sh < 32; sh <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, sh);
        const float norm = rsqrtf(ss * (1.f / kGdnDim) + p.eps_norm);
#pragma unroll
        for (int j = 0; j < kTokens; ++j) {
          const float inv = __shfl_sync(0xffffffffu, norm, j);
          const uint2 x = *reinterpret_cast<const uint2*>(&op.o[w * kTokens + j][4 * lane]);
          auto gated = [&](uint32_t ow, uint32_t zw, float w0, float w1) {
            const float2 ob = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ow)), zz = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&zw));
            const uint32_t nb = pack_bf16x2(ob.x * inv, ob.y * inv);
            const float2 normed = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&nb));
            return pack_bf16x2(normed.x * w0 * silu_fast(zz.x), normed.y * w1 * silu_fast(zz.y));
          };
          if (j < here)
            *reinterpret_cast<uint2*>(p.out + static_cast<size_t>(row0 + t0 + j) * p.ldo + head * kGdnDim + 4 * lane) = make_uint2(gated(x.x, z[j].x, nw.x, nw.y), gated(x.y, z[j].y, nw.z, nw.w));
        }
      }
      if (i >= chunks) continue;
      float beta = 0.f, decay = 1.f;                     // of token `lane`: every warp has them
      if (i * kGdnChunk + lane < n) {
        const float x = __bfloat162float(aa) + dtb;
        const float softplus = x > 20.f ? x : log1pf(__expf(x));
        beta = 1.f / (1.f + __expf(-__bfloat162float(bb)));
        decay = __expf(neg_exp_a * softplus);
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      if (tid == 0) op.wild = 0;
      gdn_bar_sync<kGdnPrepareThreads>(5);
      // ---- operands: normalised q and k (rounded to bf16 as the oracle stores them) in f16; a lane has four channels of the warp's tokens
      bool wild = !(fabsf(beta) < INFINITY) || !(fabsf(decay) < INFINITY);
      {
        constexpr int kRows = 2 * kTokens;               // q and k of every token
        uint2 x[kRows];
        float sum[kRows];
#pragma unroll
        for (int j = 0; j < kRows; ++j) x[j] = *reinterpret_cast<const uint2*>(&sm.raw[j & 1][(w * kTokens + (j >> 1)) * kGdnDim + 4 * lane]);
#pragma unroll
        for (int j = 0; j < kRows; ++j) {
          const float2 f0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x[j].x)), f1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x[j].y));
          sum[j] = fmaf(f0.x, f0.x, f0.y * f0.y) + fmaf(f1.x, f1.x, f1.y * f1.y);
        }
        // the sums over the warp, dealt to the lanes: half of them stay with each half of the lanes, three times
#pragma unroll
        for (int m = kRows / 2, o = 16; m >= 1; m >>= 1, o >>= 1)
#pragma unroll
          for (int j = 0; j < m; ++j) {
            const bool upper = lane & o;
            const float send = upper ? sum[j] : sum[j + m], keep = upper ? sum[j + m] : sum[j];
            sum[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
          }
        sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], 2);
        sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], 1);
        wild |= !(sum[0] < INFINITY);                    // an element that is not finite, or too large for its square
        const float inv = rsqrtf(sum[0] + p.eps_l2);
#pragma unroll
        for (int j = 0; j < kRows; ++j) {
          const float f = __shfl_sync(0xffffffffu, inv, 4 * j);
          auto norm = [&](uint32_t v) {
            const float2 e = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v));
            const uint32_t nb = pack_bf16x2(e.x * f, e.y * f);
            const float2 r = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&nb));
            return gdn_pack(r.x * kGdnKeyUp, r.y * kGdnKeyUp);
          };
          const int t = w * kTokens + (j >> 1);
          *reinterpret_cast<uint2*>((j & 1 ? op.k : op.q) + t * 256 + (((lane >> 1) ^ (t & 7)) << 4) + (lane & 1) * 8) = make_uint2(norm(x[j].x), norm(x[j].y));
        }
      }
      {
        uint32_t top = 0;                                // an exponent of all ones overflows into the sign's place
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint4 x = reinterpret_cast<const uint4*>(sm.v[i % 3])[j * 256 + tid];
          top |= ((x.x & 0x7F807F80u) + 0x00800080u) | ((x.y & 0x7F807F80u) + 0x00800080u) | ((x.z & 0x7F807F80u) + 0x00800080u) | ((x.w & 0x7F807F80u) + 0x00800080u);
        }
        wild |= (top & 0x80008000u) != 0;
      }
      if (__any_sync(0xffffffffu, wild) && lane == 0) op.wild = 1;
      // ---- ratios of the decays, lane = s: the products behind token s up to the warp's first token, and a decay more for each of its others.  With what the
      // products leave over (in doubles the chunk took 7 % longer)
      {
        float r = lane <= w * kTokens ? decay : 1.f, rest = 0.f;
        auto times = [](float& x, float& x_rest, float y, float y_rest) {
          const float z = x * y;
          x_rest = fmaf(x, y_rest, fmaf(x_rest, y, fmaf(x, y, -z)));
          x = z;
        };
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const float x = __shfl_down_sync(0xffffffffu, r, o), y = __shfl_down_sync(0xffffffffu, rest, o);
          if (lane + o < 32) times(r, rest, x, y);
        }
        r = __shfl_down_sync(0xffffffffu, r, 1);
        rest = __shfl_down_sync(0xffffffffu, rest, 1);
#pragma unroll
        for (int j = 0; j < kTokens; ++j) {
          const int t = w * kTokens + j;
          if (j > 0) times(r, rest, __shfl_sync(0xffffffffu, decay, t), 0.f);
          if (lane == t) {
            r = 1.f;
            rest = 0.f;
          }
          sm.ratio[t][lane] = lane <= t ? r + rest : 0.f;
        }
        if (w == 7) op.coef[lane].z = r + rest;
        if (w == 6) {
          float G = decay, G_rest = 0.f;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const float x = __shfl_up_sync(0xffffffffu, G, o), y = __shfl_up_sync(0xffffffffu, G_rest, o);
            if (lane >= o) times(G, G_rest, x, y);
          }
          op.coef[lane].x = beta;
          op.coef[lane].y = G + G_rest;
          op.coef[lane].w = decay;
        }
      }
      gdn_bar_sync<kGdnPrepareThreads>(5);
      if (i + 1 < chunks) fetch(i + 1);
      // ---- k . k and q . k of the chunk: three blocks x (k, q) x two n-tiles of keys; k . k of the blocks on the diagonal first
      for (int task = w; task < 12; task += 8) {
        const int is_q = task >= 6, in = is_q ? task - 6 : task, nt = in & 1, blk = (in >> 1) == 0 ? 0 : (in >> 1) == 1 ? 2 : 1, tb = blk > 0, sb = blk > 1;
        const uint32_t abase = smem_u32(is_q ? op.q : op.k) + (tb * 16 + (lane & 15)) * 256, bbase = smem_u32(op.k) + (sb * 16 + nt * 8 + (lane & 7)) * 256;
        float d[2][4] = {};
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
          uint32_t a0[4], a1[4], b[4];
          ldsm4(a0, abase + (((2 * k + (lane >> 4)) ^ (lane & 7)) << 4));
          ldsm4(a1, abase + (((2 * k + 2 + (lane >> 4)) ^ (lane & 7)) << 4));
          ldsm4(b, bbase + (((2 * k + (lane >> 3)) ^ (lane & 7)) << 4));
          gdn_mma(d[0], a0, b[0], b[1]);
          gdn_mma(d[1], a1, b[2], b[3]);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int tr = g + 8 * h, t = tb * 16 + tr, sc = nt * 8 + 2 * c;
          const float2 ratio = *reinterpret_cast<const float2*>(&sm.ratio[t][sb * 16 + sc]);
          constexpr float down = kGdnKeyDown * kGdnKeyDown;
          float x = (d[0][2 * h] + d[1][2 * h]) * down * ratio.x, y = (d[0][2 * h + 1] + d[1][2 * h + 1]) * down * ratio.y;
          const float bt = __shfl_sync(0xffffffffu, beta, t);
          if (!is_q) {
            x *= bt;
            y *= bt;
            if (blk != 1) {
              *reinterpret_cast<float2*>(&sm.low[sb][tr][sc]) = make_float2(x, y);        // what is not below the diagonal is not read
              continue;
            }
          }
          uint32_t hi, lo;
          gdn_split(x * kGdnUp, y * kGdnUp, hi, lo);
          __half (&to)[2][16 * 16] = is_q ? op.a[blk] : op.l10;
          *reinterpret_cast<uint32_t*>(&to[0][gdn_at16(tr, sc)]) = hi;
          *reinterpret_cast<uint32_t*>(&to[1][gdn_at16(tr, sc)]) = lo;
        }
      }
      gdn_bar_sync<kGdnPrepareThreads>(5);
      // ---- one warp inverts the blocks on the diagonal: their four 8 x 8 blocks on the diagonal, lane = block, column, then what is left of each,
      // -inverse x block x inverse
      if (w == 7) {
        {
          const int o = (lane >> 3 & 1) * 8, col = lane & 7;
          float (&m)[16][16] = sm.low[lane >> 4];
          float x[8];
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            float l[8];
#pragma unroll
            for (int j = 0; j < r; j += 4) *reinterpret_cast<float4*>(l + j) = *reinterpret_cast<const float4*>(&m[o + r][o + j]);
            float acc = r == col ? 1.f : 0.f, acc2 = 0.f;
#pragma unroll
            for (int j = 0; j < r; j += 2) {
              acc = fmaf(-l[j], x[j], acc);
              if (j + 1 < r) acc2 = fmaf(-l[j + 1], x[j + 1], acc2);
            }
            x[r] = acc + acc2;
          }
          __syncwarp();
#pragma unroll
          for (int r = 0; r < 8; ++r) m[o + r][o + col] = x[r];
          __syncwarp();
        }
        const int blk = lane >> 4, row = lane >> 1 & 7, half = (lane & 1) * 4;      // a lane has four columns of a row of the lower left block
        float (&m)[16][16] = sm.low[blk];
        auto times = [&](const float (&left)[8], int top, int first) {              // left . m[top + ..][first + half ..]
          float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 y = *reinterpret_cast<const float4*>(&m[top + j][first + half]);
            acc = make_float4(fmaf(left[j], y.x, acc.x), fmaf(left[j], y.y, acc.y), fmaf(left[j], y.z, acc.z), fmaf(left[j], y.w, acc.w));
          }
          return acc;
        };
        float left[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) left[j] = m[8 + row][j];
        const float4 lt = times(left, 0, 0);
        __syncwarp();
        *reinterpret_cast<float4*>(&m[8 + row][half]) = lt;
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; ++j) left[j] = m[8 + row][8 + j];
        const float4 t = times(left, 8, 0);
        __syncwarp();
        auto put = [&](int r, int col, float x, float y) {
          uint32_t hi, lo;
          gdn_split(x * kGdnUp, y * kGdnUp, hi, lo);
          *reinterpret_cast<uint32_t*>(&op.inv[blk][0][gdn_at16(r, col)]) = hi;
          *reinterpret_cast<uint32_t*>(&op.inv[blk][1][gdn_at16(r, col)]) = lo;
        };
        put(8 + row, half, -t.x, -t.y);
        put(8 + row, half + 2, -t.z, -t.w);
#pragma unroll
        for (int q = 0; q < 2; ++q) {                    // the blocks on the diagonal, less one, and the zeros beside them
          const int r = q * 8 + row;
#pragma unroll
          for (int j = 0; j < 4; j += 2) {
            const int cl = half + j;
            put(r, q * 8 + cl, row > cl ? m[r][q * 8 + cl] : 0.f, row > cl + 1 ? m[r][q * 8 + cl + 1] : 0.f);
            if (q == 0) put(r, 8 + cl, 0.f, 0.f);
          }
        }
      }
      gdn_bar_arrive<kGdnChunkThreads>(1 + (i & 1));
    }
    return;
  }
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kGdnRegsWalk));
  float* sp = p.state + ((static_cast<size_t>(p.seg.slot[s]) * p.Hv + head) * kGdnDim + warp * 16 + g) * kGdnDim + 2 * c;
  float S[16][4];                                        // [8 key columns][rows g: 2 c, 2 c + 1; rows g + 8: the same]
  const bool resumed = p.seg.pos0[s] > 0;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    float2 x = make_float2(0.f, 0.f), y = x;
    if (resumed) {
      x = *reinterpret_cast<const float2*>(sp + 8 * j);
      y = *reinterpret_cast<const float2*>(sp + 8 * kGdnDim + 8 * j);
    }
    S[j][0] = x.x; S[j][1] = x.y; S[j][2] = y.x; S[j][3] = y.y;
  }
  for (int i = 0; i < chunks; ++i) {
    GdnOperands& op = sm.op[i & 1];
    const __nv_bfloat16* vs = sm.v[i % 3] + warp * 16 + g;
    float o[2][2][4];                                    // [16 tokens][n-tile][value rows g, g + 8 x tokens 2 c, 2 c + 1], without 1 / sqrt(d_k)
    gdn_bar_sync<kGdnChunkThreads>(1 + (i & 1));
    uint32_t most[2] = {0, 0};
#pragma unroll
    for (int j = 0; j < 16; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) most[q >> 1] = max(most[q >> 1], gdn_bits(S[j][q]));
    gdn_row_max(most);
    // what is not finite in the warp's rows of the state, or in what the chunk adds to them, is walked with too
    bool walk = op.wild || __any_sync(0xffffffffu, max(most[0], most[1]) >= 0x7F800000u);
    if (!walk) {
      // ---- S k and S q
      constexpr float kToGrid = 1.5f * 8589934592.f;     // added and subtracted: multiples of 2^10
      float u[2][2][4], rest[2][2][4];                   // u + rest is Delta, when all is done
      float down[2];
      {
        float x[2][2][4], up[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int e = gdn_exponent(most[r]);
          up[r] = gdn_pow2(13 - e);
          down[r] = gdn_pow2(e - 13) * kGdnKeyDown;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) u[h][j][q] = o[h][j][q] = x[h][j][q] = 0.f;
        const int brow = (lane & 7) + ((lane >> 4) << 3);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int r = 0; r < 4; ++r) gdn_split(S[2 * k + (r >> 1)][2 * (r & 1)] * up[r & 1], S[2 * k + (r >> 1)][2 * (r & 1) + 1] * up[r & 1], hi[r], lo[r]);
          const uint32_t at = brow * 256 + (((2 * k + ((lane >> 3) & 1)) ^ (lane & 7)) << 4);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t bk[4], bq[4];
            ldsm4(bk, smem_u32(op.k) + at + h * 16 * 256);
            ldsm4(bq, smem_u32(op.q) + at + h * 16 * 256);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              gdn_mma(x[h][j], lo, bk[2 * j], bk[2 * j + 1]);
              gdn_mma(o[h][j], lo, bq[2 * j], bq[2 * j + 1]);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              gdn_mma(x[h][j], hi, bk[2 * j], bk[2 * j + 1]);
              gdn_mma(o[h][j], hi, bq[2 * j], bq[2 * j + 1]);
            }
            if (k & 1) {                                 // the tensor cores cut their sums off: short ones, added here
#pragma unroll
              for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                  u[h][j][r] += x[h][j][r];
                  x[h][j][r] = 0.f;
                }
            }
          }
        }
      }
      // ---- beta (v - G S k), G S q
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int t = h * 16 + j * 8 + 2 * c + q;
            const float2 bg = *reinterpret_cast<const float2*>(&op.coef[t]);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const float f = down[r] * bg.y, x = fmaf(-u[h][j][2 * r + q], f, __bfloat162float(vs[t * kGdnDim + 8 * r])), y = x * bg.x;
              u[h][j][2 * r + q] = y;
              rest[h][j][2 * r + q] = fmaf(x, bg.x, -y);
              o[h][j][2 * r + q] *= f;
            }
          }
      // ---- Delta (u + rest) of tokens 0..15, then of 16..31: what is smaller is added up beside u, so that u is rounded once
      uint32_t hi[4], lo[4];
      float d[2][4], f[2];
      auto add = [&](float (&x)[2][4], float sign) {     // x += d
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int q = 0; q < 4; ++q) x[j][q] = fmaf(sign * (1.f / kGdnUp) * f[q >> 1], d[j][q], x[j][q]);
      };
      auto sum = [&](float (&x)[2][4], float (&y)[2][4]) {                        // x + y in x, what that leaves over in y
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float z = x[j][q] + y[j][q], part = z - x[j][q];
            y[j][q] = (x[j][q] - (z - part)) + (y[j][q] - part);
            x[j][q] = z;
          }
      };
      gdn_operand(u[0], hi, lo, f);
      gdn_block(d, hi, lo, op.inv[0], lane);
      add(rest[0], 1.f);
      sum(u[0], rest[0]);
      gdn_operand(u[0], hi, lo, f);
      gdn_block(d, hi, lo, op.l10, lane);
      add(rest[1], -1.f);
      gdn_block(d, hi, lo, op.a[0], lane);
      add(o[0], 1.f);
      gdn_block(d, hi, lo, op.a[1], lane);
      add(o[1], 1.f);
      {
        float x[2][4];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int q = 0; q < 4; ++q) x[j][q] = u[1][j][q] + rest[1][j][q];
        gdn_operand(x, hi, lo, f);
      }
      gdn_block(d, hi, lo, op.inv[1], lane);
      add(rest[1], 1.f);
      sum(u[1], rest[1]);
      gdn_operand(u[1], hi, lo, f);
      gdn_block(d, hi, lo, op.a[2], lane);
      add(o[1], 1.f);
      // ---- the state: G_end S plus the products of the chunk, which the tensor cores sum from zero
      const float end = op.coef[kGdnChunk - 1].y;
      uint32_t first[2][4], second[2][4], third[2][4];
      most[0] = most[1] = 0;
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float r0 = op.coef[b * 16 + j * 8 + 2 * c].z, r1 = op.coef[b * 16 + j * 8 + 2 * c + 1].z;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float r = q & 1 ? r1 : r0, x = u[b][j][q] * r;
            rest[b][j][q] = fmaf(rest[b][j][q], r, fmaf(u[b][j][q], r, -x));
            u[b][j][q] = x;
            most[q >> 1] = max(most[q >> 1], gdn_bits(u[b][j][q]));
          }
        }
      gdn_row_max(most);
      walk = __any_sync(0xffffffffu, max(most[0], most[1]) >= 0x7F800000u);
      if (!walk) {
        float up[2], fs[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int e = gdn_exponent(most[r]);
          up[r] = gdn_pow2(13 - e);
          fs[r] = gdn_pow2(e - 13) * kGdnKeyDown;
        }
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const int at = 2 * j + r;
              float x = u[b][j][2 * r] * up[r], y = u[b][j][2 * r + 1] * up[r];
              const float xf = x + kToGrid - kToGrid, yf = y + kToGrid - kToGrid;
              first[b][at] = gdn_pack(xf, yf);
              x = x - xf + rest[b][j][2 * r] * up[r];
              y = y - yf + rest[b][j][2 * r + 1] * up[r];
              gdn_split(x, y, second[b][at], third[b][at]);
            }
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          uint32_t kb[2][4];                             // (tokens 0, columns 0) (tokens 8, columns 0) (tokens 0, columns 8) (tokens 8, columns 8)
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            const int t = b * 16 + (lane & 15);
            ldsm4_t(kb[b], smem_u32(op.k) + t * 256 + (((j + (lane >> 4)) ^ (t & 7)) << 4));
          }
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            // The tensor cores cut a sum off below its last bit, half a bit too small on average.  First parts are multiples of 2^10: their sums have no more
            // bits than fit, unless a key's element is below 2^-13; what is cut off the rest, 2^-4 of them, does not count.
            float x[4] = {0.f, 0.f, 0.f, 0.f}, y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int b = 0; b < 2; ++b) {
              gdn_mma(x, first[b], kb[b][2 * q], kb[b][2 * q + 1]);
              gdn_mma(y, third[b], kb[b][2 * q], kb[b][2 * q + 1]);
              gdn_mma(y, second[b], kb[b][2 * q], kb[b][2 * q + 1]);
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) S[j + q][r] = fmaf(fs[r >> 1], x[r], fmaf(fs[r >> 1], y[r], S[j + q][r] * end));
          }
        }
      }
    }
    if (walk) {
      // ---- token by token
#pragma unroll 1
      for (int t = 0; t < kGdnChunk; ++t) {
        const float4 co = op.coef[t];
        float m0 = 0.f, m1 = 0.f, r0 = 0.f, r1 = 0.f, kq = 0.f;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int at = t * 256 + ((j ^ (t & 7)) << 4) + c * 4;
          float2 k = __half22float2(*reinterpret_cast<const __half2*>(op.k + at)), q = __half22float2(*reinterpret_cast<const __half2*>(op.q + at));
          k.x *= kGdnKeyDown; k.y *= kGdnKeyDown;
          q.x *= kGdnKeyDown; q.y *= kGdnKeyDown;
#pragma unroll
          for (int i = 0; i < 4; ++i) S[j][i] *= co.w;
          m0 = fmaf(S[j][0], k.x, fmaf(S[j][1], k.y, m0));
          m1 = fmaf(S[j][2], k.x, fmaf(S[j][3], k.y, m1));
          r0 = fmaf(S[j][0], q.x, fmaf(S[j][1], q.y, r0));
          r1 = fmaf(S[j][2], q.x, fmaf(S[j][3], q.y, r1));
          kq = fmaf(k.x, q.x, fmaf(k.y, q.y, kq));
        }
#pragma unroll
        for (int sh = 1; sh < 4; sh <<= 1) {
          m0 += __shfl_xor_sync(0xffffffffu, m0, sh);
          m1 += __shfl_xor_sync(0xffffffffu, m1, sh);
          r0 += __shfl_xor_sync(0xffffffffu, r0, sh);
          r1 += __shfl_xor_sync(0xffffffffu, r1, sh);
          kq += __shfl_xor_sync(0xffffffffu, kq, sh);
        }
        const float d0 = (__bfloat162float(vs[t * kGdnDim]) - m0) * co.x, d1 = (__bfloat162float(vs[t * kGdnDim + 8]) - m1) * co.x;
        r0 = fmaf(d0, kq, r0);
        r1 = fmaf(d1, kq, r1);
        if (i * kGdnChunk + t < n) {                     // behind the segment's end nothing happens to the state
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            float2 k = __half22float2(*reinterpret_cast<const __half2*>(op.k + t * 256 + ((j ^ (t & 7)) << 4) + c * 4));
            k.x *= kGdnKeyDown; k.y *= kGdnKeyDown;
            S[j][0] = fmaf(d0, k.x, S[j][0]); S[j][1] = fmaf(d0, k.y, S[j][1]);
            S[j][2] = fmaf(d1, k.x, S[j][2]); S[j][3] = fmaf(d1, k.y, S[j][3]);
          }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int q = 0; q < 2; ++q)
              if (h * 16 + j * 8 + 2 * c + q == t) { o[h][j][q] = r0; o[h][j][2 + q] = r1; }
      }
    }
    // ---- outputs (stored in bf16 by the oracle) and the warp's sums of their squares
    float sq[2][2][2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int t = h * 16 + j * 8 + 2 * c + q;
          const __nv_bfloat16 x = __float2bfloat16(o[h][j][q] * 0.08838834764831845f), y = __float2bfloat16(o[h][j][2 + q] * 0.08838834764831845f);
          op.o[t][warp * 16 + g] = x;
          op.o[t][warp * 16 + g + 8] = y;
          const float xf = __bfloat162float(x), yf = __bfloat162float(y);
          sq[h][j][q] = fmaf(xf, xf, yf * yf);
        }
#pragma unroll
    for (int sh = 4; sh < 32; sh <<= 1)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int q = 0; q < 2; ++q) sq[h][j][q] += __shfl_xor_sync(0xffffffffu, sq[h][j][q], sh);
    if (g == 0) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < 2; ++j) *reinterpret_cast<float2*>(&op.squares[warp][h * 16 + j * 8 + 2 * c]) = make_float2(sq[h][j][0], sq[h][j][1]);
    }
    gdn_bar_arrive<kGdnChunkThreads>(3 + (i & 1));
  }
  if (!p.commit) return;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    *reinterpret_cast<float2*>(sp + 8 * j) = make_float2(S[j][0], S[j][1]);
    *reinterpret_cast<float2*>(sp + 8 * kGdnDim + 8 * j) = make_float2(S[j][2], S[j][3]);
  }
}

// out = x * sigmoid(gate): the output gate of the hybrid family's full-attention layers (bf16, in place allowed)
__global__ void __launch_bounds__(256)
sigmoid_gate_kernel(const __nv_bfloat16* __restrict__ x, int ldx, const __nv_bfloat16* __restrict__ gate, int ldg,
                    __nv_bfloat16* __restrict__ out, int ldo, int cols) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= (cols >> 1)) return;
  const size_t r = blockIdx.y;
  const float2 a = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(x + r * ldx)[v]);
  const float2 g = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(gate + r * ldg)[v]);
  reinterpret_cast<__nv_bfloat162*>(out + r * ldo)[v] =
      __floats2bfloat162_rn(a.x / (1.f + __expf(-g.x)), a.y / (1.f + __expf(-g.y)));
}

}  // namespace cb

extern "C" {

struct CbGdnSegments {
  const void* row0;
  const void* count;
  const void* slot;
  const void* pos0;
  int num;
};

// Whether the columns [0, C) of `rows` rows of x and of y share elements.
static bool conv_overlap(const void* x, int ldx, const void* y, int ldy, int C, int rows) {
  const long long a = static_cast<long long>(reinterpret_cast<uintptr_t>(x)), b = static_cast<long long>(reinterpret_cast<uintptr_t>(y)), cols = 2ll * C;
  const long long x_end = a + 2ll * (rows - 1) * ldx + cols, y_end = b + 2ll * (rows - 1) * ldy + cols;
  if (x_end <= b || y_end <= a) return false;
  if (ldx != ldy || ldx < C) return true;
  const long long pitch = 2ll * ldx, shift = ((b - a) % pitch + pitch) % pitch;       // neighbouring columns of one buffer
  return shift < cols || shift > pitch - cols;
}

// `rows`: rows of the step.  y may be x.
int cb_gdn_conv(const void* x, int ldx, void* y, int ldy, const void* w, const void* bias, void* state,
                const CbGdnSegments* seg, int C, int rows, int commit, void* stream) {
  if (!seg || seg->num <= 0 || C <= 0 || seg->num > 65535 || rows < 0) return -60;
  if (rows == 0) return 0;
  // A block a segment where the outputs overwrite the inputs, and where there are as many rows as segments (decode): the search for
  // the tile's segment, in up to eight rounds, made 256 one-row segments of 8192 channels 35 us instead of 27.
  const bool whole = rows == seg->num || conv_overlap(x, ldx, y, ldy, C, rows);
  const cb::Segments s{static_cast<const int*>(seg->row0), static_cast<const int*>(seg->count), static_cast<const int*>(seg->slot),
                       static_cast<const int*>(seg->pos0), seg->num, whole ? 1 : 0};
  int tile_rows = whole ? rows : cb::kConvRows;
  while (!whole && cb::max_tiles(rows, seg->num, tile_rows) > 65535) tile_rows = tile_rows > rows / 2 ? rows : 2 * tile_rows;     // at `rows` a tile a segment
  const int tiles = whole ? seg->num : cb::max_tiles(rows, seg->num, tile_rows);
  const bool pairs = C % 2 == 0 && ldx % 2 == 0 && ldy % 2 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(state)) & 3) == 0;
  const int cols = pairs ? 256 : 128;
  const dim3 grid((C + cols - 1) / cols, tiles);
  auto kernel = pairs ? cb::gdn_conv_kernel<2> : cb::gdn_conv_kernel<1>;
  kernel<<<grid, 128, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const __nv_bfloat16*>(x), ldx, static_cast<__nv_bfloat16*>(y), ldy,
                                                              static_cast<const float*>(w), static_cast<const float*>(bias),
                                                              static_cast<__nv_bfloat16*>(state), s, tile_rows, C, commit);
  return static_cast<int>(cudaGetLastError());
}

struct CbGdnDelta {
  const void* qkv; int ldqkv;
  const void* z; int ldz;
  const void* ba; int ldba;
  const void* a_log;
  const void* dt_bias;
  const void* norm_w;
  void* state;
  void* out; int ldo;
  int Hk, Hv;
  float eps_norm, eps_l2;
  int commit;
  int longest;      // rows of the longest segment, or a bound of them (the rows of the step)
};

int cb_gdn_delta(const CbGdnDelta* a, const CbGdnSegments* seg, void* stream) {
  if (!a || !seg || seg->num <= 0 || seg->num > 65535 || a->Hk <= 0 || a->Hv <= 0 || (a->Hv % a->Hk) != 0) return -61;
  cb::GdnDeltaParams p;
  p.qkv = static_cast<const __nv_bfloat16*>(a->qkv); p.ldqkv = a->ldqkv;
  p.z = static_cast<const __nv_bfloat16*>(a->z); p.ldz = a->ldz;
  p.ba = static_cast<const __nv_bfloat16*>(a->ba); p.ldba = a->ldba;
  p.a_log = static_cast<const float*>(a->a_log);
  p.dt_bias = static_cast<const float*>(a->dt_bias);
  p.norm_w = static_cast<const float*>(a->norm_w);
  p.state = static_cast<float*>(a->state);
  p.out = static_cast<__nv_bfloat16*>(a->out); p.ldo = a->ldo;
  p.Hk = a->Hk; p.Hv = a->Hv;
  p.eps_norm = a->eps_norm; p.eps_l2 = a->eps_l2;
  p.commit = a->commit;
  p.seg = cb::GdnSegments{static_cast<const int*>(seg->row0), static_cast<const int*>(seg->count),
                          static_cast<const int*>(seg->slot), static_cast<const int*>(seg->pos0)};
  // Segments of a chunk and more go to the kernel of chunks; what is shorter keeps the bits that its rows have one by one (speculative rounds).  The
  // chunks read rows in 16 bytes and write outputs and states in eight.
  auto aligned = [](const void* x, int ld, int bytes) { return (reinterpret_cast<uintptr_t>(x) | static_cast<uintptr_t>(2ll * ld)) % bytes == 0; };
  const bool chunks = a->longest >= cb::kGdnChunk && aligned(a->qkv, a->ldqkv, 16) && aligned(a->z, a->ldz, 8) && aligned(a->out, a->ldo, 8) && reinterpret_cast<uintptr_t>(a->state) % 8 == 0;
  p.most = chunks ? cb::kGdnChunk - 1 : INT_MAX;
  if (chunks) {
    static bool configured[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -18;
    if (!configured[dev]) {
      const cudaError_t e = cudaFuncSetAttribute(cb::gdn_delta_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(cb::GdnChunkSmem)));
      if (e != cudaSuccess) return static_cast<int>(e);
      // the warps' new shares come out of the registers that the block was launched with
      cudaFuncAttributes at;
      const cudaError_t e2 = cudaFuncGetAttributes(&at, cb::gdn_delta_chunk_kernel);
      if (e2 != cudaSuccess) return static_cast<int>(e2);
      if (at.numRegs < cb::kGdnRegs) return -19;
      configured[dev] = true;
    }
    const cudaError_t e = cb::launch(cb::gdn_delta_chunk_kernel, dim3(a->Hv, seg->num), dim3(cb::kGdnChunkThreads), sizeof(cb::GdnChunkSmem), static_cast<cudaStream_t>(stream), p);
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  dim3 grid(a->Hv, seg->num);
  cb::gdn_delta_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(p);
  return static_cast<int>(cudaGetLastError());
}

int cb_sigmoid_gate(const void* x, int ldx, const void* gate, int ldg, void* out, int ldo, int rows, int cols,
                    void* stream) {
  if (rows <= 0 || cols <= 0 || (cols & 1) || (ldx & 1) || (ldg & 1) || (ldo & 1)) return -62;
  for (int r0 = 0; r0 < rows; r0 += 65535) {
    const int nr = rows - r0 < 65535 ? rows - r0 : 65535;
    dim3 grid((cols / 2 + 255) / 256, nr);
    cb::sigmoid_gate_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16*>(x) + static_cast<size_t>(r0) * ldx, ldx,
        static_cast<const __nv_bfloat16*>(gate) + static_cast<size_t>(r0) * ldg, ldg,
        static_cast<__nv_bfloat16*>(out) + static_cast<size_t>(r0) * ldo, ldo, cols);
  }
  return static_cast<int>(cudaGetLastError());
}

}  // extern "C"
