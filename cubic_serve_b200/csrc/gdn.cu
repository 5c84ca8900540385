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
#include "ptx.cuh"
#include "segments.cuh"
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
  if (n <= 0) return;
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
