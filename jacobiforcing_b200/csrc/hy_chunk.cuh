// hy_chunk.cuh — matrix-state recurrences of prompt steps in chunks of 64 tokens (libjf_hybrid.so): the same recurrence as gla_kernel
// (hy_gla.cuh), S <- diag(a) S + k v^T, o = S^T q, without its chain of tokens.
//
// Token by token a head's state is a chain as long as the prompt, and a block has no more than its 16 columns to work on: 2048 tokens of 8 heads
// of 128 x 128 took 187 us on 64 of 148 SMs, about 170 cycles a token.  Within a chunk the recurrence is products of matrices:
//   state behind the chunk   S' = diag(a_0 .. a_63) S + sum_j (k_j a_j+1 .. a_63) v_j^T                       (gla_chunk_state_kernel)
//   read-outs                o_i = (q_i a_0 .. a_i)^T S + sum_(j <= i) (q_i . a_j+1 .. a_i . k_j) v_j           (gla_chunk_out_kernel)
// so the chunks' own sums are made side by side, the states at their beginnings follow element by element (gla_chunk_scan_kernel), and the
// read-outs again side by side.  All operands, sums and states are fp32 on the fp32 units, as they are token by token; decays are
// products of the given decays (no logarithms, no quotients: every factor is at most one and a decay of zero is just a zero).  Per
// channel they are applied in sub-blocks of 16: inside one, pair by pair; between two, as (q from the later one's beginning) . (whole
// sub-blocks between) . (k to the earlier one's end).
// A token's read-out and correction meet what came up to it and nothing behind it, not even times zero: an infinity or what is no number stays with
// the tokens from its own on, as it does token by token.
// Operands come from shared memory, 8 x 8 and 8 x 4 sums per thread; in turn the fma pipe (a third of the time) and the reads of shared memory (half of
// it) bound them, with two blocks of eight warps per SM.  2048 tokens, us, token by token -> chunks (three kernels): forget gates, 8
// heads of 128 x 128, 187 -> 72; state space, 32 heads of 64 x 128, 236 -> 140; two requests of gated linear attention, 16 heads of
// 128 x 128, 251 -> 137; five requests of retention, 8 heads, 118 -> 66.
#pragma once
#include "hy_gla.cuh"

namespace hy {

constexpr int CH_T = 64, CH_SUB = 16, CH_SUBS = CH_T / CH_SUB;
constexpr int CH_MAX_DIM = 128;

// The chunk'th chunk of a step's entries (entry by entry).
struct ChunkPlace {
  int e, index, t0, n;                                         // entry, its chunk, first row of the step, tokens
  __device__ ChunkPlace(const Batch& b, int chunk) {
    index = chunk;
    for (e = 0; e < b.E - 1; ++e) {
      const int nc = (b.ent_start[e + 1] - b.ent_start[e] + CH_T - 1) / CH_T;
      if (index < nc) break;
      index -= nc;
    }
    t0 = b.ent_start[e] + index * CH_T;
    n = min(CH_T, b.ent_start[e + 1] - t0);
  }
};

// Operands as gla_kernel's; states [chunk][H][DK / 2][DV][2]: a chunk's own sum, then the state at its beginning, two rows side by side so that
// the read-outs' products take pairs of rows without moving registers; ends [chunk][H][DK]: the product of a chunk's decays.
template <typename AT>
struct ChunkArgs {
  Batch b;
  const float* qk; const AT* v; int ldv;
  const float* decay; int ldd; const float* head_decay;
  int H, dim, vdim, vec, vvec, ovec;                           // 16-byte accesses: key rows and decays; value rows and the state; read-outs
  float* states; float* ends; float* state;
  float* o; int ldo;
  GlaToken tk;
};

// rows of n floats, `cols` of DK in use, to sw [64][DK] (chunks of 16 bytes xor the row's low bits with SWZ); the rest becomes `fill`
template <int DK, bool SWZ>
__device__ __forceinline__ int ch_at(int r, int c) { return r * DK + (SWZ ? (((c >> 2) ^ (r & 7)) << 2) + (c & 3) : c); }
template <int DK, bool SWZ>
__device__ __forceinline__ void ch_rows(float* dst, const float* src, size_t ld, int n, int cols, bool vec, float fill) {
  if (vec) {
    for (int i = threadIdx.x; i < CH_T * (DK / 4); i += 256) {
      const int r = i / (DK / 4), c = i % (DK / 4) * 4;
      float* d = dst + ch_at<DK, SWZ>(r, c);
      if (r < n && c < cols) jf::cp_async_16(d, src + (size_t)r * ld + c, 16u);
      else *reinterpret_cast<float4*>(d) = make_float4(fill, fill, fill, fill);
    }
  } else {
    for (int i = threadIdx.x; i < CH_T * DK; i += 256) {
      const int r = i / DK, c = i % DK;
      dst[ch_at<DK, SWZ>(r, c)] = r < n && c < cols ? src[(size_t)r * ld + c] : fill;
    }
  }
}
// A token's decay and the factor of its value, one number per head (GLA_HEAD, GLA_TOKEN).
template <typename AT, int MODE>
__device__ __forceinline__ void ch_scalars(const ChunkArgs<AT>& a, const ChunkPlace& p, int h, float* sa, float* sx) {
  if (threadIdx.x < CH_T) {
    const int t = threadIdx.x;
    float d = 1.0f, x = 1.0f;
    if (t < p.n) {
      if constexpr (MODE == GLA_HEAD) d = a.head_decay[h];
      else {
        x = softplus_f(to_f(((const AT*)a.tk.dt_raw)[(size_t)(p.t0 + t) * a.tk.lddt + h]) + a.tk.dt_bias[h]);
        d = expf(-expf(a.tk.A_log[h]) * x);
      }
    }
    sa[t] = d; sx[t] = x;
  }
}

template <int DK, int DV, int MODE>
__host__ __device__ constexpr size_t ch_state_smem() {
  return ((size_t)CH_T * DK + (MODE == GLA_CHANNEL ? (size_t)CH_T * DK : 0) + (size_t)CH_T * DV + CH_SUBS * DK + 3 * CH_T) * 4;
}

// A chunk's own sum and its decays' product.  grid (chunks, H), 256 threads, each DK / 16 x DV / 16 sums.
template <typename AT, int DK, int DV, int MODE>
__global__ void __launch_bounds__(256, 2) gla_chunk_state_kernel(ChunkArgs<AT> a) {
  pdl_begin();
  constexpr bool SCALAR = MODE == GLA_HEAD || MODE == GLA_TOKEN;
  constexpr int TD = DK / 16, TV = DV / 16;
  extern __shared__ __align__(16) unsigned char hy_smem[];
  float* sk = reinterpret_cast<float*>(hy_smem);               // [64][DK] keys (GLA_FORGET: decays first)
  float* sd = sk + CH_T * DK;                                  // [64][DK] decays (GLA_CHANNEL)
  float* sv = sd + (MODE == GLA_CHANNEL ? CH_T * DK : 0);      // [64][DV]
  float* se = sv + CH_T * DV;                                  // [4][DK] product of a sub-block's decays
  float* sa = se + CH_SUBS * DK;                               // [64] decay, [64] factor of the value
  const ChunkPlace p(a.b, blockIdx.x);
  const int h = blockIdx.y, tid = threadIdx.x;
  const int per = MODE == GLA_TOKEN ? a.tk.G : a.H, row = MODE == GLA_TOKEN ? h / (a.H / a.tk.G) : h;
  ch_rows<DK, false>(sk, a.qk + ((size_t)p.t0 * per + row) * 2 * a.dim + a.dim, (size_t)per * 2 * a.dim, p.n, a.dim, a.vec, MODE == GLA_FORGET ? 1.0f : 0.0f);
  if constexpr (MODE == GLA_CHANNEL) ch_rows<DK, false>(sd, a.decay + (size_t)p.t0 * a.ldd + h * a.dim, a.ldd, p.n, a.dim, a.vec, 1.0f);
  if constexpr (SCALAR) ch_scalars<AT, MODE>(a, p, h, sa, sa + CH_T);
  if (a.vvec) {
    for (int i = tid; i < CH_T * DV / 4; i += 256) {
      const int r = i / (DV / 4), c = i % (DV / 4) * 4;
      float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (r < p.n && c < a.vdim) {
        const VecN<AT, 4> v = *reinterpret_cast<const VecN<AT, 4>*>(a.v + (size_t)(p.t0 + r) * a.ldv + h * a.vdim + c);
        x = make_float4(to_f(v.v[0]), to_f(v.v[1]), to_f(v.v[2]), to_f(v.v[3]));
      }
      *reinterpret_cast<float4*>(sv + 4 * i) = x;
    }
  } else {
    for (int i = tid; i < CH_T * DV; i += 256) {
      const int r = i / DV, c = i % DV;
      sv[i] = r < p.n && c < a.vdim ? to_f(a.v[(size_t)(p.t0 + r) * a.ldv + h * a.vdim + c]) : 0.0f;
    }
  }
  jf::cp_async_wait_all();
  __syncthreads();
  // keys times the decays behind them in their sub-block, the sub-blocks' products
  for (int i = tid; i < CH_SUBS * DK; i += 256) {
    const int s = i / DK, d = i % DK;
    float w = 1.0f;
#pragma unroll
    for (int j = CH_SUB - 1; j >= 0; --j) {
      const int t = s * CH_SUB + j;
      float& k = sk[t * DK + d];
      if constexpr (MODE == GLA_FORGET) { const float f = k; k = (1.0f - f) * w; w *= f; }
      else if constexpr (MODE == GLA_CHANNEL) { k *= w; w *= sd[t * DK + d]; }
      else { k *= w * sa[CH_T + t]; w *= sa[t]; }
    }
    se[i] = w;
  }
  __syncthreads();
  const int tx = tid & 15, ty = tid >> 4;
  float2 acc[TD][TV / 2] = {};
  auto dcol = [&](int i) { return (i >> 2) * 64 + ty * 4 + (i & 3); };
#pragma unroll 1
  for (int s = 0; s < CH_SUBS; ++s) {
    if (s * CH_SUB >= p.n) {                                   // nothing behind the last token; its decays are ones
      break;
    }
    if (s > 0) {
#pragma unroll
      for (int i = 0; i < TD; ++i) {
        const float e = se[s * DK + dcol(i)];
#pragma unroll
        for (int c = 0; c < TV / 2; ++c) acc[i][c] = mul2(acc[i][c], make_float2(e, e));
      }
    }
#pragma unroll 4
    for (int j = s * CH_SUB; j < (s + 1) * CH_SUB; ++j) {
      float4 k[TD / 4], v[TV / 4];
#pragma unroll
      for (int i = 0; i < TD / 4; ++i) k[i] = *reinterpret_cast<const float4*>(sk + j * DK + i * 64 + ty * 4);
#pragma unroll
      for (int i = 0; i < TV / 4; ++i) v[i] = *reinterpret_cast<const float4*>(sv + j * DV + i * 64 + tx * 4);
#pragma unroll
      for (int i = 0; i < TD; ++i) {
        const float kk = reinterpret_cast<const float*>(k)[i];
#pragma unroll
        for (int c = 0; c < TV / 4; ++c) {
          acc[i][2 * c] = fma2(make_float2(kk, kk), make_float2(v[c].x, v[c].y), acc[i][2 * c]);
          acc[i][2 * c + 1] = fma2(make_float2(kk, kk), make_float2(v[c].z, v[c].w), acc[i][2 * c + 1]);
        }
      }
    }
  }
  const size_t at = (size_t)blockIdx.x * a.H + h;
  float* out = a.states + at * DK * DV;
#pragma unroll
  for (int i = 0; i < TD; i += 2)
#pragma unroll
    for (int c = 0; c < TV / 2; ++c)
      *reinterpret_cast<float4*>(out + (size_t)dcol(i) * DV + 2 * ((c >> 1) * 64 + tx * 4 + (c & 1) * 2)) =
          make_float4(acc[i][c].x, acc[i + 1][c].x, acc[i][c].y, acc[i + 1][c].y);
  if (tid < DK) {
    float e = 1.0f;
#pragma unroll
    for (int s = 0; s < CH_SUBS; ++s) e *= se[s * DK + tid];
    a.ends[at * DK + tid] = e;
  }
}

// The states at the chunks' beginnings in the place of the chunks' own sums, the last one to the slot.  grid (DK DV / 1024, H, entries), 256
// threads of two rows x two columns each; four chunks' sums are on their way at a time.
template <typename AT, int DK, int DV>
__global__ void __launch_bounds__(256) gla_chunk_scan_kernel(ChunkArgs<AT> a) {
  pdl_begin();
  const int e = blockIdx.z, h = blockIdx.y, i = (blockIdx.x * 256 + threadIdx.x) * 4, d = i / (2 * DV) * 2, c = i % (2 * DV) / 2;
  int c0 = 0;
  for (int f = 0; f < e; ++f) c0 += (a.b.ent_start[f + 1] - a.b.ent_start[f] + CH_T - 1) / CH_T;
  const int n = (a.b.ent_start[e + 1] - a.b.ent_start[e] + CH_T - 1) / CH_T;
  if (d >= a.dim || c >= a.vdim) return;                       // the padding's sums are zeros and stay
  float* st = a.state + (((size_t)a.b.ent_slot[e] * a.H + h) * a.dim + d) * a.vdim + c;
  const bool c1 = c + 1 < a.vdim, d1 = d + 1 < a.dim;
  float s[4] = {};                                             // (d, c), (d + 1, c), (d, c + 1), (d + 1, c + 1)
  if (a.b.ent_pos0[e] > 0) {
    s[0] = st[0];
    if (d1) s[1] = st[a.vdim];
    if (c1) s[2] = st[1];
    if (d1 && c1) s[3] = st[a.vdim + 1];
  }
  const size_t step = (size_t)a.H * DK * DV;
  float* p = a.states + ((size_t)c0 * a.H + h) * DK * DV + i;
  const float* w = a.ends + ((size_t)c0 * a.H + h) * DK + d;
  for (int j = 0; j < n; j += 4) {
    float4 x[4];
    float2 f[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (j + k < n) {
        x[k] = *reinterpret_cast<const float4*>(p + (j + k) * step);
        f[k] = *reinterpret_cast<const float2*>(w + (size_t)(j + k) * a.H * DK);
      }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (j + k >= n) break;
      *reinterpret_cast<float4*>(p + (j + k) * step) = make_float4(s[0], s[1], s[2], s[3]);
      s[0] = fmaf(f[k].x, s[0], x[k].x); s[1] = fmaf(f[k].y, s[1], x[k].y); s[2] = fmaf(f[k].x, s[2], x[k].z); s[3] = fmaf(f[k].y, s[3], x[k].w);
    }
  }
  st[0] = s[0];
  if (d1) st[a.vdim] = s[1];
  if (c1) st[1] = s[2];
  if (d1 && c1) st[a.vdim + 1] = s[3];
}

// Shared memory of the read-outs: queries, keys (then two slices of the state), decays (then values and weights), per sub-block products and scalars.
template <typename AT, int DK, int DV>
__host__ __device__ constexpr size_t ch_third_bytes() {
  const size_t vw = (size_t)CH_T * DV * sizeof(AT) + CH_T * CH_T * 4, d = (size_t)CH_T * DK * 4;
  return vw > d ? vw : d;
}
template <int DK, int DV>
__host__ __device__ constexpr size_t ch_second_bytes() {
  const size_t s = 2 * 32 * (size_t)DV * 4, k = (size_t)CH_T * DK * 4;
  return s > k ? s : k;
}
template <typename AT, int DK, int DV>
__host__ __device__ constexpr size_t ch_out_smem() {
  return (size_t)CH_T * DK * 4 + ch_second_bytes<DK, DV>() + ch_third_bytes<AT, DK, DV>() + (CH_SUBS * DK + 4 * CH_T) * 4;
}

// Weights of pairs inside one sub-block, decays per channel: half a warp takes key j of the sub-block, a lane 4 or 8 of its channels, and the
// running product k_j a_j+1 .. a_i meets the queries i = j .. 15; the sixteen sums are then exchanged so that lane i keeps that of query i.
// TWO: and with the keys in the queries' place (w2).
template <int DK, bool FORGET, bool TWO = false>
__device__ __forceinline__ float ch_pairs(const float* sq, const float* sk, const float* sd, int s, int j, int jw, int l, float* w2 = nullptr) {
  constexpr int NC = DK / 64;
  float p[CH_SUB], p2[TWO ? CH_SUB : 1];
  float2 w[2 * NC];
#pragma unroll
  for (int c = 0; c < 2 * NC; ++c) w[c] = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int i = 0; i < CH_SUB; ++i) {
    p[i] = 0.0f;
    if constexpr (TWO) p2[i] = 0.0f;
    if (i < CH_SUB / 2 && jw >= CH_SUB / 2) continue;          // the same for the whole warp
    const int r = s * CH_SUB + i;
    float2 sum = make_float2(0.0f, 0.0f), sum2 = sum;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int at = ch_at<DK, true>(r, c * 64 + l * 4);
      const float4 d = *reinterpret_cast<const float4*>(sd + at), q = *reinterpret_cast<const float4*>(sq + at);
      if (i == j) {
        const float4 k = FORGET ? make_float4(1.0f - d.x, 1.0f - d.y, 1.0f - d.z, 1.0f - d.w) : *reinterpret_cast<const float4*>(sk + at);
        w[2 * c] = make_float2(k.x, k.y); w[2 * c + 1] = make_float2(k.z, k.w);
      } else {
        w[2 * c] = mul2(w[2 * c], make_float2(d.x, d.y)); w[2 * c + 1] = mul2(w[2 * c + 1], make_float2(d.z, d.w));
      }
      sum = fma2(w[2 * c], make_float2(q.x, q.y), sum);
      sum = fma2(w[2 * c + 1], make_float2(q.z, q.w), sum);
      if constexpr (TWO) {
        const float4 k = *reinterpret_cast<const float4*>(sk + at);
        sum2 = fma2(w[2 * c], make_float2(k.x, k.y), sum2);
        sum2 = fma2(w[2 * c + 1], make_float2(k.z, k.w), sum2);
      }
    }
    p[i] = sum.x + sum.y;
    if constexpr (TWO) p2[i] = sum2.x + sum2.y;
  }
  auto exchange = [&](float* v) {
    int n = CH_SUB;
#pragma unroll
    for (int x = 8; x >= 1; x >>= 1) {
      n >>= 1;
      const bool hi = (l & x) != 0;
#pragma unroll
      for (int u = 0; u < CH_SUB / 2; ++u) {
        if (u >= n) break;
        const float other = __shfl_xor_sync(0xffffffffu, hi ? v[u] : v[u + n], x);
        v[u] = (hi ? v[u + n] : v[u]) + other;
      }
    }
  };
  exchange(p);
  if constexpr (TWO) { exchange(p2); *w2 = p2[0]; }
  return p[0];                                                 // of query l
}

// Weights of the queries of sub-block I and the keys of the sub-blocks before it: x [i][d] . y [j][d], both carried to I's beginning.  A thread
// takes 4 queries x I keys over a quarter of the channels; the quarters meet by shuffles.
// put(query of the chunk, sub-block of the key, key of the sub-block, weight).
template <int DK, typename Put>
__device__ __forceinline__ void ch_block_row(const float* x, const float* y, int I, Put put) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, dg = lane >> 3, jt = (warp & 1) * 8 + (lane & 7), i0 = I * CH_SUB + (warp >> 1) * 4;
  float2 acc[4][3] = {};
#pragma unroll 2
  for (int c = 0; c < DK / 16; ++c) {
    const int d = (c * 4 + dg) * 4;
    float4 q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = *reinterpret_cast<const float4*>(x + ch_at<DK, true>(i0 + i, d));
#pragma unroll
    for (int jj = 0; jj < 3; ++jj) {
      if (jj >= I) break;
      const float4 k = *reinterpret_cast<const float4*>(y + ch_at<DK, true>(jj * CH_SUB + jt, d));
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc[i][jj] = fma2(make_float2(q[i].x, q[i].y), make_float2(k.x, k.y), acc[i][jj]);
        acc[i][jj] = fma2(make_float2(q[i].z, q[i].w), make_float2(k.z, k.w), acc[i][jj]);
      }
    }
  }
#pragma unroll
  for (int jj = 0; jj < 3; ++jj) {
    if (jj >= I) break;
    float mine = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float s = acc[i][jj].x + acc[i][jj].y;
      s += __shfl_xor_sync(0xffffffffu, s, 8);
      s += __shfl_xor_sync(0xffffffffu, s, 16);
      if (i == dg) mine = s;
    }
    put(i0 + dg, jj, jt, mine);
  }
}

// The read-outs of a chunk.  grid (chunks, H), 256 threads; the products with the state and with the values run with 8 rows per warp and DV / 32
// columns per lane.
template <typename AT, int DK, int DV, int MODE>
__global__ void __launch_bounds__(256, 2) gla_chunk_out_kernel(ChunkArgs<AT> a) {
  pdl_begin();
  constexpr bool SCALAR = MODE == GLA_HEAD || MODE == GLA_TOKEN;
  constexpr int TV = DV / 32;
  extern __shared__ __align__(16) unsigned char hy_smem[];
  float* sq = reinterpret_cast<float*>(hy_smem);               // [64][DK] queries
  float* sk = sq + CH_T * DK;                                  // [64][DK] keys, then [2][32][DV] rows of the state
  float* sd = reinterpret_cast<float*>(hy_smem + (size_t)CH_T * DK * 4 + ch_second_bytes<DK, DV>());     // [64][DK] decays, then:
  AT* sv = reinterpret_cast<AT*>(sd);                          // [64][DV] values
  float* sw = reinterpret_cast<float*>(sv + CH_T * DV);        // [64][64] weights
  float* se = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(sd) + ch_third_bytes<AT, DK, DV>());   // [4][DK]
  float* sa = se + CH_SUBS * DK;                               // [64] decay, [64] factor of the value, [64] from the sub-block's beginning, [64] to its end
  const ChunkPlace p(a.b, blockIdx.x);
  const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int per = MODE == GLA_TOKEN ? a.tk.G : a.H, row = MODE == GLA_TOKEN ? h / (a.H / a.tk.G) : h;
  const float* rows = a.qk + ((size_t)p.t0 * per + row) * 2 * a.dim;
  const size_t ld = (size_t)per * 2 * a.dim;
  ch_rows<DK, true>(sq, rows, ld, p.n, a.dim, a.vec, 0.0f);
  if constexpr (MODE == GLA_FORGET) ch_rows<DK, true>(sd, rows + a.dim, ld, p.n, a.dim, a.vec, 1.0f);
  else ch_rows<DK, true>(sk, rows + a.dim, ld, p.n, a.dim, a.vec, 0.0f);
  if constexpr (MODE == GLA_CHANNEL) ch_rows<DK, true>(sd, a.decay + (size_t)p.t0 * a.ldd + h * a.dim, a.ldd, p.n, a.dim, a.vec, 1.0f);
  if constexpr (SCALAR) ch_scalars<AT, MODE>(a, p, h, sa, sa + CH_T);
  auto values = [&]() {
    constexpr int CH = 16 / (int)sizeof(AT);
    const AT* src = a.v + (size_t)p.t0 * a.ldv + h * a.vdim;
    if (a.vvec) {
      for (int i = tid; i < CH_T * (DV / CH); i += 256) {
        const int r = i / (DV / CH), c = i % (DV / CH) * CH;
        AT* d = sv + r * DV + c;
        if (r < p.n && c < a.vdim) jf::cp_async_16(d, src + (size_t)r * a.ldv + c, 16u);
        else *reinterpret_cast<uint4*>(d) = make_uint4(0u, 0u, 0u, 0u);
      }
    } else {
      for (int i = tid; i < CH_T * DV; i += 256) {
        const int r = i / DV, c = i % DV;
        sv[i] = r < p.n && c < a.vdim ? src[(size_t)r * a.ldv + c] : from_f<AT>(0.0f);
      }
    }
    jf::cp_async_commit();
  };
  const bool first = p.index == 0 && a.b.ent_pos0[p.e] == 0;   // behind nothing: the state is zero
  const float* S = a.states + ((size_t)blockIdx.x * a.H + h) * DK * DV;
  auto slice = [&](int i) {                                    // rows 32 i .. of the state
    float* d = sk + (i & 1) * 32 * DV;
    for (int k = tid; k < 32 * DV / 4; k += 256) jf::cp_async_16(d + 4 * k, S + (size_t)i * 32 * DV + 4 * k, 16u);
    jf::cp_async_commit();
  };
  if constexpr (SCALAR) values();
  jf::cp_async_commit();
  jf::cp_async_wait_all();
  __syncthreads();
  if constexpr (!SCALAR) {
    float own[CH_SUBS];                                        // weight (query l, key j) of each sub-block
    const int l = tid & 15, hw = tid >> 4;
#pragma unroll
    for (int s = 0; s < CH_SUBS; ++s) {
      const int j = s & 1 ? 15 - hw : hw, jw = s & 1 ? 14 - 2 * warp : 2 * warp;
      own[s] = s * CH_SUB < p.n ? ch_pairs<DK, MODE == GLA_FORGET>(sq, sk, sd, s, j, jw, l) : 0.0f;
    }
    __syncthreads();
    for (int i = tid; i < CH_SUBS * DK; i += 256) {            // queries from their sub-block's beginning, keys to its end
      const int s = i / DK, d = i % DK;
      float w = 1.0f, dec[CH_SUB];
#pragma unroll
      for (int t = 0; t < CH_SUB; ++t) {
        const int at = ch_at<DK, true>(s * CH_SUB + t, d);
        dec[t] = sd[at];
        w *= dec[t];
        sq[at] *= w;
      }
      se[i] = w;
      w = 1.0f;
#pragma unroll
      for (int t = CH_SUB - 1; t >= 0; --t) {
        const int at = ch_at<DK, true>(s * CH_SUB + t, d);
        sk[at] = (MODE == GLA_FORGET ? 1.0f - dec[t] : sk[at]) * w;
        w *= dec[t];
      }
    }
    __syncthreads();                                           // the decays are done with: values and weights take their place
    values();
#pragma unroll
    for (int s = 0; s < CH_SUBS; ++s) sw[(s * CH_SUB + l) * CH_T + s * CH_SUB + (s & 1 ? 15 - hw : hw)] = own[s];
#pragma unroll 1
    for (int I = 1; I < CH_SUBS && I * CH_SUB < p.n; ++I) {
      if (I > 1) {                                             // keys of the earlier sub-blocks: on over sub-block I - 1
        for (int i = tid; i < (I - 1) * CH_SUB * DK; i += 256) {
          const int r = i / DK, d = i % DK;
          sk[ch_at<DK, true>(r, d)] *= se[(I - 1) * DK + d];
        }
        __syncthreads();
      }
      ch_block_row<DK>(sq, sk, I, [&](int i, int J, int j, float v) { sw[i * CH_T + J * CH_SUB + j] = v; });
      __syncthreads();
    }
    if (!first) {                                              // queries from the chunk's beginning
      constexpr int PER = 256 / DK;
      const int d = tid % DK;
      float w = 1.0f;
#pragma unroll
      for (int I = 1; I < CH_SUBS; ++I) {
        w *= se[(I - 1) * DK + d];
#pragma unroll
        for (int r = 0; r < CH_SUB / PER; ++r) sq[ch_at<DK, true>(I * CH_SUB + r * PER + tid / DK, d)] *= w;
      }
    }
    __syncthreads();
  } else {
    float* sl = sa + 2 * CH_T;                                 // from the sub-block's beginning on; to its end
    float* sr = sa + 3 * CH_T;
    if (tid < 2 * CH_SUBS) {
      const int s = tid >> 1;
      float w = 1.0f;
      if ((tid & 1) == 0) {
        for (int t = 0; t < CH_SUB; ++t) { w *= sa[s * CH_SUB + t]; sl[s * CH_SUB + t] = w; }
        se[s] = w;
      } else {
        for (int t = CH_SUB - 1; t >= 0; --t) { sr[s * CH_SUB + t] = w; w *= sa[s * CH_SUB + t]; }
      }
    }
    // q . k of 4 queries x 4 keys per thread (keys tx, tx + 16, ..); what lies above the diagonal's blocks is left out
    const int tx = tid & 15, ty = tid >> 4, I = ty >> 2;
    float2 acc[4][4] = {};
#pragma unroll 2
    for (int d = 0; d < DK; d += 4) {
      float4 q[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) q[i] = *reinterpret_cast<const float4*>(sq + ch_at<DK, true>(ty * 4 + i, d));
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        if (jj > I) break;
        const float4 k = *reinterpret_cast<const float4*>(sk + ch_at<DK, true>(jj * 16 + tx, d));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[i][jj] = fma2(make_float2(q[i].x, q[i].y), make_float2(k.x, k.y), acc[i][jj]);
          acc[i][jj] = fma2(make_float2(q[i].z, q[i].w), make_float2(k.z, k.w), acc[i][jj]);
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = ty * 4 + i;
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        if (jj > I) break;
        const int j = jj * 16 + tx;
        if (j > r) continue;
        float w = sa[CH_T + j];                                // the value's factor
        if (jj == I) { for (int m = j + 1; m <= r; ++m) w *= sa[m]; }
        else {
          w *= sl[r] * sr[j];
          for (int s = jj + 1; s < I; ++s) w *= se[s];
        }
        sw[r * CH_T + j] = (acc[i][jj].x + acc[i][jj].y) * w;
      }
    }
    __syncthreads();                                           // the keys are done with
  }
  const int r0 = warp * 8, c0 = lane * TV;
  float2 acc[8][TV] = {};                                      // sums over even and over odd rows of the second operand
  if (!first) {
    slice(0);
#pragma unroll 1
    for (int i = 0; i < DK / 32; ++i) {
      if (i + 1 < DK / 32) { slice(i + 1); jf::cp_async_wait_1(); }
      else jf::cp_async_wait_all();
      __syncthreads();
      const float* s = sk + (i & 1) * 32 * DV + 2 * c0;
      const float* q = sq + r0 * DK + i * 32;
#pragma unroll
      for (int d = 0; d < 32; d += 4) {
        VecN<float, 4> x[TV];                                  // two row pairs of TV columns
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int c = 0; c < TV / 2; ++c) x[k * (TV / 2) + c] = *reinterpret_cast<const VecN<float, 4>*>(s + (d + 2 * k) * DV + 4 * c);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const float4 qq = *reinterpret_cast<const float4*>(q + r * DK + (((d >> 2) ^ r) << 2));
#pragma unroll
          for (int c = 0; c < TV; ++c) {
            const VecN<float, 4>&u = x[c / 2], &v = x[TV / 2 + c / 2];
            acc[r][c] = fma2(make_float2(qq.x, qq.y), make_float2(u.v[2 * (c & 1)], u.v[2 * (c & 1) + 1]), acc[r][c]);
            acc[r][c] = fma2(make_float2(qq.z, qq.w), make_float2(v.v[2 * (c & 1)], v.v[2 * (c & 1) + 1]), acc[r][c]);
          }
        }
      }
      __syncthreads();                                         // the slice may be written over
    }
    if constexpr (SCALAR) {                                    // the decays from the chunk's beginning on
      float e = 1.0f;
      for (int s = 0; s < r0 / CH_SUB; ++s) e *= se[s];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float w = e * sa[2 * CH_T + r0 + r];
#pragma unroll
        for (int c = 0; c < TV; ++c) acc[r][c] = mul2(acc[r][c], make_float2(w, w));
      }
    }
  } else {
    jf::cp_async_wait_all();
    __syncthreads();
  }
  auto value = [&](int j, float (&x)[TV]) {
    const VecN<AT, TV> v = *reinterpret_cast<const VecN<AT, TV>*>(sv + j * DV + c0);
#pragma unroll
    for (int c = 0; c < TV; ++c) x[c] = to_f(v.v[c]);
  };
  // Values j .. j + 3; own: where they begin among the warp's eight tokens, of which a query meets those up to itself (negative: all come before).
  auto weigh = [&](int j, auto own) {
    constexpr int OWN = decltype(own)::value;
    float x[4][TV];
#pragma unroll
    for (int k = 0; k < 4; ++k) value(j + k, x[k]);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (r < OWN) continue;
      const float4 w = *reinterpret_cast<const float4*>(sw + (r0 + r) * CH_T + j);
#pragma unroll
      for (int c = 0; c < TV; ++c) {
        if (OWN < 0 || r > OWN) acc[r][c] = fma2(make_float2(w.x, w.y), make_float2(x[0][c], x[1][c]), acc[r][c]);
        else acc[r][c].x = fmaf(w.x, x[0][c], acc[r][c].x);
        if (OWN < 0 || r > OWN + 2) acc[r][c] = fma2(make_float2(w.z, w.w), make_float2(x[2][c], x[3][c]), acc[r][c]);
        else if (r == OWN + 2) acc[r][c].x = fmaf(w.z, x[2][c], acc[r][c].x);
      }
    }
  };
  const int before = min(r0, p.n);
#pragma unroll 1
  for (int j = 0; j < before; j += 4) weigh(j, std::integral_constant<int, -1>{});
  if (r0 < p.n) weigh(r0, std::integral_constant<int, 0>{});
  if (r0 + 4 < p.n) weigh(r0 + 4, std::integral_constant<int, 4>{});
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int t = r0 + r;
    if (t >= p.n) break;
    VecN<float, TV> y;
#pragma unroll
    for (int c = 0; c < TV; ++c) y.v[c] = acc[r][c].x + acc[r][c].y;
    if constexpr (MODE == GLA_TOKEN) {
      float x[TV];
      value(t, x);
      const float skip = a.tk.D[h];
#pragma unroll
      for (int c = 0; c < TV; ++c) y.v[c] = fmaf(skip, x[c], y.v[c]);
    }
    float* out = a.o + (size_t)(p.t0 + t) * a.ldo + h * a.vdim + c0;
    if (a.ovec) {
      if (c0 < a.vdim) *reinterpret_cast<VecN<float, TV>*>(out) = y;
      continue;
    }
#pragma unroll
    for (int c = 0; c < TV; ++c)
      if (c0 + c < a.vdim) out[c] = y.v[c];
  }
}

// ---- the delta rule -------------------------------------------------------------------------------------------------------------------
// S <- a S ;  u = beta (v - S^T k) ;  S <- S + k u^T ;  o = S^T q  (hy_delta.cuh).  Within a chunk, with K' = k carried from the chunk's beginning, the
// corrections u solve a unit lower triangular system,  (I + M) U = beta (V - K' S),  M_ij = beta_i (k_i . a_j+1 .. a_i . k_j),  so
//   U = U0 - W S   with (I + M) [W | U0] = beta [K' | V]        and then as above        S' = diag(a_0 .. a_63) S + k''^T U,   O = Q' S + A U.
// delta_chunk_prep_kernel makes W, U0, Q', k'', A and the decays' product of all chunks side by side; delta_chunk_chain_kernel walks the chunks of
// a head, 16 columns per block (columns do not meet).  |u| stays within beta times the state, so the system's solution does not grow.  One
// decay per head is taken as the same for all channels.
// The chain: what a chunk brings travels in two halves while the other half is worked on.  5.2 us a chunk (5.9 when a row's corrections met the
// zeros behind its token as well), bound by reading operands from shared memory (eight 16-byte reads for 32 fma.rn.f32x2): half of it products
// with the state, then corrections of the state and starting copies.
// 2048 tokens, 16 heads of 128 x 128 with channel decays: 430 us token by token; prep 128 and chain 165.
template <typename AT>
struct DeltaArgs {
  Batch b;
  const float* qk; const AT* v; int ldv; const float4* sc; const float* dec; int ldd;      // as delta_head_kernel's; dec NULL: one decay per head in sc
  int H, G, dim, vdim, vec;
  float* work; float* state; float* o; int ldo;
};
// Floats of a chunk and head: W | Q' | k'' (rows in pairs, [32][DK][2]) | U0 | A | decays' product.
template <int DK, int DV>
struct DeltaWork {
  static constexpr int W = 0, Q = CH_T * DK, K = 2 * CH_T * DK, U = 3 * CH_T * DK, A = U + CH_T * DV, E = A + CH_T * CH_T, SIZE = E + DK;
};
__host__ __device__ constexpr size_t delta_work_floats(int dk, int dv) { return (size_t)3 * CH_T * dk + (size_t)CH_T * dv + CH_T * CH_T + dk; }

// M of the sub-blocks (I, J <= I), [key][query] each.
__device__ __forceinline__ int ch_tri(int I, int J) { return (I * (I + 1) / 2 + J) * CH_SUB * CH_SUB; }
template <int DK, int DV>
__host__ __device__ constexpr size_t delta_prep_smem() {
  const size_t y = (size_t)CH_T * (DK + DV) * 4, qk = 2 * (size_t)CH_T * DK * 4;
  return (y > qk ? y : qk) + ((size_t)CH_T * DK + 10 * CH_SUB * CH_SUB + CH_SUBS * DK + CH_T) * 4;
}
// grid (chunks, H), 256 threads.
template <typename AT, int DK, int DV>
__global__ void __launch_bounds__(256, 2) delta_chunk_prep_kernel(DeltaArgs<AT> a) {
  pdl_begin();
  typedef DeltaWork<DK, DV> Work;
  extern __shared__ __align__(16) unsigned char hy_smem[];
  float* sq = reinterpret_cast<float*>(hy_smem);               // [64][DK] queries | [64][DK] keys, at last the solution [64][DK + DV]
  float* sk = sq + CH_T * DK;
  float* sd = sq + (DK + DV > 2 * DK ? CH_T * (DK + DV) : 2 * CH_T * DK);      // [64][DK] decays, then keys from their sub-block's beginning
  float* sm = sd + CH_T * DK;                                  // M
  float* se = sm + 10 * CH_SUB * CH_SUB;                       // [4][DK] products of a sub-block's decays
  float* sb = se + CH_SUBS * DK;                               // [64] step sizes
  const ChunkPlace p(a.b, blockIdx.x);
  const int h = blockIdx.y, g = h / (a.H / a.G), tid = threadIdx.x, warp = tid >> 5;
  const float* rows = a.qk + ((size_t)p.t0 * a.G + g) * 2 * a.dim;
  const size_t ld = (size_t)a.G * 2 * a.dim;
  ch_rows<DK, true>(sq, rows, ld, p.n, a.dim, a.vec, 0.0f);
  ch_rows<DK, true>(sk, rows + a.dim, ld, p.n, a.dim, a.vec, 0.0f);
  if (a.dec) ch_rows<DK, true>(sd, a.dec + (size_t)p.t0 * a.ldd + h * a.dim, a.ldd, p.n, a.dim, a.vec, 1.0f);
  if (tid < CH_T) {
    const float4 sc = tid < p.n ? a.sc[(size_t)(p.t0 + tid) * a.H + h] : make_float4(1.0f, 0.0f, 0.0f, 0.0f);
    sb[tid] = sc.y;
    se[tid] = sc.x;
  }
  if (!a.dec) {
    __syncthreads();
    for (int i = tid; i < CH_T * DK; i += 256) sd[i] = se[i / DK];
  }
  jf::cp_async_commit();
  jf::cp_async_wait_all();
  __syncthreads();
  float* work = a.work + ((size_t)blockIdx.x * a.H + h) * Work::SIZE;
  const int l = tid & 15, hw = tid >> 4;
#pragma unroll 1
  for (int s = 0; s < CH_SUBS; ++s) {                          // weights inside a sub-block: (query l, key j)
    const int j = s & 1 ? 15 - hw : hw, jw = s & 1 ? 14 - 2 * warp : 2 * warp;
    float m;
    const float w = ch_pairs<DK, false, true>(sq, sk, sd, s, j, jw, l, &m);
    work[Work::A + (s * CH_SUB + l) * CH_T + s * CH_SUB + j] = w;
    sm[ch_tri(s, s) + j * CH_SUB + l] = m * sb[s * CH_SUB + l];
  }
  __syncthreads();
  for (int i = tid; i < CH_SUBS * DK; i += 256) {              // queries and keys from their sub-block's beginning, keys to its end
    const int s = i / DK, d = i % DK;
    float w = 1.0f, dec[CH_SUB], key[CH_SUB];
#pragma unroll
    for (int t = 0; t < CH_SUB; ++t) {
      const int at = ch_at<DK, true>(s * CH_SUB + t, d);
      dec[t] = sd[at]; key[t] = sk[at];
      w *= dec[t];
      sq[at] *= w;
      sd[at] = key[t] * w;
    }
    se[i] = w;
    w = 1.0f;
#pragma unroll
    for (int t = CH_SUB - 1; t >= 0; --t) {
      sk[ch_at<DK, true>(s * CH_SUB + t, d)] = key[t] * w;
      w *= dec[t];
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int I = 1; I < CH_SUBS; ++I) {
    if (I > 1) {                                               // keys of the earlier sub-blocks: on over sub-block I - 1
      for (int i = tid; i < (I - 1) * CH_SUB * DK; i += 256) sk[ch_at<DK, true>(i / DK, i % DK)] *= se[(I - 1) * DK + i % DK];
      __syncthreads();
    }
    ch_block_row<DK>(sq, sk, I, [&](int i, int J, int j, float v) { work[Work::A + i * CH_T + J * CH_SUB + j] = v; });
    ch_block_row<DK>(sd, sk, I, [&](int i, int J, int j, float v) { sm[ch_tri(I, J) + j * CH_SUB + i - I * CH_SUB] = v * sb[i]; });
    __syncthreads();
  }
  {                                                            // from the chunk's beginning and to its end
    constexpr int PER = 256 / DK;
    const int d = tid % DK;
    const float last = se[(CH_SUBS - 1) * DK + d];
    float w = 1.0f;
#pragma unroll
    for (int I = 0; I < CH_SUBS; ++I) {
#pragma unroll
      for (int r = 0; r < CH_SUB / PER; ++r) {
        const int row = I * CH_SUB + r * PER + tid / DK, at = ch_at<DK, true>(row, d);
        work[Work::Q + row * DK + d] = sq[at] * w;
        sd[at] *= w;
        work[Work::K + (row >> 1) * 2 * DK + 2 * d + (row & 1)] = sk[at] * (I < CH_SUBS - 1 ? last : 1.0f);
      }
      w *= se[I * DK + d];
    }
    if (tid < DK) work[Work::E + d] = w;
  }
  __syncthreads();
  // (I + M) Y = beta [K' | V], a column per thread; what is solved stays in shared memory for the sub-blocks behind it
  for (int c = tid; c < DK + DV; c += 256) {
    float* y = sq + c;
    constexpr int LD = DK + DV;
#pragma unroll 1
    for (int I = 0; I < CH_SUBS; ++I) {
      float2 r[CH_SUB / 2];
#pragma unroll
      for (int t = 0; t < CH_SUB; ++t) {
        const int row = I * CH_SUB + t;
        float x;
        if (c < DK) x = sd[ch_at<DK, true>(row, c)];
        else x = row < p.n && c - DK < a.vdim ? to_f(a.v[(size_t)(p.t0 + row) * a.ldv + h * a.vdim + c - DK]) : 0.0f;
        (t & 1 ? r[t / 2].y : r[t / 2].x) = x * sb[row];
      }
#pragma unroll 1
      for (int J = 0; J < I; ++J) {
        const float* m = sm + ch_tri(I, J);
#pragma unroll 4
        for (int j = 0; j < CH_SUB; ++j) {
          const float u = -y[(J * CH_SUB + j) * LD];
#pragma unroll
          for (int t = 0; t < CH_SUB / 4; ++t) {
            const float4 mm = *reinterpret_cast<const float4*>(m + j * CH_SUB + 4 * t);
            r[2 * t] = fma2(make_float2(mm.x, mm.y), make_float2(u, u), r[2 * t]);
            r[2 * t + 1] = fma2(make_float2(mm.z, mm.w), make_float2(u, u), r[2 * t + 1]);
          }
        }
      }
      const float* m = sm + ch_tri(I, I);
#pragma unroll
      for (int j = 0; j < CH_SUB; ++j) {
        const float u = j & 1 ? r[j / 2].y : r[j / 2].x;
#pragma unroll
        for (int t = j / 4; t < CH_SUB / 4; ++t) {             // of row j's own four those behind it
          if (4 * t + 3 == j) continue;
          const float4 mm = *reinterpret_cast<const float4*>(m + j * CH_SUB + 4 * t);
          if (4 * t > j) r[2 * t] = fma2(make_float2(mm.x, mm.y), make_float2(-u, -u), r[2 * t]);
          else if (4 * t == j) r[2 * t].y = fmaf(mm.y, -u, r[2 * t].y);
          if (4 * t + 1 >= j) r[2 * t + 1] = fma2(make_float2(mm.z, mm.w), make_float2(-u, -u), r[2 * t + 1]);
          else r[2 * t + 1].y = fmaf(mm.w, -u, r[2 * t + 1].y);
        }
      }
#pragma unroll
      for (int t = 0; t < CH_SUB; ++t) {
        const int row = I * CH_SUB + t;
        const float x = t & 1 ? r[t / 2].y : r[t / 2].x;
        y[row * LD] = x;
        work[c < DK ? Work::W + row * DK + c : Work::U + row * DV + c - DK] = x;
      }
    }
  }
}

// Columns of a block of the chain, and its shared memory: W and Q' (chunks of 16 bytes xor the row's low bits), k'' and A, U0, the state and the
// corrections with rows in pairs, sums of the second half of the channels.
constexpr int DELTA_COLS = 16;
template <int DK>
__host__ __device__ constexpr size_t delta_chain_smem() {
  return ((size_t)3 * CH_T * DK + CH_T * CH_T + CH_T * DELTA_COLS + DK * DELTA_COLS + CH_T * DELTA_COLS + 128 * DELTA_COLS) * 4;
}
// grid (H * DV / 16, entries), 256 threads.
template <typename AT, int DK, int DV>
__global__ void __launch_bounds__(256) delta_chunk_chain_kernel(DeltaArgs<AT> a) {
  pdl_begin();
  typedef DeltaWork<DK, DV> Work;
  constexpr int C = DELTA_COLS;
  extern __shared__ __align__(16) unsigned char hy_smem[];
  float* swq = reinterpret_cast<float*>(hy_smem);              // [128][DK]
  float* skk = swq + 2 * CH_T * DK;                            // [32][DK][2]
  float* sA = skk + CH_T * DK;                                 // [64][64]
  float* su0 = sA + CH_T * CH_T;                               // [64][16]
  float* sS = su0 + CH_T * C;                                  // [DK / 2][16][2]
  float* sU = sS + DK * C;                                     // [32][16][2]
  float* sr = sU + CH_T * C;                                   // [128][16]
  const int e = blockIdx.y, h = blockIdx.x / (DV / C), c0 = blockIdx.x % (DV / C) * C, tid = threadIdx.x;
  if (c0 >= a.vdim) return;
  const int start = a.b.ent_start[e], cnt = a.b.ent_start[e + 1] - start, n = (cnt + CH_T - 1) / CH_T;
  int chunk = 0;
  for (int f = 0; f < e; ++f) chunk += (a.b.ent_start[f + 1] - a.b.ent_start[f] + CH_T - 1) / CH_T;
  float* st = a.state + ((size_t)a.b.ent_slot[e] * a.H + h) * a.dim * a.vdim;
  for (int i = tid; i < DK * C; i += 256) {
    const int d = i / C, c = i % C;
    sS[(d >> 1) * 2 * C + 2 * c + (d & 1)] = d < a.dim && c0 + c < a.vdim && a.b.ent_pos0[e] > 0 ? st[(size_t)d * a.vdim + c0 + c] : 0.0f;
  }
  const float* work = a.work + ((size_t)chunk * a.H + h) * Work::SIZE;
  const size_t step = (size_t)a.H * Work::SIZE;
  auto first_half = [&](const float* w) {
    for (int i = tid; i < 2 * CH_T * (DK / 4); i += 256) {
      const int r = i / (DK / 4), c = i % (DK / 4);
      jf::cp_async_16(swq + r * DK + ((c ^ (r & 7)) << 2), w + Work::W + r * DK + 4 * c, 16u);
    }
    jf::cp_async_16(su0 + tid * 4, w + Work::U + (tid >> 2) * DV + c0 + (tid & 3) * 4, 16u);
    jf::cp_async_commit();
  };
  auto second_half = [&](const float* w) {
    for (int i = tid; i < CH_T * DK / 4; i += 256) jf::cp_async_16(skk + 4 * i, w + Work::K + 4 * i, 16u);
    for (int i = tid; i < CH_T * CH_T / 4; i += 256) {
      const int r = i / 16, c = i % 16;
      jf::cp_async_16(sA + r * CH_T + ((c ^ (r & 7)) << 2), w + Work::A + 4 * i, 16u);
    }
    jf::cp_async_commit();
  };
  first_half(work);
  second_half(work);
  const int kh = tid >> 7, rg = (tid & 127) >> 2, cg = (tid & 3) * 4;
#pragma unroll 1
  for (int j = 0; j < n; ++j, work += step) {
    jf::cp_async_wait_1();                                     // the second half of this chunk may still travel
    __syncthreads();
    float2 acc[4][4] = {};                                     // rows rg + 32 i of W and Q' times columns cg .. + 3 of the state, half of its channels
#pragma unroll 4
    for (int k = kh * (DK / 2); k < (kh + 1) * (DK / 2); k += 4) {
      VecN<float, 4> s[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) s[i] = *reinterpret_cast<const VecN<float, 4>*>(sS + (k / 2 + (i >> 1)) * 2 * C + 2 * cg + (i & 1) * 4);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 w = *reinterpret_cast<const float4*>(swq + (rg + 32 * i) * DK + (((k >> 2) ^ (rg & 7)) << 2));
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          acc[i][c] = fma2(make_float2(w.x, w.y), make_float2(s[c / 2].v[2 * (c & 1)], s[c / 2].v[2 * (c & 1) + 1]), acc[i][c]);
          acc[i][c] = fma2(make_float2(w.z, w.w), make_float2(s[2 + c / 2].v[2 * (c & 1)], s[2 + c / 2].v[2 * (c & 1) + 1]), acc[i][c]);
        }
      }
    }
    if (kh) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float4*>(sr + (rg + 32 * i) * C + cg) = make_float4(acc[i][0].x + acc[i][0].y, acc[i][1].x + acc[i][1].y, acc[i][2].x + acc[i][2].y, acc[i][3].x + acc[i][3].y);
    }
    __syncthreads();
    float out[2][4];                                           // Q' S of rows rg and rg + 32
    if (!kh) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = rg + 32 * i;
        const float4 more = *reinterpret_cast<const float4*>(sr + r * C + cg);
        const float m[4] = {more.x, more.y, more.z, more.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float v = acc[i][c].x + acc[i][c].y + m[c];
          if (i < 2) sU[(r >> 1) * 2 * C + 2 * (cg + c) + (r & 1)] = su0[r * C + cg + c] - v;
          else out[i - 2][c] = v;
        }
      }
    }
    __syncthreads();
    if (j + 1 < n) { first_half(work + step); jf::cp_async_wait_1(); }
    else jf::cp_async_wait_all();
    __syncthreads();                                           // the second half of this chunk is there
    if (!kh) {
      float2 o2[2][4] = {};
      // Corrections t .. t + 3 times A, for the rows rg + 32 i from i = `from` on; `own`: the row that is one of these four and meets those up to itself.
      auto weigh = [&](int t, auto from, auto own) {
        VecN<float, 4> u[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) u[i] = *reinterpret_cast<const VecN<float, 4>*>(sU + (t / 2 + (i >> 1)) * 2 * C + 2 * cg + (i & 1) * 4);
#pragma unroll
        for (int i = decltype(from)::value; i < 2; ++i) {
          const float4 w = *reinterpret_cast<const float4*>(sA + (rg + 32 * i) * CH_T + (((t >> 2) ^ (rg & 7)) << 2));
          const int last = i == decltype(own)::value ? rg & 3 : 3;
          auto upto = [&](int k, float v) { return k <= last ? v : 0.0f; };
          const float2 w0 = make_float2(w.x, upto(1, w.y)), w1 = make_float2(upto(2, w.z), upto(3, w.w));
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float *x = u[c / 2].v + 2 * (c & 1), *y = u[2 + c / 2].v + 2 * (c & 1);
            o2[i][c] = fma2(w0, make_float2(x[0], upto(1, x[1])), o2[i][c]);
            o2[i][c] = fma2(w1, make_float2(upto(2, y[0]), upto(3, y[1])), o2[i][c]);
          }
        }
      };
      typedef std::integral_constant<int, 0> first; typedef std::integral_constant<int, 1> second; typedef std::integral_constant<int, 2> none;
      const int four = rg & ~3;
#pragma unroll 2
      for (int t = 0; t < four; t += 4) weigh(t, first{}, none{});
      weigh(four, first{}, first{});
#pragma unroll 2
      for (int t = four + 4; t < four + 32; t += 4) weigh(t, second{}, none{});
      weigh(four + 32, second{}, second{});
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int t = j * CH_T + rg + 32 * i;
        if (t >= cnt) continue;
        float* po = a.o + (size_t)(start + t) * a.ldo + h * a.vdim + c0 + cg;
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (c0 + cg + c < a.vdim) po[c] = out[i][c] + (o2[i][c].x + o2[i][c].y);
      }
    } else {
#pragma unroll 1
      for (int d = rg * 4; d < DK; d += 128) {                 // four channels x four columns of the state
        float2 up[4][4] = {};
#pragma unroll 4
        for (int t = 0; t < CH_T / 2; ++t) {
          const VecN<float, 4> k0 = *reinterpret_cast<const VecN<float, 4>*>(skk + t * 2 * DK + 2 * d), k1 = *reinterpret_cast<const VecN<float, 4>*>(skk + t * 2 * DK + 2 * d + 4);
          const VecN<float, 4> u0 = *reinterpret_cast<const VecN<float, 4>*>(sU + t * 2 * C + 2 * cg), u1 = *reinterpret_cast<const VecN<float, 4>*>(sU + t * 2 * C + 2 * cg + 4);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const VecN<float, 4>& k = i < 2 ? k0 : k1;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const VecN<float, 4>& u = c < 2 ? u0 : u1;
              up[i][c] = fma2(make_float2(k.v[2 * (i & 1)], k.v[2 * (i & 1) + 1]), make_float2(u.v[2 * (c & 1)], u.v[2 * (c & 1) + 1]), up[i][c]);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float w = __ldg(work + Work::E + d + i);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float& S = sS[((d + i) >> 1) * 2 * C + 2 * (cg + c) + ((d + i) & 1)];
            S = fmaf(w, S, up[i][c].x + up[i][c].y);
          }
        }
      }
    }
    __syncthreads();                                           // state and second half are done with
    if (j + 1 < n) second_half(work + step);
  }
  for (int i = tid; i < DK * C; i += 256) {
    const int d = i / C, c = i % C;
    if (d < a.dim && c0 + c < a.vdim) st[(size_t)d * a.vdim + c0 + c] = sS[(d >> 1) * 2 * C + 2 * c + (d & 1)];
  }
}

// ---- host: which recurrences run in chunks, in which steps (see step_chunks) ------------------------------------------------------------
// From 512 tokens of the longest request on: three launches and a block's own time cost 40 us, the chain of tokens 0.1 us each.  Token by token and in
// chunks, us: 8 heads with forget gates 512 tokens 66 and 62, 384 tokens 53 and 61; state space 512 tokens 78 and 61; gated linear, 16 heads, 512
// tokens 97 and 75, 320 tokens 70 and 71.  Key and value sizes up to 32 have too little work per chunk for it.
constexpr int HY_CHUNK_TOKENS = 512, HY_CHUNK_ENTRIES = 64;
inline bool chunk_sizes(int dk, int dv) { return dk > 32 && dk <= CH_MAX_DIM && dv > 32 && dv <= CH_MAX_DIM; }
// The delta rule's chain has a block per SM, and its blocks behind the first wave wait: 512 tokens of the longest request per wave.  Token by token and in
// chunks, us, channel decays, 16 heads of 128 x 128: one request of 512 tokens 122 and 107, 1024 232 and 178, 2048 452 and 345; two of 2048
// 424 and 351, four of 2048 (longest 780) 322 and 366.  One decay per head, 8 heads: 2048 tokens 365 and 263, four requests 187 and 198.  (With a
// chain of 5.9 us a chunk; at 5.2, one request of 2048 tokens 320, four about 330.)
inline bool delta_pays(int heads, int dv, int entries, int longest) {
  const long long blocks = (long long)heads * ((dv + DELTA_COLS - 1) / DELTA_COLS) * entries;
  return longest >= HY_CHUNK_TOKENS * ((blocks + 147) / 148);
}
// chunks that a step of max_step_tokens may be cut into
inline int chunk_cap(int max_tokens) { return (5 * max_tokens + 4 * CH_T) / (4 * CH_T); }

}  // namespace hy
