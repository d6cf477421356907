// hy_experts.cuh — routed gated feed-forward of the layered hybrid decoders (libjf_hybrid.so).
//
//   route     per token: sigmoid scores of the router logits, group-limited choice of `top` experts, normalised weights;
//             per-expert pair counts by atomic add (the counts, not their order, decide the layout)
//   place     every (token, choice) pair gets a row in its expert's range of the sorted order, and the token's activation row is
//             copied there; the exclusive prefix of the counts and the list of (expert, first row) tiles of the grouped products
//   products  gate/up with the gated activation in the epilogue, then down, both grouped by expert: a tile of the list reads its
//             rows of the sorted copy and its expert's weight matrix; a handful of pairs skip the order and take one block row each
//   combine   per token the weighted sum of its pairs' rows in the order of its choices, then the sublayer's output norm,
//             layer scale and the residual sum
// A token's choices, its weights and the order of its sum are its own, and a row of a product does not depend on the other rows of its
// tile; whether the few-pair kernel or the tiles make it depends on the number of pairs in the step.  Router scores, weights and the combine are fp32.
#pragma once
#include "hy_kernels.cuh"

namespace hy {

struct RouteCfg { int experts, top, groups, keep; float scale; };

// What a token chooses when no score compares (scores that are no numbers, or fewer finite ones than choices): the lowest expert that is not among
// its k choices so far.  A token's choices are distinct in every case: the products of few rows rely on it.  Out of line, where it costs choices that
// compare nothing (in line, steps of eight tokens took 0.5 to 0.9 % longer).
__device__ __noinline__ int lowest_free(const int* chosen, int k) {
  for (int e = 0;; ++e) {
    bool taken = false;
    for (int i = 0; i < k; ++i) taken |= chosen[i] == e;
    if (!taken) return e;
  }
}

// One warp per token.  Scores live in shared memory; lane 0 makes the (tiny, serial) choice.  Ties go to the lower index.
// A group is worth the sum of its two best scores (its single score when groups hold one expert).
__global__ void __launch_bounds__(32) route_kernel(const float* __restrict__ logits, int ldl, RouteCfg c, int* __restrict__ ids,
                                                   float* __restrict__ wts, int* __restrict__ counts) {
  pdl_begin();
  extern __shared__ __align__(16) unsigned char hy_smem[];
  float* s = reinterpret_cast<float*>(hy_smem);                // [experts] scores, negated once chosen
  float* gs = s + c.experts;                                   // [groups]; -1 once kept
  const int t = blockIdx.x, lane = threadIdx.x;
  for (int e = lane; e < c.experts; e += 32) s[e] = sigmoid_f(logits[(size_t)t * ldl + e]);
  __syncwarp();
  const int per = c.experts / c.groups;
  for (int g = lane; g < c.groups; g += 32) {
    float m1 = -1.0f, m2 = -1.0f;
    for (int i = 0; i < per; ++i) {
      const float v = s[g * per + i];
      if (v > m1) { m2 = m1; m1 = v; } else if (v > m2) { m2 = v; }
    }
    gs[g] = per >= 2 ? m1 + m2 : m1;
  }
  __syncwarp();
  if (lane != 0) return;
  // keep the best groups: kept groups are marked by a score below every real one (scores are sums of sigmoids, > 0)
  for (int k = 0; k < c.keep; ++k) {
    int best = 0; float bv = -1.0f;
    for (int g = 0; g < c.groups; ++g) if (gs[g] > bv) { bv = gs[g]; best = g; }
    gs[best] = -2.0f;
  }
  float sum = 0.0f;
  for (int k = 0; k < c.top; ++k) {
    int best = -1; float bv = -1.0f;
    for (int g = 0; g < c.groups; ++g) {
      if (gs[g] != -2.0f) continue;
      for (int i = 0; i < per; ++i) { const float v = s[g * per + i]; if (v > bv) { bv = v; best = g * per + i; } }
    }
    if (best < 0) best = lowest_free(ids + (size_t)t * c.top, k);
    ids[(size_t)t * c.top + k] = best;
    wts[(size_t)t * c.top + k] = bv;
    sum += bv;
    s[best] = -1.0f;
    if (counts) atomicAdd(&counts[best], 1);
  }
  const float f = c.scale / (sum + 1e-20f);
  for (int k = 0; k < c.top; ++k) wts[(size_t)t * c.top + k] *= f;
}

// The other way to score: the `top` largest router logits (bias added here, ties to the lower index), weights = softmax
// over the chosen logits alone.  One warp per token, lane 0 makes the choice.
__global__ void __launch_bounds__(32) route_top_kernel(const float* __restrict__ logits, int ldl, const float* __restrict__ bias,
                                                       int experts, int top, int* __restrict__ ids, float* __restrict__ wts,
                                                       int* __restrict__ counts) {
  pdl_begin();
  extern __shared__ __align__(16) unsigned char hy_smem[];
  float* s = reinterpret_cast<float*>(hy_smem);                // [experts] logits, -inf once chosen
  const int t = blockIdx.x, lane = threadIdx.x;
  for (int e = lane; e < experts; e += 32) s[e] = logits[(size_t)t * ldl + e] + (bias ? bias[e] : 0.0f);
  __syncwarp();
  if (lane != 0) return;
  float mx = 0.0f, sum = 0.0f;
  for (int k = 0; k < top; ++k) {
    int best = -1; float bv = -INFINITY;
    for (int e = 0; e < experts; ++e) if (s[e] > bv) { bv = s[e]; best = e; }
    if (best < 0) best = lowest_free(ids + (size_t)t * top, k);
    if (k == 0) mx = bv;                                       // the first choice is the largest: the softmax's maximum
    const float w = expf(bv - mx);
    ids[(size_t)t * top + k] = best;
    wts[(size_t)t * top + k] = w;
    sum += w;
    s[best] = -INFINITY;
    if (counts) atomicAdd(&counts[best], 1);
  }
  const float f = 1.0f / sum;
  for (int k = 0; k < top; ++k) wts[(size_t)t * top + k] *= f;
}

// A third way: softmax scores s over all `outputs` router outputs (experts, then identity experts), choice by the largest
// s + correction (ties to the lower index), weights = s of the chosen, not renormalised.  With groups > 1 only outputs of the
// `keep` groups of neighbouring outputs with the largest single choice score can be chosen.  Identity choices (index >= experts)
// take no row of the sorted order, so they are not counted.  One warp per token; every choice is a warp-wide maximum.
__global__ void __launch_bounds__(32) route_corrected_kernel(const float* __restrict__ logits, int ldl, const float* __restrict__ correction,
                                                             int experts, int outputs, int top, int groups, int keep, int* __restrict__ ids,
                                                             float* __restrict__ wts, int* __restrict__ counts) {
  pdl_begin();
  extern __shared__ __align__(16) unsigned char hy_smem[];
  float* s = reinterpret_cast<float*>(hy_smem);                // [outputs] scores
  float* ch = s + outputs;                                     // [outputs] choice scores, -inf once chosen
  float* gs = ch + outputs;                                    // [groups] largest choice score
  const int t = blockIdx.x, lane = threadIdx.x;
  const float* z = logits + (size_t)t * ldl;
  float mx = -INFINITY;
  for (int e = lane; e < outputs; e += 32) mx = fmaxf(mx, z[e]);
  mx = warp_max(mx);
  float sum = 0.0f;
  for (int e = lane; e < outputs; e += 32) { const float v = expf(z[e] - mx); s[e] = v; sum += v; }
  const float inv = 1.0f / warp_sum(sum);
  for (int e = lane; e < outputs; e += 32) { const float v = s[e] * inv; s[e] = v; ch[e] = v + correction[e]; }
  __syncwarp();
  if (groups > 1) {
    const int per = outputs / groups;
    for (int g = lane; g < groups; g += 32) {
      float m = -INFINITY;
      for (int i = 0; i < per; ++i) m = fmaxf(m, ch[g * per + i]);
      gs[g] = m;
    }
    __syncwarp();
    for (int g = lane; g < groups; g += 32) {
      int better = 0;                                          // groups that come before this one
      for (int i = 0; i < groups; ++i) better += gs[i] > gs[g] || (gs[i] == gs[g] && i < g);
      if (better >= keep)
        for (int i = 0; i < per; ++i) ch[g * per + i] = -INFINITY;
    }
    __syncwarp();
  }
  for (int k = 0; k < top; ++k) {
    float bv = -INFINITY; int best = 0x7fffffff;
    for (int e = lane; e < outputs; e += 32) if (ch[e] > bv) { bv = ch[e]; best = e; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oi = __shfl_xor_sync(0xffffffffu, best, o);
      if (ov > bv || (ov == bv && oi < best)) { bv = ov; best = oi; }
    }
    if (best >= outputs) best = lowest_free(ids + (size_t)t * top, k);      // the warp has seen lane 0's choices (__syncwarp below)
    if (lane == 0) {
      ids[(size_t)t * top + k] = best;
      wts[(size_t)t * top + k] = s[best];
      ch[best] = -INFINITY;
      if (counts && best < experts) atomicAdd(&counts[best], 1);
    }
    __syncwarp();
  }
}

// out[t, f] = act(in[t, f]) * in[t, n + f] (or the clamped pair, see gated_pair_f): the gated pair of a dense feed-forward whose gate and up rows are stacked.
template <typename AT>
__global__ void gated_act_kernel(const AT* __restrict__ in, int ldi, int n, int act, float limit, AT* __restrict__ out, int ldo) {
  pdl_begin();
  const int t = blockIdx.y;
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f < n) out[(size_t)t * ldo + f] = from_f<AT>(gated_pair_f(act, to_f(in[(size_t)t * ldi + f]), to_f(in[(size_t)t * ldi + n + f]), limit));
}

// The expert-sorted order.  One block per (token, choice) pair and one more: a pair's block finds the pair's row (behind the
// rows of the experts before its own, in order of arrival among its own) and copies the token's activation row there; the last block
// leaves the offsets, the tiles of tile_rows rows of one expert each (meta[0]: their number), and clears the counters of the
// routed layer before this one (most_experts of them; counts and fill of two layers alternate, so nobody clears what another
// block still reads).  A choice that is no expert (an identity choice) gets no row: pair_row -1.  vec: rows are copied 16 bytes
// at a time.  Offsets by one thread, the order, and rows fetched through it inside the products took 7 + 4 us and held the products
// back; this takes 11 us for 2048 tokens x 4 choices of 1024 channels.
constexpr int HY_XT = 64;
// Rows of a tile of expert_gemm_simt_kernel: most of a tile of 64 is padding where an expert has a handful of rows.  32 experts with ten rows each, width
// 256, of 128 (gate and up) and back: 33.6 and 9.8 us with 64 rows, 12.6 and 6.1 with 32.  A step of two layers, rows an expert, us with 64 -> 32: 10 218 -> 205,
// 16 233 -> 222, 24 264 -> 247, 31 282 -> 296, 50 314 -> 329.
inline int simt_tile_rows(int pairs, int experts) { return pairs <= 24 * experts ? 32 : HY_XT; }
template <typename AT>
__global__ void __launch_bounds__(128) route_place_kernel(int pairs, int top, int experts, int most_experts, int tile_rows,
                                                          const int* __restrict__ ids, const int* __restrict__ counts, int* __restrict__ fill,
                                                          int* __restrict__ old_counts, int* __restrict__ old_fill, const AT* __restrict__ h,
                                                          int width, int vec, int* __restrict__ offs, int* __restrict__ tile_expert,
                                                          int* __restrict__ tile_row0, int* __restrict__ meta, int* __restrict__ pair_row,
                                                          AT* __restrict__ rows) {
  pdl_begin();
  const int i = blockIdx.x, lane = threadIdx.x & 31;
  if (i == pairs) {
    for (int e = threadIdx.x; e < most_experts; e += blockDim.x) { old_counts[e] = 0; old_fill[e] = 0; }
    if (threadIdx.x >= 32) return;
    int at = 0, nt = 0;
    for (int e0 = 0; e0 < experts; e0 += 32) {                 // running sums of rows and of tiles, 32 experts at a time
      const int e = e0 + lane, n = e < experts ? counts[e] : 0, m = (n + tile_rows - 1) / tile_rows;
      int sn = n, sm = m;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, sn, s), c = __shfl_up_sync(0xffffffffu, sm, s);
        if (lane >= s) { sn += a; sm += c; }
      }
      if (e < experts) {
        offs[e] = at + sn - n;
        for (int r = 0; r < m; ++r) { tile_expert[nt + sm - m + r] = e; tile_row0[nt + sm - m + r] = at + sn - n + r * tile_rows; }
      }
      at += __shfl_sync(0xffffffffu, sn, 31);
      nt += __shfl_sync(0xffffffffu, sm, 31);
    }
    if (lane == 0) { offs[experts] = at; meta[0] = nt; }
    return;
  }
  const int e = ids[i];
  if (e >= experts) { if (threadIdx.x == 0) pair_row[i] = -1; return; }
  __shared__ int srow;
  if (threadIdx.x < 32) {
    int before = 0;
    for (int k = lane; k < e; k += 32) before += counts[k];
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) before += __shfl_xor_sync(0xffffffffu, before, s);
    if (lane == 0) { srow = before + atomicAdd(&fill[e], 1); pair_row[i] = srow; }
  }
  __syncthreads();
  const AT* src = h + (size_t)(i / top) * width;
  AT* dst = rows + (size_t)srow * width;
  if (vec) {
    constexpr int CH = 16 / (int)sizeof(AT);
    for (int k = threadIdx.x; k < width / CH; k += blockDim.x) reinterpret_cast<uint4*>(dst)[k] = reinterpret_cast<const uint4*>(src)[k];
  } else {
    for (int k = threadIdx.x; k < width; k += blockDim.x) dst[k] = src[k];
  }
}

// Grouped product over the sorted rows: C[row, n] = sum_k A[row, k] W_e[n, k], e the expert of the row's tile.
// GLU: W_e is [2 N, K] (gate rows, then up rows) and the result is the gated pair (see gated_pair_f); without GLU the result passes through
// the activation when act >= 0 (act: 0 silu, 1 tanh-gelu, 2 erf-gelu; see act_f).  Tiled SIMT, fp32 FMAs in k order: both builds can use it.
// Bound by the chain of its k blocks (few rows per expert): the next block travels while this one is summed up, and 32 columns per block give
// twice the blocks of 64; two layers of 77 tokens x 2 experts, width 256: 134 -> 44 us.
template <typename TA, typename TW, typename TO, bool GLU, int BM>
__global__ void __launch_bounds__(256) expert_gemm_simt_kernel(const TA* __restrict__ A, int lda,
                                                               const TW* __restrict__ W, size_t w_stride, int N, int K,
                                                               const int* __restrict__ offs, const int* __restrict__ tile_expert,
                                                               const int* __restrict__ tile_row0, const int* __restrict__ meta,
                                                               TO* __restrict__ out, int ldo, int act, float limit) {
  pdl_begin();
  constexpr int BN = 32, R = BM / 16, C = BN / 16, NA = BM * SIMT_BK / 1024;
  static_assert(BM % 32 == 0 && (R == 2 || R == 4), "a thread's rows are one read of two or four");
  __shared__ __align__(16) float As[2][SIMT_BK][BM];
  __shared__ __align__(16) float Ws[2][GLU ? 2 : 1][SIMT_BK][BN];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int lr = threadIdx.x / 8, lk = threadIdx.x % 8 * 4;
  const int n0 = blockIdx.x * BN, n = n0 + lr;
  const bool av = simt_vec(A, lda, K), wv = simt_vec(W, K, K) && w_stride % 4 == 0;
  for (int tile = blockIdx.y; tile < meta[0]; tile += gridDim.y) {
    const int e = tile_expert[tile], r0 = tile_row0[tile];
    const int rows = min(BM, offs[e + 1] - r0);
    const TW* We = W + (size_t)e * w_stride;
    float4 ra[NA], rw[GLU ? 2 : 1];
    auto fetch = [&](int k0) {
#pragma unroll
      for (int i = 0; i < NA; ++i) ra[i] = simt_load(A + (size_t)(r0 + lr + 32 * i) * lda, k0 + lk, K, lr + 32 * i < rows, av);
      rw[0] = simt_load(We + (size_t)n * K, k0 + lk, K, n < N, wv);
      if (GLU) rw[GLU ? 1 : 0] = simt_load(We + (size_t)(N + n) * K, k0 + lk, K, n < N, wv);
    };
    auto put = [&](int buf) {
#pragma unroll
      for (int i = 0; i < NA; ++i) simt_put<BM>(As[buf], lk, lr + 32 * i, ra[i]);
#pragma unroll
      for (int g = 0; g < (GLU ? 2 : 1); ++g) simt_put<BN>(Ws[buf][g], lk, lr, rw[g]);
    };
    float2 acc[R][C / 2] = {}, acc2[GLU ? R : 1][C / 2] = {};
    fetch(0);
    put(0);                                                    // the tile before ended with a barrier behind its last read
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += SIMT_BK, buf ^= 1) {
      const bool more = k0 + SIMT_BK < K;
      if (more) fetch(k0 + SIMT_BK);
      simt_block<BM, BN, R, C>(As[buf], Ws[buf][0], ty, tx, acc);
      if constexpr (GLU) simt_block<BM, BN, R, C>(As[buf], Ws[buf][1], ty, tx, acc2);
      if (more) put(buf ^ 1);
      __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = ty * R + i;
      if (r >= rows) continue;
#pragma unroll
      for (int j = 0; j < C; ++j) {
        const int c = n0 + tx * C + j;
        if (c >= N) continue;
        const float2 pa = acc[i][j / 2], pu = acc2[GLU ? i : 0][j / 2];
        const float va = j & 1 ? pa.y : pa.x, vu = j & 1 ? pu.y : pu.x;
        const float v = GLU ? gated_pair_f(act, va, vu, limit) : act >= 0 ? act_f(act, va) : va;
        out[(size_t)(r0 + r) * ldo + c] = from_f<TO>(v);
      }
    }
  }
}

// Few pairs (decode steps): one block row per pair, a warp per output column, the expert's weight rows streamed 16 bytes
// per lane; the pair's activation row is staged in shared memory.  pair = (token, choice); no sorted order is needed:
// A row = row_map ? row_map[pair] : pair, expert = ids[pair], output row = pair.  A choice that is no expert has no row.
template <typename TA, typename TW, typename TO, bool GLU>
__global__ void __launch_bounds__(256) expert_rows_kernel(const TA* __restrict__ A, int lda, const int* __restrict__ ids, int top,
                                                          int a_per_token, int experts, const TW* __restrict__ W, size_t w_stride,
                                                          int N, int K, TO* __restrict__ out, int ldo, int act, float limit) {
  pdl_begin();
  extern __shared__ __align__(16) unsigned char hy_smem[];
  TA* As = reinterpret_cast<TA*>(hy_smem);
  constexpr int VEC = 16 / sizeof(TW);
  const int pair = blockIdx.y;
  if (ids[pair] >= experts) return;
  const TA* ar = A + (size_t)(a_per_token ? pair / top : pair) * lda;
  for (int k = threadIdx.x; k < K; k += blockDim.x) As[k] = ar[k];
  __syncthreads();
  const TW* We = W + (size_t)ids[pair] * w_stride;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool vec_ok = K % VEC == 0 && (reinterpret_cast<uintptr_t>(We) & 15) == 0;
  for (int n = blockIdx.x * 8 + warp; n < N; n += gridDim.x * 8) {
    float acc = 0.0f, acc2 = 0.0f;
    const TW* wr = We + (size_t)n * K;
    const TW* ur = We + (size_t)(N + n) * K;
    if (vec_ok) {
#pragma unroll 2
      for (int k = lane * VEC; k < K; k += 32 * VEC) {
        const VecN<TW, VEC> wv = *reinterpret_cast<const VecN<TW, VEC>*>(wr + k);
        VecN<TW, VEC> uv;
        if (GLU) uv = *reinterpret_cast<const VecN<TW, VEC>*>(ur + k);
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
          const float a = to_f(As[k + j]);
          acc = fmaf(a, to_f(wv.v[j]), acc);
          if (GLU) acc2 = fmaf(a, to_f(uv.v[j]), acc2);
        }
      }
    } else {
      for (int k = lane; k < K; k += 32) {
        const float a = to_f(As[k]);
        acc = fmaf(a, to_f(wr[k]), acc);
        if (GLU) acc2 = fmaf(a, to_f(ur[k]), acc2);
      }
    }
    acc = warp_sum(acc);
    if (GLU) acc2 = warp_sum(acc2);
    if (lane == 0) out[(size_t)pair * ldo + n] = from_f<TO>(GLU ? gated_pair_f(act, acc, acc2, limit) : act >= 0 ? act_f(act, acc) : acc);
  }
}

// x[t] += ls * (tanh(alpha y) w + b),  y = sum_k wts[t, k] rows[pair_row ? pair_row[t top + k] : t top + k]  (k in order).
// post.w == NULL: x[t] += y (designs without an output norm on the feed-forward).
// next.w != NULL: the updated stream also leaves through the next layer's input norm into next_out [T, width].
template <typename AT, int V>
__global__ void expert_combine_kernel(const float* __restrict__ rows, int ldr, const int* __restrict__ pair_row,
                                      const float* __restrict__ wts, int top, int width, TanhNorm post,
                                      const float* __restrict__ ls, float* __restrict__ x, TanhNorm next,
                                      AT* __restrict__ next_out) {
  pdl_begin();
  const int t = blockIdx.x;
  for (int c = threadIdx.x * V; c < width; c += blockDim.x * V) {
    float y[V] = {}, f[V], w[V], b[V];
#pragma unroll 4
    for (int k = 0; k < top; ++k) {
      const int i = t * top + k;
      load_f(f, rows + (size_t)(pair_row ? pair_row[i] : i) * ldr + c);
      const float wt = wts[i];
#pragma unroll
      for (int j = 0; j < V; ++j) y[j] = fmaf(wt, f[j], y[j]);
    }
    if (post.w) {
      load_f(f, ls + c); load_f(w, post.w + c); load_f(b, post.b + c);
#pragma unroll
      for (int j = 0; j < V; ++j) y[j] = f[j] * fmaf(tanhf(post.alpha * y[j]), w[j], b[j]);
    }
    load_f(f, x + (size_t)t * width + c);
#pragma unroll
    for (int j = 0; j < V; ++j) f[j] += y[j];
    store_f(x + (size_t)t * width + c, f);
    if (next.w) {
      load_f(w, next.w + c); load_f(b, next.b + c);
#pragma unroll
      for (int j = 0; j < V; ++j) y[j] = fmaf(tanhf(next.alpha * f[j]), w[j], b[j]);
      store_f(next_out + (size_t)t * width + c, y);
    }
  }
}

}  // namespace hy
