// hy_kernels.cuh — device kernels of the layered hybrid decoders (libjf_hybrid.so).
//
// Precision rule shared by every kernel here: the residual stream, norms, attention scores and weights, positions and
// angles, recurrent states, decays, step sizes, gates of a recurrence and unit norms are fp32; projections, short
// convolutions with their activations and the operands of the matrix products are AT (bf16 in the serving build, fp32 in
// the all-fp32 build).  A step is a packed batch of entries (portions of prompts beside single decoded tokens).  A request's
// result depends on how it was cut and on what else is in the batch only by the rounding of its sums: the sizes of a step choose the kernel
// of a product (up to eight rows, or tiles), into how many ranges of k the tiles of a small product are cut, how many key ranges
// attention is split into and merged from, and the form of latent attention; within each of them the order of a sum is fixed (key
// ranges at absolute positions, k in order).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "jf_pair.cuh"

namespace hy {

typedef __nv_bfloat16 bf16;

// Every kernel of a step may start while the one before it still runs (see go_kernel; jf_pair.cuh has the two instructions).
using jf::pdl_trigger;
using jf::pdl_wait;
__device__ __forceinline__ void pdl_begin() { pdl_trigger(); pdl_wait(); }
// Ahead of pdl_wait a kernel of a step may read weights, the step's batch (its copy is over before the step's first kernel begins) and what a recurrence or
// convolution keeps of a request between steps: of a layer's run that is read and written by one kernel of a step, where launches overlap.

template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<bf16>(bf16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ bf16 from_f<bf16>(float v) { return __float2bfloat16_rn(v); }

template <typename T, int N>
struct alignas(sizeof(T) * N < 16 ? sizeof(T) * N : 16) VecN { T v[N]; };

// 1 / (1 + exp(-z)), the reciprocal by one step of Newton's iteration on the approximate one (1 ulp, squared by the step): IEEE division gives
// the same to half an ulp, but has a branch for the divisors that do not occur here, which keeps neighbouring elements of a loop from overlapping.
// The divisor is a quarter of the sum, so that its reciprocal is a normal number where the value is below 2^-126 (z below -87.3) too: silu of such a z
// is a normal number again.  exp(-z) is infinite below z = -88.72, where the value is zero and the step would have none.
// Whole steps, us, division -> this: 2048 tokens of state-space and forget-gate layers 773 -> 757,
// 1999 of retention and delta rule 808 -> 791, fp32 of 77 tokens 267 -> 255; where products bound a step, the same.  The quarter takes 2 to 5 us of the
// first two back (kernels: forget rows 11.8 -> 12.4, convolutions 18.4 -> 18.9, gate and up's epilogue 92.5 -> 94.4).
__device__ __forceinline__ float sigmoid_f(float z) {
  const float d = fmaf(expf(-z), 0.25f, 0.25f);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  return d > 8.5070592e37f ? 0.0f : 0.25f * fmaf(r, fmaf(-d, r, 1.0f), r);
}
__device__ __forceinline__ float silu_f(float z) { return z * sigmoid_f(z); }
__device__ __forceinline__ float softplus_f(float z) { return z > 20.0f ? z : log1pf(expf(z)); }
__device__ __forceinline__ float log_sigmoid_f(float z) { return fminf(z, 0.0f) - log1pf(expf(-fabsf(z))); }
__device__ __forceinline__ float gelu_tanh_f(float z) { return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z))); }
__device__ __forceinline__ float gelu_erf_f(float z) { return 0.5f * z * (1.0f + erff(z * 0.7071067811865476f)); }
// activation by kind: 0 silu, 1 the tanh form of gelu, 2 gelu with the error function
__device__ __forceinline__ float act_f(int kind, float z) { return kind == 1 ? gelu_tanh_f(z) : kind == 2 ? gelu_erf_f(z) : silu_f(z); }
// a gated pair by kind: act(gate) * up, or (kind 3) the clamped pair g = min(gate, limit), u = clamp(up, -limit, limit),
// g sigmoid(1.702 g) (u + 1)
__device__ __forceinline__ float gated_pair_f(int kind, float g, float u, float limit) {
  if (kind == 3) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return g * sigmoid_f(1.702f * g) * (u + 1.0f);
  }
  return act_f(kind, g) * u;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// Sum over the block; every thread gets the result.  red: >= 33 floats of shared memory.  Deterministic order.
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  if (w == 0) {
    float s = lane < nw ? red[lane] : 0.0f;
    s = warp_sum(s);
    if (lane == 0) red[32] = s;
  }
  __syncthreads();
  return red[32];
}

// Per-step batch description (device pointers, all int32).
struct Batch {
  const int* tok;        // [T] token ids
  const int* tok_ent;    // [T] entry of a token
  const int* tok_pos;    // [T] absolute position in its request
  const int* ent_start;  // [E + 1]
  const int* ent_pos0;   // [E]
  const int* ent_slot;   // [E]
  const int* pages;      // [E, max_pages]
  int T, E, max_pages, page_size;
};

// ---- embedding: table row times a scale, plus the sinusoid of the position ----------------------------------------------
// entry 2i = sin(p f_i), entry 2i+1 = cos(p f_i); f_i = 10000^(-2i / width) comes from a host-made fp64 table and the angle
// is formed and reduced in fp64 (at position 1000 an fp32 angle is already 6e-5 off), the result enters the fp32 stream.
// inv_freq == NULL: no positional term (designs whose positions enter through a rotation inside attention).
template <typename WT>
__global__ void embed_kernel(Batch b, const WT* __restrict__ table, const double* __restrict__ inv_freq, float scale,
                             int width, float* __restrict__ x) {
  pdl_begin();
  const int t = blockIdx.x;
  const int tok = b.tok[t];
  const double p = (double)b.tok_pos[t];
  // a pair of channels shares its angle, and the reduction of it to a quadrant is most of what sine and cosine take
  for (int c = 2 * threadIdx.x; c < width; c += 2 * blockDim.x) {
    double sn = 0.0, cs = 0.0;
    if (inv_freq) sincos(p * inv_freq[c >> 1], &sn, &cs);
    x[(size_t)t * width + c] = to_f(table[(size_t)tok * width + c]) * scale + (float)sn;
    if (c + 1 < width) x[(size_t)t * width + c + 1] = to_f(table[(size_t)tok * width + c + 1]) * scale + (float)cs;
  }
}

// ---- rows V elements at a time ------------------------------------------------------------------------------------------------------------
// The kernels over rows below take V = 4 elements per thread (16 bytes of fp32) where sizes and leading dimensions are multiples of four and rows begin on
// 16 (fp32) or 8 bytes, else one: with one element, too few bytes were in flight: 2048 rows, us, one -> four:
// RMS norm of 2048 channels 10.5 -> 5.3, output norm and gate of 2048 columns 17.0 -> 12.1, forget-gate rows of 1024 columns 11.4 -> 6.8, gated group
// norm of 2048 columns 24 -> 19.1, mixture of four experts' rows of 1024 channels 15.5 -> 9.2.  Positions of the embedding: 29.5 -> 12.4.
template <typename T, int V>
__device__ __forceinline__ void load_f(float (&f)[V], const T* p) {
  const VecN<T, V> v = *reinterpret_cast<const VecN<T, V>*>(p);
#pragma unroll
  for (int i = 0; i < V; ++i) f[i] = to_f(v.v[i]);
}
template <typename T, int V>
__device__ __forceinline__ void store_f(T* p, const float (&f)[V]) {
  VecN<T, V> v;
#pragma unroll
  for (int i = 0; i < V; ++i) v.v[i] = from_f<T>(f[i]);
  *reinterpret_cast<VecN<T, V>*>(p) = v;
}

// ---- element-wise tanh norm: tanh(alpha x) w + b, no statistics ------------------------------------------------------------
// rows: NULL = row r of x, else x row rows[r].  Parameters are fp32.
struct TanhNorm { const float* w; const float* b; float alpha; };
template <typename OT, int V>
__global__ void tanh_norm_kernel(const float* __restrict__ x, const int* __restrict__ rows, TanhNorm n, int width,
                                 OT* __restrict__ out) {
  pdl_begin();
  const int r = blockIdx.x;
  const float* xr = x + (size_t)(rows ? rows[r] : r) * width;
  for (int c = threadIdx.x * V; c < width; c += blockDim.x * V) {
    float v[V], w[V], b[V];
    load_f(v, xr + c); load_f(w, n.w + c); load_f(b, n.b + c);
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = fmaf(tanhf(n.alpha * v[i]), w[i], b[i]);
    store_f(out + (size_t)r * width + c, v);
  }
}

// ---- RMS norm; the weight is w_offset + w (1: stored as an offset from one, 0: plain) -----------------------------------------
// rows: NULL = row r of x, else x row rows[r].  out row r.
template <typename WT, typename OT, int V>
__global__ void rmsnorm_kernel(const float* __restrict__ x, const int* __restrict__ rows, const WT* __restrict__ w,
                               float eps, int width, float w_offset, OT* __restrict__ out) {
  pdl_begin();
  __shared__ float red[33];
  const int r = blockIdx.x;
  const float* xr = x + (size_t)(rows ? rows[r] : r) * width;
  float ss = 0.0f;
  for (int c = threadIdx.x * V; c < width; c += blockDim.x * V) {
    float v[V];
    load_f(v, xr + c);
#pragma unroll
    for (int i = 0; i < V; ++i) ss += v[i] * v[i];
  }
  ss = block_sum(ss, red);
  const float inv = 1.0f / sqrtf(ss / (float)width + eps);
  for (int c = threadIdx.x * V; c < width; c += blockDim.x * V) {
    float v[V], g[V];
    load_f(v, xr + c); load_f(g, w + c);
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = v[i] * inv * (w_offset + g[i]);
    store_f(out + (size_t)r * width + c, v);
  }
}

// ---- generic matrix product C[t, n] = sum_k A[t, k] W[n, k], fp32 accumulation in k order -----------------------------------
// Destinations: resid != NULL: resid[t, n] += alpha * c (fp32, the residual stream).  Otherwise columns < split go to
// out1[t * ld1 + n], columns >= split to out2[t * ld2 + n - split], squared ReLU first when act2 (the feed-forward's
// hidden activation leaves the merged input projection already activated).  With post_w set, the residual receives
// post_ls[n] * (tanh(post_alpha c) post_w[n] + post_b[n]): a sublayer's output norm (element-wise, so it needs no second
// pass) and its layer scale, applied to the fp32 accumulator.
// With next_w set as well, the element of the updated residual also leaves through the NEXT sublayer's input norm
// (tanh(next_alpha x) next_w[n] + next_b[n]) into next_out [T, ldr] in the activation type: no separate norm launch.
// act2 == 3: every column passes through the activation act_kind (act_f) before it is stored.  out2_f32: the columns from
// `split` on leave as fp32 whatever the output type (gate pre-activations of a recurrence beside its bf16 operands).
// bias: added to the scaled accumulator of column n before anything else (projections with biases).  act_limit: the limit
// of the clamped gated pair (act2 == 2 with act_kind 3).
// act2 == 4: every column leaves as sigmoid(c)^act_limit (the decays of a recurrence, formed as exp(act_limit log sigmoid)).
// act2 == 5 (tensor-core product only): the columns [pair_lo, pair_hi) (multiples of 32) are gated pairs in alternating
// blocks of 16, as with act2 == 2, and leave activated through pair_out (pair_n features); the others as without act2.
struct GemmOut {
  void* out1; int ld1; int split; void* out2; int ld2; int act2;
  float* resid; int ldr; float alpha;
  const float* post_w; const float* post_b; const float* post_ls; float post_alpha;
  const float* next_w; const float* next_b; float next_alpha; void* next_out; int next_f32;
  int act_kind; int out2_f32;
  const float* bias; float act_limit;
  int pair_lo, pair_hi; void* pair_out; int ld_pair, pair_n;
};

template <typename TO>
__device__ __forceinline__ void gemm_store(const GemmOut& o, int t, int n, float c) {
  c *= o.alpha;
  if (o.bias) c += o.bias[n];
  if (o.resid) {
    if (o.post_w) c = o.post_ls[n] * fmaf(tanhf(o.post_alpha * c), o.post_w[n], o.post_b[n]);
    const float v = o.resid[(size_t)t * o.ldr + n] + c;
    o.resid[(size_t)t * o.ldr + n] = v;
    if (o.next_w) {
      const float y = fmaf(tanhf(o.next_alpha * v), o.next_w[n], o.next_b[n]);
      if (o.next_f32) ((float*)o.next_out)[(size_t)t * o.ldr + n] = y;
      else ((bf16*)o.next_out)[(size_t)t * o.ldr + n] = __float2bfloat16_rn(y);
    }
    return;
  }
  if (o.act2 == 3) c = act_f(o.act_kind, c);
  else if (o.act2 == 4) c = expf(o.act_limit * log_sigmoid_f(c));
  if (n < o.split) { ((TO*)o.out1)[(size_t)t * o.ld1 + n] = from_f<TO>(c); return; }
  if (o.act2 == 1) { c = fmaxf(c, 0.0f); c = c * c; }
  if (o.out2_f32) ((float*)o.out2)[(size_t)t * o.ld2 + (n - o.split)] = c;
  else ((TO*)o.out2)[(size_t)t * o.ld2 + (n - o.split)] = from_f<TO>(c);
}

// ---- RMS norm on a sublayer's output, layer scale and the residual sum --------------------------------------------------------
// x[t] <- (add ? x[t] : 0) + ls * y[t] / sqrt(mean(y[t]^2) + eps) * w   (ls == NULL: one), and the updated row also leaves
// in the activation type (the next sublayer reads the stream itself).  y[t] is row t of ybuf, or, when `rows` is given,
// the mixture of a routed feed-forward: sum_k wts[t, k] rows[pair_row ? pair_row[t top + k] : t top + k] in the order of
// the token's choices, plus shared_rows[t] (an expert every token uses) when given.  ybuf may be x itself (add = 0).
template <typename AT>
__global__ void post_norm_add_kernel(const float* ybuf, int ldy, const float* __restrict__ rows, int ldr,
                                     const int* __restrict__ pair_row, const float* __restrict__ wts, int top,
                                     const float* __restrict__ shared_rows, const float* __restrict__ w,
                                     const float* __restrict__ ls, float eps, int width, int add, float* x,
                                     AT* __restrict__ next_out) {
  pdl_begin();
  extern __shared__ __align__(16) unsigned char hy_smem[];
  float* ys = reinterpret_cast<float*>(hy_smem);               // [width]
  __shared__ float red[33];
  const int t = blockIdx.x;
  float ss = 0.0f;
  for (int c = threadIdx.x; c < width; c += blockDim.x) {
    float y;
    if (rows) {
      y = 0.0f;
      for (int k = 0; k < top; ++k) {
        const int i = t * top + k;
        y = fmaf(wts[i], rows[(size_t)(pair_row ? pair_row[i] : i) * ldr + c], y);
      }
      if (shared_rows) y += shared_rows[(size_t)t * ldr + c];
    } else {
      y = ybuf[(size_t)t * ldy + c];
    }
    ys[c] = y;
    ss = fmaf(y, y, ss);
  }
  ss = block_sum(ss, red);
  const float inv = w ? 1.0f / sqrtf(ss / (float)width + eps) : 1.0f;      // w == NULL: no norm, the row passes as it is
  for (int c = threadIdx.x; c < width; c += blockDim.x) {
    const float n = ys[c] * inv * (w ? w[c] : 1.0f) * (ls ? ls[c] : 1.0f);
    const float v = add ? x[(size_t)t * width + c] + n : n;
    x[(size_t)t * width + c] = v;
    if (next_out) next_out[(size_t)t * width + c] = from_f<AT>(v);
  }
}

// Two fp32 lanes per instruction: the same roundings as two scalar ones at half the issue slots.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(reinterpret_cast<unsigned long long&>(d)) : "l"(reinterpret_cast<const unsigned long long&>(a)),
      "l"(reinterpret_cast<const unsigned long long&>(b)), "l"(reinterpret_cast<const unsigned long long&>(c)));
  return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<unsigned long long&>(d)) : "l"(reinterpret_cast<const unsigned long long&>(a)),
      "l"(reinterpret_cast<const unsigned long long&>(b)));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<unsigned long long&>(d)) : "l"(reinterpret_cast<const unsigned long long&>(a)),
      "l"(reinterpret_cast<const unsigned long long&>(b)));
  return d;
}

// The SIMT products' operand tile [rows][32 k], staged k-major in shared memory: a thread carries four k of a row per load, and the rows are
// permuted by groups of four with k / 4, so that the transposing stores and the 16-byte reads along the rows are free of conflicts.
constexpr int SIMT_BK = 32;
__device__ __forceinline__ int simt_at(int k, int r) { return r ^ (((k >> 2) & 7) << 2); }
template <typename T>
__device__ __forceinline__ float4 simt_load(const T* row, int k, int K, bool ok, bool vec) {
  float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (!ok || k >= K) return x;
  if (vec) {
    const VecN<T, 4> v = *reinterpret_cast<const VecN<T, 4>*>(row + k);
    return make_float4(to_f(v.v[0]), to_f(v.v[1]), to_f(v.v[2]), to_f(v.v[3]));
  }
  x.x = to_f(row[k]);
  if (k + 1 < K) x.y = to_f(row[k + 1]);
  if (k + 2 < K) x.z = to_f(row[k + 2]);
  if (k + 3 < K) x.w = to_f(row[k + 3]);
  return x;
}
// four k at a time by one load: every row starts on the load's own size
template <typename T>
__device__ __forceinline__ bool simt_vec(const T* base, size_t ld, int K) {
  return K % 4 == 0 && ld % 4 == 0 && (reinterpret_cast<uintptr_t>(base) & (4 * sizeof(T) - 1)) == 0;
}
template <int ROWS>
__device__ __forceinline__ void simt_put(float (*tile)[ROWS], int k, int r, float4 x) {
  const int at = simt_at(k, r);
  tile[k][at] = x.x; tile[k + 1][at] = x.y; tile[k + 2][at] = x.z; tile[k + 3][at] = x.w;
}
// one staged k block: acc[i][j] += a[R ty + i] w[C tx + 2 j ..], in k order
template <int BM, int BN, int R, int C>
__device__ __forceinline__ void simt_block(const float (*As)[BM], const float (*Ws)[BN], int ty, int tx, float2 (&acc)[R][C / 2]) {
#pragma unroll
  for (int kk = 0; kk < SIMT_BK; ++kk) {
    const VecN<float, R> a = *reinterpret_cast<const VecN<float, R>*>(&As[kk][simt_at(kk, ty * R)]);
    const VecN<float, C> w = *reinterpret_cast<const VecN<float, C>*>(&Ws[kk][simt_at(kk, tx * C)]);
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < C / 2; ++j) acc[i][j] = fma2(make_float2(a.v[i], a.v[i]), make_float2(w.v[2 * j], w.v[2 * j + 1]), acc[i][j]);
  }
}

// Tiled SIMT kernel: any shape, any leading dimensions; the all-fp32 build's matrix product (true fp32 FMAs in k order).  The next k block
// travels in registers while this one is summed up, one barrier per block.  The seven
// products of 77 tokens at width 256 took 337 us with a 16-wide k block that every step waited for, 62 now; few tiles leave SMs idle, so they
// are 32 wide there (see gemm).
template <typename TA, typename TW, typename TO, int BM>
__global__ void __launch_bounds__(256) gemm_simt_kernel(const TA* __restrict__ A, int lda, const TW* __restrict__ W, int ldw,
                                                        int T, int N, int K, GemmOut o) {
  pdl_begin();
  constexpr int R = BM / 16, NV = BM * SIMT_BK / 1024;
  __shared__ __align__(16) float As[2][SIMT_BK][BM];
  __shared__ __align__(16) float Ws[2][SIMT_BK][BM];
  const int t0 = blockIdx.y * BM, n0 = blockIdx.x * BM;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;     // tx: R columns, ty: R rows
  const int lr = threadIdx.x / 8, lk = threadIdx.x % 8 * 4;   // loads: rows lr, lr + 32, four k from lk
  const bool av = simt_vec(A, lda, K), wv = simt_vec(W, ldw, K);
  float4 ra[NV], rw[NV];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int t = t0 + lr + 32 * i, n = n0 + lr + 32 * i;
      ra[i] = simt_load(A + (size_t)t * lda, k0 + lk, K, t < T, av);
      rw[i] = simt_load(W + (size_t)n * ldw, k0 + lk, K, n < N, wv);
    }
  };
  auto put = [&](int buf) {
#pragma unroll
    for (int i = 0; i < NV; ++i) { simt_put<BM>(As[buf], lk, lr + 32 * i, ra[i]); simt_put<BM>(Ws[buf], lk, lr + 32 * i, rw[i]); }
  };
  float2 acc[R][R / 2] = {};
  fetch(0);
  put(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < K; k0 += SIMT_BK, buf ^= 1) {
    const bool more = k0 + SIMT_BK < K;
    if (more) fetch(k0 + SIMT_BK);
    simt_block<BM, BM, R, R>(As[buf], Ws[buf], ty, tx, acc);
    if (more) put(buf ^ 1);                                    // its last readers passed the barrier below a block ago
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int t = t0 + ty * R + i;
    if (t >= T) continue;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int n = n0 + tx * R + j;
      if (n < N) gemm_store<TO>(o, t, n, j & 1 ? acc[i][j / 2].y : acc[i][j / 2].x);
    }
  }
}

// Few-row kernel (decode steps): the weight matrix is streamed once, 16 bytes per lane per load, four loads in flight per
// lane; one warp owns one output column for up to ROWS rows; the rows' operand sits in shared memory in its own type and
// is read back 16 bytes at a time (conflict-free).  K order: lane-strided partial sums, then an xor tree.

template <typename TA, typename TW, typename TO, int ROWS>
__global__ void __launch_bounds__(256) gemm_rows_kernel(const TA* __restrict__ A, int lda, const TW* __restrict__ W, int ldw,
                                                        int T, int N, int K, int ksplit, GemmOut o) {
  extern __shared__ __align__(16) unsigned char hy_smem[];
  __shared__ float parts[8][ROWS];
  TA* As = reinterpret_cast<TA*>(hy_smem);                     // [ROWS][Kp], Kp = K rounded up to the vector width
  constexpr int VEC = 16 / sizeof(TW);
  const int Kp = (K + VEC - 1) / VEC * VEC;
  const int t0 = blockIdx.y * ROWS;
  pdl_trigger();
  // ksplit warps share a column (long k, few columns: more loads in flight); their sums are added in part order
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cpb = 8 / ksplit, part = warp % ksplit, cib = warp / ksplit;
  const int Kc = ((K + ksplit - 1) / ksplit + 32 * VEC - 1) / (32 * VEC) * (32 * VEC);
  const int lo = part * Kc, hi = min(K, lo + Kc), kv = min(hi, K / VEC * VEC);
  // Up to four rows: the first AHEAD vectors of a column travel while the columns before it are summed up; those of the warp's first column
  // while the kernel before this one ends (weights do not depend on it).  What they hold in registers is paid for in blocks per SM: behind a small
  // kernel, N 2112, K 2048, us: one row 10.3 without overlapping launches, 8.2 with four vectors ahead (80 registers), 6.5 with two (48); eight rows
  // 22.5, 24.9 with four (128 registers, two blocks per SM), 25.0 with two, 16.9 with none (62).
  constexpr int AHEAD = ROWS <= 4 ? 2 : 0;
  VecN<TW, VEC> w0[AHEAD ? AHEAD : 1];
  auto fetch = [&](int n) {
    const TW* wr = W + (size_t)n * ldw;
    if (AHEAD && n < N && (reinterpret_cast<uintptr_t>(wr) & 15) == 0) {
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) {
        const int k = lo + (lane + 32 * i) * VEC;
        if (k < kv) w0[i] = *reinterpret_cast<const VecN<TW, VEC>*>(wr + k);
      }
    }
  };
  fetch(blockIdx.x * cpb + cib);
  pdl_wait();
  constexpr int VA = 16 / sizeof(TA);
  if (K % VA == 0 && lda % VA == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0 && Kp == K) {
    const int kv = K / VA;                                     // 16 bytes per thread per load
    for (int i = threadIdx.x; i < ROWS * kv; i += blockDim.x) {
      const int r = i / kv, k = (i % kv) * VA;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (t0 + r < T) v = *reinterpret_cast<const uint4*>(A + (size_t)(t0 + r) * lda + k);
      *reinterpret_cast<uint4*>(As + r * Kp + k) = v;
    }
  } else {
    for (int i = threadIdx.x; i < ROWS * Kp; i += blockDim.x) {
      const int r = i / Kp, k = i % Kp;
      As[i] = (t0 + r < T && k < K) ? A[(size_t)(t0 + r) * lda + k] : from_f<TA>(0.0f);
    }
  }
  __syncthreads();
  for (int base = blockIdx.x * cpb; base < N; base += gridDim.x * cpb) {
    const int n = base + cib;
    float acc[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) acc[r] = 0.0f;
    if (n < N) {
      const TW* wr = W + (size_t)n * ldw;
      const bool vec_ok = ((reinterpret_cast<uintptr_t>(wr) & 15) == 0);
      int kdone = lo;
      if (vec_ok) {
        auto add = [&](const VecN<TW, VEC>& wv, int k) {
#pragma unroll
          for (int r = 0; r < ROWS; ++r) {
            const VecN<TA, VEC> av = *reinterpret_cast<const VecN<TA, VEC>*>(As + r * Kp + k);
#pragma unroll
            for (int j = 0; j < VEC; ++j) acc[r] = fmaf(to_f(av.v[j]), to_f(wv.v[j]), acc[r]);
          }
        };
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
          const int k = lo + (lane + 32 * i) * VEC;
          if (k < kv) add(w0[i], k);
        }
        fetch(n + gridDim.x * cpb);
#pragma unroll 4
        for (int k = lo + (lane + 32 * AHEAD) * VEC; k < kv; k += 32 * VEC) add(*reinterpret_cast<const VecN<TW, VEC>*>(wr + k), k);
        kdone = max(lo, kv);
      }
      for (int k = kdone + lane; k < hi; k += 32) {
        const float w = to_f(wr[k]);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) acc[r] = fmaf(to_f(As[r * Kp + k]), w, acc[r]);
      }
#pragma unroll
      for (int r = 0; r < ROWS; ++r) acc[r] = warp_sum(acc[r]);
    }
    if (ksplit > 1) {
      if (lane == 0) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r) parts[warp][r] = acc[r];
      }
      __syncthreads();
      if (lane == 0 && part == 0) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          float v = 0.0f;
          for (int p = 0; p < ksplit; ++p) v += parts[warp + p][r];
          acc[r] = v;
        }
      }
    }
    if (lane == 0 && part == 0 && n < N) {
#pragma unroll
      for (int r = 0; r < ROWS; ++r)
        if (t0 + r < T) gemm_store<TO>(o, t0 + r, n, acc[r]);
    }
    if (ksplit > 1) __syncthreads();
  }
}

// ---- short causal convolution over time with a carried tail ------------------------------------------------------------------
// u [T, ldu] (columns col0 .. col0 + C), w [C, taps] (last tap = current token), state [slot][taps - 1][C] fp32 holds the
// last taps - 1 inputs of the request in time order.  Inputs before the request's start are zero.
// Where a column goes: [out_lo, out_hi) to out (from its column 0 on, activation type); [r_lo, r_lo + 2 G n) to fp32 rows
// [T][G][2 n], the operands of a matrix-state recurrence: the span's first half to the first n of a head's row, the second half
// to the last n (flip: the other way round); the columns from k_lo on (when cache is given: kv heads of dim) to their pages.
template <typename AT>
struct ConvOut {
  AT* out; int ldo, out_lo, out_hi;
  float* rows; int r_lo, G, n, flip;
  AT* cache; int k_lo, kv_heads, dim;
};
constexpr int HY_MAX_TAPS = 16;
constexpr int HY_CONV_TT = 16;                                 // tokens per thread: taps - 1 at most, so that only an entry's
                                                               // first chunk meets the carried tail
// V columns per thread (V = 4: every boundary above, C, col0 and the leading dimensions are multiples of 4), HY_CONV_TT tokens of
// one entry: weights and the last taps - 1 inputs stay in registers (TAPS = 0: any number of taps, inputs read again per tap).
// The thread of an entry's first chunk is the only one that reads the carried tail, so it also leaves the new one.
// One token and one column per thread with the tail, the cache rows and the unit vectors as kernels of their own took 63 us for
// 2048 tokens x 4096 columns (0.5 TB/s) and 4.5 us per launch in decode steps; this form 23 us and one launch.
template <typename AT, typename WT, int V, int TAPS>
__global__ void __launch_bounds__(128) conv_kernel(Batch b, const AT* __restrict__ u, int ldu, int col0, int C, int taps_, const WT* __restrict__ w,
                                                   const WT* __restrict__ bias, int act_silu, float* __restrict__ state, ConvOut<AT> o) {
  pdl_trigger();
  const int taps = TAPS ? TAPS : taps_;
  int e = 0, chunk = blockIdx.y, start, cnt;
  for (;; ++e) {                                               // entry and chunk of this block
    start = b.ent_start[e]; cnt = b.ent_start[e + 1] - start;
    const int n = (cnt + HY_CONV_TT - 1) / HY_CONV_TT;
    if (chunk < n) break;
    chunk -= n;
  }
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * V;
  if (c >= C) return;
  const int j0 = chunk * HY_CONV_TT, j1 = min(cnt, j0 + HY_CONV_TT), pos0 = b.ent_pos0[e];
  float* st = state + (size_t)b.ent_slot[e] * (taps - 1) * C + c;
  const AT* uc = u + (size_t)start * ldu + col0 + c;
  auto input = [&](int j, int k) {                             // column c + k of the entry's token j (j < 0: before the entry)
    if (j >= 0) return to_f(uc[(size_t)j * ldu + k]);
    return pos0 + j >= 0 ? st[(size_t)(taps - 1 + j) * C + k] : 0.0f;
  };
  constexpr int NW = TAPS > 1 ? TAPS - 1 : 1;
  float win[NW][V], wv[V][TAPS ? TAPS : 1], bv[V];
  auto window = [&] {
#pragma unroll
    for (int k = 0; k < V; ++k)
#pragma unroll
      for (int i = 0; i < TAPS - 1; ++i) win[i][k] = input(j0 - (TAPS - 1) + i, k);
  };
  // The entry, weights and an entry's first window come while the kernel before this one ends, as the states of recurrences do: a request of 24 tokens, one
  // each step, 7847 -> 7665 us, eight requests 8800 -> 8716.
#pragma unroll
  for (int k = 0; k < V; ++k) {
    bv[k] = bias ? to_f(bias[c + k]) : 0.0f;
#pragma unroll
    for (int i = 0; i < TAPS; ++i) wv[k][i] = to_f(w[(size_t)(c + k) * TAPS + i]);
  }
  if (j0 == 0) window();
  pdl_wait();
  if (j0 > 0) window();
#pragma unroll 4
  for (int j = j0; j < j1; ++j) {
    const int t = start + j;
    float y[V];
    if constexpr (TAPS > 0) {
      const VecN<AT, V> x = *reinterpret_cast<const VecN<AT, V>*>(uc + (size_t)j * ldu);
#pragma unroll
      for (int k = 0; k < V; ++k) {
        float acc = bv[k];
#pragma unroll
        for (int i = 0; i < TAPS - 1; ++i) acc = fmaf(wv[k][i], win[i][k], acc);
        const float xk = to_f(x.v[k]);
        y[k] = fmaf(wv[k][TAPS - 1], xk, acc);
#pragma unroll
        for (int i = 0; i + 1 < TAPS - 1; ++i) win[i][k] = win[i + 1][k];
        if (TAPS > 1) win[NW - 1][k] = xk;
      }
    } else {
#pragma unroll
      for (int k = 0; k < V; ++k) {
        y[k] = bv[k];
        for (int i = 0; i < taps; ++i) y[k] = fmaf(to_f(w[(size_t)(c + k) * taps + i]), input(j - (taps - 1) + i, k), y[k]);
      }
    }
    if (act_silu) {
#pragma unroll
      for (int k = 0; k < V; ++k) y[k] = silu_f(y[k]);
    }
    if (o.rows && c >= o.r_lo && c < o.r_lo + 2 * o.G * o.n) {
      const int r = c - o.r_lo, half = r >= o.G * o.n, g = (r - half * o.G * o.n) / o.n, k0 = r - half * o.G * o.n - g * o.n;
      float* p = o.rows + ((size_t)t * o.G + g) * 2 * o.n + (half ^ o.flip) * o.n + k0;
      *reinterpret_cast<VecN<float, V>*>(p) = *reinterpret_cast<VecN<float, V>*>(y);
      continue;
    }
    VecN<AT, V> q;
#pragma unroll
    for (int k = 0; k < V; ++k) q.v[k] = from_f<AT>(y[k]);
    if (o.cache && c >= o.k_lo) {
      const int g = (c - o.k_lo) / o.dim, d = (c - o.k_lo) % o.dim, pos = pos0 + j;
      const int page = b.pages[(size_t)e * b.max_pages + pos / b.page_size];
      *reinterpret_cast<VecN<AT, V>*>(o.cache + (((size_t)page * o.kv_heads + g) * b.page_size + pos % b.page_size) * o.dim + d) = q;
    } else if (c >= o.out_lo && c < o.out_hi) {
      *reinterpret_cast<VecN<AT, V>*>(o.out + (size_t)t * o.ldo + c - o.out_lo) = q;
    }
  }
  if (chunk == 0)
    for (int s = 0; s < taps - 1; ++s)                         // ascending: row s is read (as row cnt + s) only before it is written
#pragma unroll
      for (int k = 0; k < V; ++k) st[(size_t)s * C + k] = input(cnt - (taps - 1) + s, k);
}

// New tail = the last taps - 1 of (old tail ++ this entry's inputs).  Runs after the convolution of the same step.
template <typename AT>
__global__ void conv_tail_kernel(Batch b, const AT* __restrict__ u, int ldu, int col0, int C, int taps, float* __restrict__ state) {
  pdl_begin();
  const int e = blockIdx.y;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const int start = b.ent_start[e], cnt = b.ent_start[e + 1] - start, pos0 = b.ent_pos0[e];
  float* st = state + (size_t)b.ent_slot[e] * (taps - 1) * C;
  float nv[HY_MAX_TAPS];
  for (int s = 0; s < taps - 1; ++s) {
    const int i = cnt + s;                                   // index in old tail ++ inputs
    float v;
    if (i >= taps - 1) v = to_f(u[(size_t)(start + i - (taps - 1)) * ldu + col0 + c]);
    else v = (pos0 - (taps - 1) + i >= 0) ? st[(size_t)i * C + c] : 0.0f;
    nv[s] = v;
  }
  for (int s = 0; s < taps - 1; ++s) st[(size_t)s * C + c] = nv[s];
}

// first position that the query at p sees through a sliding window (0: no window)
__host__ __device__ __forceinline__ int first_seen(int p, int window) { return window > 0 && p - window + 1 > 0 ? p - window + 1 : 0; }

// ---- causal softmax attention with a sink; values are the keys -----------------------------------------------------------------
// One warp per (token, query head).  Keys are walked in groups of 32 aligned to absolute positions; the running maximum
// starts at the sink logit and the denominator at exp(sink - sink) = 1: the sink has no key and no value (sink NULL: an
// ordinary softmax).  The query is
// multiplied by its position's temperature in fp32.  The value of a key is its first vdim dimensions (vdim == dim: the
// values are the keys; vdim < dim: a latent followed by a part that only enters the score).  window > 0: only the keys j with
// pos - j < window.  Output: heads concatenated
// [H, vdim], times sigmoid(gate) when there is a gate, times out_scale.
constexpr int HY_ATT_MAXD = 20;     // dims per lane: dim <= 640
template <typename AT, typename WT, typename OT>
__global__ void __launch_bounds__(128) attn_sink_kernel(Batch b, const AT* __restrict__ q, int ldq, const AT* __restrict__ cache,
                                                        const WT* __restrict__ sink, const AT* __restrict__ gate, int ldg,
                                                        int H, int G, int dim, int vdim, float scale, float qt_coef,
                                                        int qt_every, int window, float out_scale, OT* __restrict__ out, int ldo) {
  pdl_begin();
  extern __shared__ __align__(16) unsigned char hy_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* qs = reinterpret_cast<float*>(hy_smem) + warp * dim;
  const int unit = blockIdx.x * 4 + warp;
  if (unit >= b.T * H) return;
  const int t = unit / H, h = unit % H;
  const int e = b.tok_ent[t], pos = b.tok_pos[t];
  const int g = h / (H / G);
  const float temp = 1.0f + qt_coef * logf(floorf((float)(pos + 1) / (float)qt_every) + 1.0f);
  for (int d = lane; d < dim; d += 32) qs[d] = to_f(q[(size_t)t * ldq + h * dim + d]) * temp;
  __syncwarp();
  const int* pg = b.pages + (size_t)e * b.max_pages;
  float m = sink ? to_f(sink[h]) : -INFINITY, l = sink ? 1.0f : 0.0f;
  float acc[HY_ATT_MAXD];
#pragma unroll
  for (int i = 0; i < HY_ATT_MAXD; ++i) acc[i] = 0.0f;
  const int first = first_seen(pos, window);
  for (int j0 = first / 32 * 32; j0 <= pos; j0 += 32) {
    const int j = j0 + lane;
    const bool sees = j <= pos && j >= first;
    float s = -INFINITY;
    const AT* kr = nullptr;
    if (sees) {
      kr = cache + (((size_t)pg[j / b.page_size] * G + g) * b.page_size + j % b.page_size) * dim;
      float dot = 0.0f;
      for (int d = 0; d < dim; ++d) dot = fmaf(qs[d], to_f(kr[d]), dot);
      s = dot * scale;
    }
    const float mn = fmaxf(m, warp_max(s));
    const float corr = expf(m - mn);
    const float p = sees ? expf(s - mn) : 0.0f;
    l = l * corr + warp_sum(p);
    m = mn;
#pragma unroll
    for (int i = 0; i < HY_ATT_MAXD; ++i) acc[i] *= corr;
    const int cnt = min(32, pos + 1 - j0);
    for (int jj = max(first - j0, 0); jj < cnt; ++jj) {
      const float pj = __shfl_sync(0xffffffffu, p, jj);
      const int ja = j0 + jj;
      const AT* kj = cache + (((size_t)pg[ja / b.page_size] * G + g) * b.page_size + ja % b.page_size) * dim;
#pragma unroll
      for (int i = 0; i < HY_ATT_MAXD; ++i) {
        const int d = lane + 32 * i;
        if (d < vdim) acc[i] = fmaf(pj, to_f(kj[d]), acc[i]);
      }
    }
  }
  const float inv = 1.0f / l;
#pragma unroll
  for (int i = 0; i < HY_ATT_MAXD; ++i) {
    const int d = lane + 32 * i;
    if (d < vdim) {
      const float gt = gate ? sigmoid_f(to_f(gate[(size_t)t * ldg + h * vdim + d])) : 1.0f;
      out[(size_t)t * ldo + h * vdim + d] = from_f<OT>(acc[i] * inv * gt * out_scale);
    }
  }
}

// ---- decays exp(dt a) of two states at a time ---------------------------------------------------------------------------------------
// dt a log2(e) as a rounded product and its remainder: 2^(y + e) = 2^y + 2^y e ln 2 for the |e| <= 2^-24 |y| that is left; for two states the products
// run as pairs.  The error against 64 bits is 2.0e-7 at most and 6.5e-8 root mean square from |dt a| = 1 to 87, where expf of the rounded product
// comes to 3.9e-6 and 7.1e-7, and below one the same as expf's (1.9e-7 and 4.2e-8 against 1.6e-7 and 3.6e-8).
struct RatePair {
  float2 hi, neg, lo;                                          // a log2(e), its negative, what rounding took off it
  RatePair() = default;
  __device__ __forceinline__ RatePair(float a0, float a1) {
    const float l2 = 1.4426950408889634f, l2_rest = 1.9259629911266175e-8f, most = -1e18f;      // products with dt <= 1e18 stay finite
    a0 = a0 < most ? most : a0; a1 = a1 < most ? most : a1;
    hi = make_float2(a0 * l2, a1 * l2);
    neg = make_float2(-hi.x, -hi.y);
    lo = make_float2(fmaf(a0, l2_rest, fmaf(a0, l2, neg.x)), fmaf(a1, l2_rest, fmaf(a1, l2, neg.y)));
  }
};
__device__ __forceinline__ float ex2_f(float y) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y)); return r; }
__device__ __forceinline__ float2 exp_rates(float dt, const RatePair& a) {
  const float2 d = make_float2(dt, dt), y = mul2(d, a.hi);
  float2 e = fma2(d, a.hi, mul2(d, a.neg));
  e = mul2(fma2(d, a.lo, e), make_float2(0.6931471805599453f, 0.6931471805599453f));
  const float2 x = make_float2(ex2_f(y.x), ex2_f(y.y));
  return fma2(x, e, x);
}
__device__ __forceinline__ float finite_step(float dt) { return dt > 1e18f ? 1e18f : dt; }

// ---- selective scan -------------------------------------------------------------------------------------------------------------
// S[c, n] <- exp(dt_c A[c, n]) S[c, n] + dt_c x_c B_n ; y_c = sum_n S[c, n] C_n + D_c x_c ; out = y silu(z) out_scale.
// dt_raw is the step-size projection before bias and softplus.  low [T, ldl] holds [dt-rank part | B | C].
// state [slot][inner][nstate] fp32.
// L lanes share a channel, each holding NPER CONSECUTIVE states (NPER * L >= nstate; the staged B and C are zero beyond nstate).
// Inputs of TB tokens are copied asynchronously while the batch before them runs; the read-outs of eight tokens are reduced
// in one exchange in which every step halves the tokens a lane keeps, so eight tokens run without a shuffle between them.
// The arithmetic bounds it: half a dozen operations and one exponential per state and token (exp_rates), so the fewer lanes
// share a channel the less is spent on the exchange and on indices: four states per lane.
// 2048 tokens, 4096 channels of 16 states: one state per lane, a five-step exchange per token and loads waited for took 949 us
// (0.46 us per token), this form 369 us.
// That is a chain of tokens with less than a warp per scheduler, so long portions of few requests are cut into segments that run side by side: a first
// pass (SCAN_OWN) leaves each segment's own state (the first one's behind the request's, the others' from zero; in the last one's place
// the request's, which the second pass writes over) and the sum of its step sizes, of which exp(A sum) is the decay over the segment; the
// second (SCAN_READ) begins with what the segments before it add up to and makes the read-outs.  Most of the arithmetic is
// done twice, so with many requests, whose blocks fill the SMs, a scan stays whole (see scan_segments).  2048 tokens, 4096 channels of 16 states, us, whole -> segments: one
// request 371 -> 221 (195 with exp_rates), two 286 -> 250 (224); 288 tokens of one request 60 -> 49 (44), of two 49 -> 46 (43).
enum ScanPass : int { SCAN_WHOLE = 0, SCAN_OWN = 1, SCAN_READ = 2 };
// tokens per segment, segments per entry (grid y: entry by entry); own states [entry, segment][inner][nstate], sums of step sizes
// [entry, segment][inner]
struct ScanSegments { int tokens, count; float* own; float* dt; };
__host__ __device__ constexpr int scan_tb(int np) { return np <= 64 ? 32 : np <= 128 ? 16 : 8; }
__host__ __device__ constexpr size_t scan_smem(int np, int pb, size_t esz) {
  return 2 * (size_t)scan_tb(np) * (2 * (size_t)np * 4 + (size_t)pb * (4 + 2 * esz));
}
// vec: rows of B, C and dt (fp32) and of x, z may travel by 16-byte copies (bits 0 and 1; see launch_scan)
template <typename AT, typename WT, int NPER, int L, int PASS>
__global__ void __launch_bounds__(128) scan_kernel(Batch b, const AT* __restrict__ x, int ldx, const AT* __restrict__ z, int ldz,
                                                   const float* __restrict__ dt_raw, int lddt, const WT* __restrict__ dt_bias,
                                                   const float* __restrict__ low, int ldl, int col_b, int col_c,
                                                   const float* __restrict__ A, const WT* __restrict__ D, int inner, int nstate,
                                                   int vec, float out_scale, float* __restrict__ state, AT* __restrict__ out, int ldo, ScanSegments seg) {
  pdl_trigger();
  if (PASS != SCAN_WHOLE) pdl_wait();
  constexpr int NP = NPER * L, PB = 128 / L, TB = scan_tb(NP), TG = 8, CH = 16 / (int)sizeof(AT);
  extern __shared__ __align__(16) unsigned char hy_smem[];
  float* sB = reinterpret_cast<float*>(hy_smem);               // [2][TB][NP]
  float* sC = sB + 2 * TB * NP;                                // [2][TB][NP]
  float* sdt = sC + 2 * TB * NP;                               // [2][TB][PB], step sizes once their batch has landed
  AT* sx = reinterpret_cast<AT*>(sdt + 2 * TB * PB);           // [2][TB][PB]
  AT* sz = sx + 2 * TB * PB;                                   // [2][TB][PB]
  const int e = PASS == SCAN_WHOLE ? blockIdx.y : blockIdx.y / seg.count, tid = threadIdx.x, c0 = blockIdx.x * PB;
  const int cl = tid / L, sub = tid % L, n0 = sub * NPER, c = c0 + cl;
  const bool live = c < inner;
  const int cc = live ? c : inner - 1, npb = min(PB, inner - c0);
  const int at = PASS == SCAN_WHOLE ? 0 : (int)blockIdx.y % seg.count, all = b.ent_start[e + 1] - b.ent_start[e], pos0 = b.ent_pos0[e];
  const int start = b.ent_start[e] + (PASS == SCAN_WHOLE ? 0 : at * seg.tokens);
  const int cnt = PASS == SCAN_WHOLE ? all : min(seg.tokens, all - at * seg.tokens);
  const bool ends = PASS == SCAN_WHOLE || (at + 1) * seg.tokens >= all;          // the entry's last segment
  if (cnt <= 0) return;
  float* st = state + ((size_t)b.ent_slot[e] * inner + cc) * nstate;
  float2 S[NPER / 2];
  RatePair a[NPER / 2];
  auto from_rows = [&](const float* row, bool there) {         // this lane's states of a row of nstate
#pragma unroll
    for (int i = 0; i < NPER; i += 2)
      S[i / 2] = make_float2(there && n0 + i < nstate ? row[n0 + i] : 0.0f, there && n0 + i + 1 < nstate ? row[n0 + i + 1] : 0.0f);
  };
  auto to_rows = [&](float* row) {
#pragma unroll
    for (int i = 0; i < NPER; i += 2) {
      if (n0 + i < nstate) row[n0 + i] = S[i / 2].x;
      if (n0 + i + 1 < nstate) row[n0 + i + 1] = S[i / 2].y;
    }
  };
  from_rows(st, PASS != SCAN_READ && (at == 0 || ends) && pos0 > 0);
#pragma unroll
  for (int i = 0; i < NPER; i += 2) {
    const float* row = A + (size_t)cc * nstate;
    a[i / 2] = RatePair(n0 + i < nstate ? row[n0 + i] : 0.0f, n0 + i + 1 < nstate ? row[n0 + i + 1] : 0.0f);
  }
  if (PASS == SCAN_WHOLE) pdl_wait();
  if (PASS == SCAN_OWN && ends) {                              // what the request came with, for the first segment of the second pass
    if (live) to_rows(seg.own + ((size_t)blockIdx.y * inner + c) * nstate);
    return;
  }
  if constexpr (PASS == SCAN_READ) {
    if (at == 0) from_rows(seg.own + ((size_t)(e * seg.count + (all - 1) / seg.tokens) * inner + cc) * nstate, true);
    for (int k = 0; k < at; ++k) {
      const size_t row = (size_t)(e * seg.count + k) * inner + cc;
      const float dt = finite_step(seg.dt[row]);
      const float* own = seg.own + row * nstate;
#pragma unroll
      for (int i = 0; i < NPER; i += 2)
        S[i / 2] = fma2(exp_rates(dt, a[i / 2]), S[i / 2], make_float2(n0 + i < nstate ? own[n0 + i] : 0.0f, n0 + i + 1 < nstate ? own[n0 + i + 1] : 0.0f));
    }
  }
  float dt_sum = 0.0f;
  const float dd = to_f(D[cc]);
  if (nstate < NP)                                             // states beyond the last stay zero
    for (int i = tid; i < 2 * TB * NP; i += 128) if (i % NP >= nstate) { sB[i] = 0.0f; sC[i] = 0.0f; }
  auto fetch = [&](int j0, int buf) {
    const int nb = min(TB, cnt - j0);
    const size_t t0 = (size_t)(start + j0);
    float* db = sB + buf * TB * NP;
    float* dc = sC + buf * TB * NP;
    float* dt = sdt + buf * TB * PB;
    if (vec & 1) {
      const int nc = nstate / 4, nd = npb / 4;
      for (int i = tid; i < nb * nc; i += 128) {
        const int r = i / nc, k = i % nc * 4;
        const float* src = low + (t0 + r) * ldl + k;
        jf::cp_async_16(db + r * NP + k, src + col_b, 16u);
        if (PASS != SCAN_OWN) jf::cp_async_16(dc + r * NP + k, src + col_c, 16u);
      }
      for (int i = tid; i < nb * nd; i += 128) jf::cp_async_16(dt + i / nd * PB + i % nd * 4, dt_raw + (t0 + i / nd) * lddt + c0 + i % nd * 4, 16u);
    } else {
      for (int i = tid; i < nb * nstate; i += 128) {
        const int r = i / nstate, k = i % nstate;
        db[r * NP + k] = low[(t0 + r) * ldl + col_b + k];
        dc[r * NP + k] = low[(t0 + r) * ldl + col_c + k];
      }
      for (int i = tid; i < nb * npb; i += 128) dt[i / npb * PB + i % npb] = dt_raw[(t0 + i / npb) * lddt + c0 + i % npb];
    }
    AT* dx = sx + buf * TB * PB;
    AT* dz = sz + buf * TB * PB;
    if (vec & 2) {
      const int nx = npb / CH;
      for (int i = tid; i < nb * nx; i += 128) {
        const int r = i / nx, k = i % nx * CH;
        jf::cp_async_16(dx + r * PB + k, x + (t0 + r) * ldx + c0 + k, 16u);
        if (PASS != SCAN_OWN) jf::cp_async_16(dz + r * PB + k, z + (t0 + r) * ldz + c0 + k, 16u);
      }
    } else {
      for (int i = tid; i < nb * npb; i += 128) {
        dx[i / npb * PB + i % npb] = x[(t0 + i / npb) * ldx + c0 + i % npb];
        dz[i / npb * PB + i % npb] = z[(t0 + i / npb) * ldz + c0 + i % npb];
      }
    }
    jf::cp_async_commit();
  };
  fetch(0, 0);
  int buf = 0;
  for (int j0 = 0; j0 < cnt; j0 += TB, buf ^= 1) {
    const int nb = min(TB, cnt - j0);
    jf::cp_async_wait_all();
    __syncthreads();                                           // this batch has landed; the batch before it is finished
    if (j0 + TB < cnt) fetch(j0 + TB, buf ^ 1);
    float* bdt = sdt + buf * TB * PB;
    for (int i = tid; i < nb * PB; i += 128)
      if (i % PB < npb) bdt[i] = softplus_f(bdt[i] + to_f(dt_bias[c0 + i % PB]));
    __syncthreads();
    const float* rb = sB + buf * TB * NP + n0;
    const float* rc = sC + buf * TB * NP + n0;
    const int ck = min(cl, npb - 1);
    const AT* rx = sx + buf * TB * PB + ck;
    const AT* rz = sz + buf * TB * PB + ck;
    AT* po = out + (size_t)(start + j0) * ldo + cc;
    auto update = [&](int tt) {                                // one token; returns this lane's part of the read-out
      const float raw = bdt[tt * PB + ck], dx = raw * to_f(rx[tt * PB]), dt = finite_step(raw);
      if constexpr (PASS == SCAN_OWN) dt_sum += raw;
      float2 y = make_float2(0.0f, 0.0f);
#pragma unroll
      for (int i = 0; i < NPER; i += 4) {
        const float4 bb = *reinterpret_cast<const float4*>(rb + tt * NP + i);
        const float4 cv = *reinterpret_cast<const float4*>(rc + tt * NP + i);
        float2 &s0 = S[i / 2], &s1 = S[i / 2 + 1];
        s0 = fma2(exp_rates(dt, a[i / 2]), s0, mul2(make_float2(dx, dx), make_float2(bb.x, bb.y)));
        s1 = fma2(exp_rates(dt, a[i / 2 + 1]), s1, mul2(make_float2(dx, dx), make_float2(bb.z, bb.w)));
        y = fma2(s0, make_float2(cv.x, cv.y), y);
        y = fma2(s1, make_float2(cv.z, cv.w), y);
      }
      return y.x + y.y;
    };
    auto leave = [&](int tt, float y) {
      y = fmaf(dd, to_f(rx[tt * PB]), y);
      po[(size_t)tt * ldo] = from_f<AT>(y * silu_f(to_f(rz[tt * PB])) * out_scale);
    };
    int tt = 0;
    if constexpr (PASS == SCAN_OWN) {
#pragma unroll 4
      for (; tt < nb; ++tt) update(tt);
    } else {
      for (; tt + TG <= nb; tt += TG) {
        float p[TG];
#pragma unroll
        for (int u = 0; u < TG; ++u) p[u] = update(tt + u);
        int n = TG, base = 0;
#pragma unroll
        for (int s = L >> 1; s >= 1; s >>= 1) {
          const bool hi = (sub & s) != 0;
          if (n > 1) {
            n >>= 1;
#pragma unroll
            for (int u = 0; u < TG / 2; ++u) {
              if (u >= n) break;
              const float other = __shfl_xor_sync(0xffffffffu, hi ? p[u] : p[u + n], s);
              p[u] = (hi ? p[u + n] : p[u]) + other;
            }
            base += hi ? n : 0;
          } else {
            p[0] += __shfl_xor_sync(0xffffffffu, p[0], s);
          }
        }
        constexpr int LEFT = TG > L ? TG / L : 1, SAME = L > TG ? L / TG : 1;        // tokens per lane, lanes per token
        if (live && (sub & (SAME - 1)) == 0) {
#pragma unroll
          for (int u = 0; u < LEFT; ++u) leave(tt + base + u, p[u]);
        }
      }
      for (; tt < nb; ++tt) {
        float y = update(tt);
#pragma unroll
        for (int s = L >> 1; s >= 1; s >>= 1) y += __shfl_xor_sync(0xffffffffu, y, s);
        if (live && sub == 0) leave(tt, y);
      }
    }
  }
  if constexpr (PASS == SCAN_OWN) {
    if (!live) return;
    const size_t row = (size_t)blockIdx.y * inner + c;
    if (sub == 0) seg.dt[row] = dt_sum;
    to_rows(seg.own + row * nstate);
    return;
  }
  if (live && ends) to_rows(st);
}

// Segments of a scan: as many as give every SM SCAN_BLOCKS blocks, at least three (four with four requests and more) of at least SCAN_SEG_TOKENS tokens.
// 16 states, us, whole -> segments.  4096 channels: 288 tokens 45 -> 39, 512 78 -> 57, 1024 152 -> 106, 2048 298 -> 190; 2048 tokens of two requests 251 -> 218
// in three segments, of three 171 -> 180 in four (for which SCAN_BLOCKS has no room).  2048 channels: 288 tokens 45 -> 33, 512 77 -> 45, 2048 297 -> 103; of two
// requests 218 -> 119, of three 157 -> 105, of four 125 -> 136 in three segments and 104 in six, of eight 80 -> 114 in three.  Segments of no less than 192
// tokens: 288 tokens 45 (none), 512 78 (none).
constexpr int SCAN_BLOCKS = 6, SCAN_SEG_TOKENS = 96;
inline int scan_segment_rows(int blocks) { return 148 * SCAN_BLOCKS / (blocks < 1 ? 1 : blocks); }      // entries x segments at most
inline ScanSegments scan_segments(float* own, int blocks, int entries, int longest, int inner, int nstate) {
  const int fit = scan_segment_rows(blocks) / entries, n = fit < longest / SCAN_SEG_TOKENS ? fit : longest / SCAN_SEG_TOKENS;
  if (!own || n < (entries < 4 ? 3 : 4)) return ScanSegments{0, 1, nullptr, nullptr};
  const int tokens = ((longest + n - 1) / n + 31) / 32 * 32, count = (longest + tokens - 1) / tokens;
  return ScanSegments{tokens, count, own, own + (size_t)entries * count * inner * nstate};
}

// Sum of two values over the block in one pass (same order rules as block_sum).  red: >= 66 floats.
__device__ __forceinline__ float2 block_sum2(float a, float b, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  a = warp_sum(a); b = warp_sum(b);
  __syncthreads();
  if (lane == 0) { red[w] = a; red[33 + w] = b; }
  __syncthreads();
  if (w == 0) {
    float sa = lane < nw ? red[lane] : 0.0f, sb = lane < nw ? red[33 + lane] : 0.0f;
    sa = warp_sum(sa); sb = warp_sum(sb);
    if (lane == 0) { red[32] = sa; red[65] = sb; }
  }
  __syncthreads();
  return make_float2(red[32], red[65]);
}

// ---- sampling: argmax, or Gumbel-max at a temperature with a counter-based generator ---------------------------------------------
__device__ __forceinline__ uint32_t mix32(uint64_t key, uint32_t ctr) {
  uint64_t z = key + 0x9E3779B97F4A7C15ull * (uint64_t)(ctr + 1);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return (uint32_t)((z ^ (z >> 31)) >> 32);
}
// One block per row.  256 threads with one 4-byte load in flight each took 62 us for 32000 logits; 1024 threads with four
// independent loads 10 us.
__global__ void __launch_bounds__(1024) sample_kernel(const float* __restrict__ logits, int vocab, const float* __restrict__ temperature,
                                                      uint64_t seed, int* __restrict__ out) {
  pdl_begin();
  __shared__ float bv[32];
  __shared__ int bi[32];
  const int r = blockIdx.x;
  const float temp = temperature ? temperature[r] : 0.0f;
  const float* row = logits + (size_t)r * vocab;
  float best = -INFINITY;
  int besti = 0x7fffffff;
  for (int v0 = threadIdx.x; v0 < vocab; v0 += 4 * blockDim.x) {
    float x[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) x[k] = v0 + k * (int)blockDim.x < vocab ? row[v0 + k * blockDim.x] : 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int v = v0 + k * blockDim.x;
      if (v >= vocab) break;
      float s = x[k];
      if (temp > 0.0f) {
        const float uu = ((float)mix32(seed + (uint64_t)r * 0x100000001B3ull, (uint32_t)v) + 0.5f) * (1.0f / 4294967296.0f);
        s = s / temp - logf(-logf(uu));
      }
      if (s > best || (s == best && v < besti)) { best = s; besti = v; }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, besti, o);
    if (ov > best || (ov == best && oi < besti)) { best = ov; besti = oi; }
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) { bv[w] = best; bi[w] = besti; }
  __syncthreads();
  if (w == 0) {
    const int nw = blockDim.x >> 5;
    best = lane < nw ? bv[lane] : -INFINITY;
    besti = lane < nw ? bi[lane] : 0x7fffffff;
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, besti, o);
      if (ov > best || (ov == best && oi < besti)) { best = ov; besti = oi; }
    }
    if (lane == 0) out[r] = besti;
  }
}

}  // namespace hy
