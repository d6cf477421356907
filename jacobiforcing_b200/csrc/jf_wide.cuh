// jf_wide.cuh — a planned forward of many rows (prompt chunks) as one kernel per stage instead of one persistent kernel.
//
// The persistent kernel is built around few rows: 128-feature tiles with all rows beside them, split-K partial sums in HBM, one
// pass over 64 keys per attention unit.  At 1000 rows of the 7B shape its products take in more activations than weights (gate/up
// 445 us a layer), and the stages between them move partial sums (rotary 90, attention 161 + merge 108, norms 153 + 166 us).
// Here the products run on pairs of SMs (jf_pair.cuh) with biases, residual sums and SwiGLU in their epilogues, and attention
// keeps its output in tensor memory (jf_flash.cuh).  Buffers, operand layouts and rounding points are the persistent kernel's: linear
// outputs, rotary products and sums, normalised values, SwiGLU operands, residual sums and attention weights are rounded to bf16
// where it rounds them, so both leave the same kind of keys and values behind.  A row's result depends neither on the rows beside it nor
// on where a prompt was cut into chunks: products add k in one order, and since all rows are committed, every key is read from its page, in
// tiles of 128 aligned to absolute positions.
#pragma once
#include <utility>
#include <vector>

#include "jf_flash.cuh"
#include "jf_types.h"

namespace jf {

constexpr int kWideRows = 256;

// ---- epilogues -----------------------------------------------------------------------------------------------------------------------
struct WideQkv {                                              // bf16(acc + bias), row-major
  __nv_bfloat16* out; int ld; const float* bias;
  __device__ __forceinline__ void operator()(uint32_t taddr, int n, int t0, int cols, int T, int N, int) const {
    const bool in = n < N;
    const float b = in ? bias[n] : 0.0f;
    tp_columns(taddr, t0, cols, T, [&](const uint32_t (&v)[16], int t, int rows) {
      if (!in) return;
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j < rows) out[(size_t)(t + j) * ld + n] = __float2bfloat16_rn(__uint_as_float(v[j]) + b);
    });
  }
};
struct WideResidual {                                         // hidden <- bf16(hidden + bf16(acc))
  __nv_bfloat16* hidden; int ld;
  __device__ __forceinline__ void operator()(uint32_t taddr, int n, int t0, int cols, int T, int N, int) const {
    tp_columns(taddr, t0, cols, T, [&](const uint32_t (&v)[16], int t, int rows) {
      if (n >= N) return;
      __nv_bfloat16* p = hidden + (size_t)t * ld + n;
      float x[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) x[j] = j < rows ? __bfloat162float(p[(size_t)j * ld]) : 0.0f;
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j < rows) p[(size_t)j * ld] = __float2bfloat16_rn(x[j] + bf16_round(__uint_as_float(v[j])));
    });
  }
};
// up <- bf16(g / (1 + exp(-g))) * up for bf16 values of N rows, with the quotients that IEEE division gives.  The fast division is within
// 2 ulp of it, so both round to the same bf16 unless its lower half lies within 4 of the middle between two; those, and divisors beyond its
// range, are divided behind all others: a division's rare path is a branch, and one behind every quotient leaves one row in flight
// (gate and up of the 7B shape at 128 rows, jf_step.cuh: 54.7 us, 45.6 so).
template <int N>
__device__ __forceinline__ void swiglu_rows(const float (&gate)[N], float (&up)[N]) {
  float q[N];
  uint32_t bad = 0u;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const float d = 1.f + __expf(-gate[j]);
    q[j] = __fdividef(gate[j], d);
    const uint32_t off = (__float_as_uint(q[j]) & 0xffffu) - 0x7ffcu;
    bad |= (off <= 8u || d > 1e36f) ? 1u << j : 0u;
  }
  if (bad) {
#pragma unroll
    for (int j = 0; j < N; ++j)
      if ((bad >> j) & 1u) q[j] = gate[j] / (1.f + __expf(-gate[j]));
  }
#pragma unroll
  for (int j = 0; j < N; ++j) up[j] *= bf16_round(q[j]);
}

struct WideSwiglu {                                           // silu(gate) * up into the next product's operand layout
  uint8_t* out; int rows_cap, inter;
  __device__ __forceinline__ void operator()(uint32_t taddr, int n, int t0, int cols, int T, int, int lane) const {
    const int f = ((n - lane) >> 1) + (lane & 15);             // lanes l and l + 16 hold the gate and the up value of feature f
    const bool low = lane < 16, in = f < inter;
    uint8_t* chunk = out + (size_t)(f >> 6) * rows_cap * 128;
    tp_columns(taddr, t0, cols, T, [&](const uint32_t (&v)[16], int t, int rows) {
      float g[8], u[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {                            // both halves of the warp work on 8 of the 16 tokens each
        const float give = __uint_as_float(low ? v[j + 8] : v[j]);
        const float got = __shfl_xor_sync(0xffffffffu, give, 16);
        g[j] = bf16_round(low ? __uint_as_float(v[j]) : got);
        u[j] = bf16_round(low ? got : __uint_as_float(v[j + 8]));
      }
      swiglu_rows(g, u);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int row = low ? j : j + 8;
        if (in && row < rows)
          *reinterpret_cast<__nv_bfloat16*>(chunk + sw128_offset((uint32_t)(t + row), (uint32_t)(f & 63))) = __float2bfloat16_rn(u[j]);
      }
    });
  }
};
struct WideLogits {
  float* out; size_t ld;
  __device__ __forceinline__ void operator()(uint32_t taddr, int n, int t0, int cols, int T, int N, int) const {
    tp_columns(taddr, t0, cols, T, [&](const uint32_t (&v)[16], int t, int rows) {
      if (n >= N) return;
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j < rows) out[(size_t)(t + j) * ld + n] = __uint_as_float(v[j]);
    });
  }
};

// ---- row kernels ---------------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void wide_unpack8(const uint4& u, float (&f)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) { f[2 * i] = __uint_as_float(w[i] << 16); f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
}
// RMS norm of a row into the operand layout; tok given: the row is the token's embedding and enters the stream here.  One block per
// row, 16 bytes per thread and pass.
constexpr int WIDE_NORM_THREADS = 256, WIDE_NORM_VECS = 4;      // rows of up to 256 * 4 * 8 = 8192 channels
__global__ void __launch_bounds__(WIDE_NORM_THREADS) wide_norm_kernel(const int* __restrict__ tok, const __nv_bfloat16* __restrict__ embed, int vocab,
                                                                      __nv_bfloat16* __restrict__ hidden, const __nv_bfloat16* __restrict__ w, int h,
                                                                      float eps, uint8_t* __restrict__ xn, int rows_cap) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[WIDE_NORM_THREADS / 32];
  const int t = blockIdx.x, nvec = h >> 3;
  uint4* row = reinterpret_cast<uint4*>(hidden + (size_t)t * h);
  const uint4* src = row;
  if (tok) { const int id = min(max(tok[t], 0), vocab - 1); src = reinterpret_cast<const uint4*>(embed + (size_t)id * h); }
  float x[WIDE_NORM_VECS][8], ss = 0.0f;
#pragma unroll
  for (int i = 0; i < WIDE_NORM_VECS; ++i) {
    const int v = threadIdx.x + i * WIDE_NORM_THREADS;
    if (v >= nvec) continue;
    const uint4 raw = src[v];
    if (tok) row[v] = raw;
    wide_unpack8(raw, x[i]);
#pragma unroll
    for (int k = 0; k < 8; ++k) ss = fmaf(x[i][k], x[i][k], ss);
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  ss = 0.0f;
#pragma unroll
  for (int i = 0; i < WIDE_NORM_THREADS / 32; ++i) ss += red[i];
  const float rstd = 1.0f / sqrtf(ss / (float)h + eps);
#pragma unroll
  for (int i = 0; i < WIDE_NORM_VECS; ++i) {
    const int v = threadIdx.x + i * WIDE_NORM_THREADS;
    if (v >= nvec) continue;
    float g[8];
    wide_unpack8(reinterpret_cast<const uint4*>(w)[v], g);
    uint32_t o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) o[k] = pack_bf16x2(g[2 * k] * bf16_round(x[i][2 * k] * rstd), g[2 * k + 1] * bf16_round(x[i][2 * k + 1] * rstd));
    *reinterpret_cast<uint4*>(xn + ((size_t)(v >> 3) * rows_cap + t) * 128 + (((v & 7) ^ (t & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// Rotary positions: queries to qbuf, keys and values to the in-flight rows and to their pages.  qkv [T][(n_q + 2 n_kv) d] with biases added.
// One block per row.
__global__ void __launch_bounds__(256) wide_rope_kernel(const __nv_bfloat16* __restrict__ qkv, ModelDims md, const int* __restrict__ row_pos,
                                                        const int* __restrict__ row_group, const Group* __restrict__ groups,
                                                        const int* __restrict__ tables, int max_pages, const __nv_bfloat16* __restrict__ cosb,
                                                        const __nv_bfloat16* __restrict__ sinb, __nv_bfloat16* __restrict__ qbuf, __nv_bfloat16* __restrict__ k,
                                                        __nv_bfloat16* __restrict__ v, __nv_bfloat16* __restrict__ k_pages, __nv_bfloat16* __restrict__ v_pages) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x, d = md.d, half = d >> 1, at = row_pos[t], pos = min(max(at, 0), md.max_pos - 1);
  const int page = tables[(size_t)groups[row_group[t]].seq * max_pages + at / kPage];
  const __nv_bfloat16* row = qkv + (size_t)t * md.qkv_dim;
  const int pairs = half >> 1, turned = md.n_q + md.n_kv;       // two neighbouring pairs per thread: 4-byte accesses
  for (int i = threadIdx.x; i < (turned + md.n_kv) * pairs; i += blockDim.x) {
    const int slot = i / pairs, e = i % pairs * 2;
    const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(row + slot * d + e), hi = *reinterpret_cast<const __nv_bfloat162*>(row + slot * d + half + e);
    float l0 = __low2float(lo), l1 = __high2float(lo), h0 = __low2float(hi), h1 = __high2float(hi);
    if (slot < turned) {
      const __nv_bfloat162 c = *reinterpret_cast<const __nv_bfloat162*>(cosb + (size_t)pos * half + e), s = *reinterpret_cast<const __nv_bfloat162*>(sinb + (size_t)pos * half + e);
      const float c0 = __low2float(c), c1 = __high2float(c), s0 = __low2float(s), s1 = __high2float(s);
      const float a0 = bf16_round(bf16_round(l0 * c0) - bf16_round(h0 * s0)), b0 = bf16_round(bf16_round(h0 * c0) + bf16_round(l0 * s0));
      const float a1 = bf16_round(bf16_round(l1 * c1) - bf16_round(h1 * s1)), b1 = bf16_round(bf16_round(h1 * c1) + bf16_round(l1 * s1));
      l0 = a0; h0 = b0; l1 = a1; h1 = b1;
    }
    const uint32_t a = pack_bf16x2(l0, l1), b = pack_bf16x2(h0, h1);
    auto put = [&](__nv_bfloat16* dst) {
      *reinterpret_cast<uint32_t*>(dst + e) = a;
      *reinterpret_cast<uint32_t*>(dst + half + e) = b;
    };
    if (slot < md.n_q) { put(qbuf + (size_t)t * md.q_dim + slot * d); continue; }
    const int kvh = slot < turned ? slot - md.n_q : slot - turned;
    put((slot < turned ? k : v) + ((size_t)t * md.n_kv + kvh) * d);
    put((slot < turned ? k_pages : v_pages) + (((size_t)page * md.n_kv + kvh) * kPage + at % kPage) * d);
  }
}

// First largest bf16-rounded logit of a row.  One block per row.
__global__ void __launch_bounds__(1024) wide_argmax_kernel(const float* __restrict__ logits, int vocab, int* __restrict__ greedy) {
  pdl_trigger();
  pdl_wait();
  __shared__ unsigned long long best[32];
  const float* row = logits + (size_t)blockIdx.x * vocab;
  unsigned long long b = 0ull;
  for (int v0 = threadIdx.x; v0 < vocab; v0 += 4096) {
    float x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = v0 + i * 1024 < vocab ? row[v0 + i * 1024] : 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (v0 + i * 1024 >= vocab) break;
      uint32_t u = __float_as_uint(bf16_round(x[i]));
      u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
      const unsigned long long key = ((unsigned long long)u << 32) | (0xFFFFFFFFu - (uint32_t)(v0 + i * 1024));
      b = key > b ? key : b;
    }
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) { const unsigned long long o = __shfl_xor_sync(0xffffffffu, b, s); b = o > b ? o : b; }
  if ((threadIdx.x & 31) == 0) best[threadIdx.x >> 5] = b;
  __syncthreads();
  if (threadIdx.x < 32) {
    b = best[threadIdx.x];
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) { const unsigned long long o = __shfl_xor_sync(0xffffffffu, b, s); b = o > b ? o : b; }
    if (threadIdx.x == 0) greedy[blockIdx.x] = (int)(0xFFFFFFFFu - (uint32_t)(b & 0xFFFFFFFFull));
  }
}

// ---- host ----------------------------------------------------------------------------------------------------------------------------
// Ends of a forward's stages on the device, for a stage profile: an event behind each (jf_profile_enable).
struct StageClock {
  std::vector<cudaEvent_t> events;                              // the first: the forward's start
  std::vector<int> ids;
  void mark(cudaStream_t s, int id) {
    cudaEvent_t e;
    if (cudaEventCreate(&e) != cudaSuccess) return;
    events.push_back(e); ids.push_back(id);
    cudaEventRecord(e, s);
  }
  ~StageClock() { for (cudaEvent_t e : events) cudaEventDestroy(e); }
};

// The launches of a forward: behind the first that fails nothing else is launched (a stage over what another one did not make would
// leave keys and values of stale rows in the pages).
struct WideStream {
  cudaStream_t s;
  int launches = 0;
  const char* failed = nullptr;                                 // what failed first
  StageClock* clock = nullptr;                                  // of a profiled forward
  void mark(int id) { if (clock && !failed) clock->mark(s, id); }
  template <typename... P, typename... A>
  void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, A&&... args) {
    if (failed) return;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid; c.blockDim = block; c.dynamicSmemBytes = smem; c.stream = s; c.attrs = &at; c.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);
    if (e == cudaSuccess) ++launches;
    else failed = cudaGetErrorString(e);
  }
};

// Opts the kernels in to their shared memory on the current device, for heads of d.  Once per engine, like the persistent kernel: the limit belongs to
// a device, and a process may hold engines on several.
inline cudaError_t wide_opt_in(int d) {
  auto opt = [](auto kernel, size_t bytes) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); };
  cudaError_t e = opt(pair_kernel<WideQkv, 256>, tp_smem_bytes(256));
  if (e == cudaSuccess) e = opt(pair_kernel<WideResidual, 256>, tp_smem_bytes(256));
  if (e == cudaSuccess) e = opt(pair_kernel<WideSwiglu, 256>, tp_smem_bytes(256));
  if (e == cudaSuccess) e = opt(pair_kernel<WideLogits, 256>, tp_smem_bytes(256));
  if (e == cudaSuccess) e = d == 64 ? opt(flash_kernel<64, 64, false>, fl_smem_bytes(64, 64)) : opt(flash_kernel<128, 128, false>, fl_smem_bytes(128, 128));
  return e;
}

// C[t, n] over packed activations [K / 64][rows_cap][64] (T rows from x_row0 on) and packed weight tiles; up_tiles > 0: a gate and an up
// matrix of that many 128-row tiles, N = 2 * features.  Tiles of 256 rows and whole ranges of k whatever T is: a row's sums are added
// in the same order in every forward.
template <class Epi>
inline void wide_product(WideStream& w, const void* X, int rows_cap, int x_row0, const void* W, int up_tiles, int T, int N, int K, const Epi& epi, int* err) {
  if (w.failed) return;
  const int KT = (K + 63) / 64, nt = (N + 127) / 128;
  CUtensorMap xm, wm;
  if (!tp_map(&xm, X, (uint64_t)KT * rows_cap, 64, 64, 128, false) ||
      !(up_tiles ? tp_map_pairs(&wm, W, up_tiles, KT) : tp_map(&wm, W, (uint64_t)nt * KT * 128, 64, 64, 128, false))) {
    w.failed = "a tensor map of a product could not be made";
    return;
  }
  const int tiles = (N + 255) / 256 * ((T + 255) / 256), grid = 2 * std::min(tiles, TP_CLUSTERS);
  w.launch(pair_kernel<Epi, 256>, grid, TP_THREADS, tp_smem_bytes(256), xm, wm, T, N, K, epi, err, TpGroup{}, PairLayout{rows_cap, x_row0, up_tiles > 0},
           PairSplit{1, nullptr, nullptr});
}

template <int D>
inline void wide_attention(WideStream& w, const DevCtx& c, int layer, const FlashUnit* units, int n_units, int* err) {
  if (w.failed) return;
  const ModelDims& md = c.md;
  CUtensorMap paged[2];
  for (int kv = 0; kv < 2; ++kv) {
    if (!tp_map(&paged[kv], c.kv_cache + kv_cache_offset(md, c.num_pages, layer, kv, 0, 0, 0), (uint64_t)c.num_pages * md.n_kv * kPage, D, D, FL_KEYS, true)) {
      w.failed = "a tensor map of the attention could not be made";
      return;
    }
  }
  const FlashArgs a{units, c.qbuf, (size_t)md.q_dim, D, c.block_tables, md.n_kv, rsqrtf((float)D), 0, nullptr, nullptr, 0, c.xa, 0, c.xrows_cap, err};
  w.launch(flash_kernel<D, D, false>, n_units, FL_THREADS, fl_smem_bytes(D, D), paged[0], paged[1], a);
}

// Row units of a forward: 128 (head, token) pairs of one key head of one group each, most key tiles first.
inline std::vector<FlashUnit> wide_units(const ModelDims& md, const std::vector<Group>& groups, int max_pages) {
  std::vector<FlashUnit> u;
  for (const Group& g : groups)
    for (int kvh = 0; kvh < md.n_kv; ++kvh)
      for (int p = 0; p < md.n_rep * g.len; p += 128)
        u.push_back(FlashUnit{g.row0, g.len, p, md.n_rep * g.len, kvh * md.n_rep, kvh, g.ctx, 0, g.seq * max_pages});
  auto last = [](const FlashUnit& x) {
    const int a = x.pair0 % x.len, b = a + std::min(128, x.pairs - x.pair0) - 1;
    return x.pos0 + std::min(b, x.len - 1);
  };
  std::stable_sort(u.begin(), u.end(), [&](const FlashUnit& x, const FlashUnit& y) { return last(x) > last(y); });
  return u;
}

// The whole forward on w's stream; the plan's arrays (tokens, positions, groups, tables) are on the device already.  Without rows that anybody
// asks for (no logits, no hidden rows: the chunks of a prompt ahead of its end) the last layer ends with its keys and values.
inline void wide_forward(WideStream& w, const DevCtx& c, int T, const FlashUnit* units, int n_units, int lm_row0, int lm_rows, bool want_hidden, int* err) {
  const ModelDims& md = c.md;
  __nv_bfloat16* qkv = reinterpret_cast<__nv_bfloat16*>(c.part);       // the split-K partial sums' buffer: T_cap rows of qkv_dim floats and more
  uint8_t* xn = reinterpret_cast<uint8_t*>(c.xn);
  const int nt_i = (md.inter + 127) >> 7;
  auto norm = [&](bool first, const __nv_bfloat16* weight) {
    w.launch(wide_norm_kernel, T, WIDE_NORM_THREADS, 0, first ? c.tok : nullptr, c.embed, md.vocab_embed, c.hidden, weight, md.h, md.eps, xn, c.xrows_cap);
  };
  norm(true, c.layer[0].ln1);
  for (int l = 0; l < md.layers && !w.failed; ++l) {
    const LayerW& L = c.layer[l];
    wide_product(w, c.xn, c.xrows_cap, 0, L.wqkv, 0, T, md.qkv_dim, md.h, WideQkv{qkv, md.qkv_dim, L.bqkv}, err);
    w.launch(wide_rope_kernel, T, 256, 0, qkv, md, c.row_pos, c.row_group, c.groups, c.block_tables, c.max_pages_per_seq, c.rope_cos, c.rope_sin, c.qbuf,
             c.kv_scratch + kv_scratch_offset(md, c.T_cap, l, 0, 0, 0), c.kv_scratch + kv_scratch_offset(md, c.T_cap, l, 1, 0, 0),
             c.kv_cache + kv_cache_offset(md, c.num_pages, l, 0, 0, 0, 0), c.kv_cache + kv_cache_offset(md, c.num_pages, l, 1, 0, 0, 0));
    if (l + 1 == md.layers && lm_rows == 0 && !want_hidden) return;
    if (md.d == 64) wide_attention<64>(w, c, l, units, n_units, err);
    else wide_attention<128>(w, c, l, units, n_units, err);
    wide_product(w, c.xa, c.xrows_cap, 0, L.wo, 0, T, md.h, md.q_dim, WideResidual{c.hidden, md.h}, err);
    norm(false, L.ln2);
    wide_product(w, c.xn, c.xrows_cap, 0, L.wgu, nt_i, T, 2 * md.inter, md.h, WideSwiglu{reinterpret_cast<uint8_t*>(c.xact), c.xrows_cap, md.inter}, err);
    wide_product(w, c.xact, c.xrows_cap, 0, L.wd, 0, T, md.h, md.inter, WideResidual{c.hidden, md.h}, err);
    norm(false, l + 1 < md.layers ? c.layer[l + 1].ln1 : c.final_norm);
  }
  if (lm_rows > 0) {
    wide_product(w, c.xn, c.xrows_cap, lm_row0, c.lm_head, 0, lm_rows, md.vocab, md.h, WideLogits{c.logits, (size_t)md.vocab}, err);
    w.launch(wide_argmax_kernel, lm_rows, 1024, 0, c.logits, md.vocab, c.greedy + lm_row0);
  }
}

}  // namespace jf
