// hy_gemm.cuh — the hybrid decoders' use of the product on pairs of SMs (jf_pair.cuh): what leaves with the accumulators, and the
// packing of weights into its tiles.
#pragma once
#include <vector>

#include "hy_kernels.cuh"
#include "jf_pair.cuh"

namespace hy {

// Epilogue of one warp: the accumulators at taddr (its 32 lanes, `cols` columns, a multiple of 32: two loads in flight) leave
// through GemmOut.  n: this lane's feature, t0: the token of the first column.
// GemmOut.act2 == 2 (gated pair): the weight rows alternate 16 gate features and the 16 up features that go with them, so
// lanes l and l + 16 of an epilogue warp hold one pair; act(gate) * up (act = GemmOut.act_kind) leaves through out1 at
// feature n / 2.  act2 == 5: the same for the columns of one range, see GemmOut.
// What a column does with its elements, and its parameters, are decided and read once per tile: gemm_store's chain of tests and loads
// per element took longer than the products of the next tile (N 20992, T 2048, K 2048 with the squared ReLU: 409 us against 118).
template <typename TO>
__device__ __forceinline__ void tc_store_columns(const GemmOut& o, uint32_t taddr, int n, int t0, int cols, int T, int N, int lane) {
  const bool pairs = o.act2 == 2 || (o.act2 == 5 && n - lane >= o.pair_lo && n - lane < o.pair_hi);
  const bool second = n >= o.split, wide = second ? (o.out2_f32 || sizeof(TO) == 4) : sizeof(TO) == 4, in = n < N;
  const float bias = o.bias && in ? o.bias[n] : 0.0f;
  // one pass over the columns with what to do with sixteen of them (rows: how many exist) given as a function
  auto each = [&](auto store16) { jf::tp_columns(taddr, t0, cols, T, store16); };
  if (pairs) {
    const int pf = (o.act2 == 5 ? (n - lane - o.pair_lo) >> 1 : (n - lane) >> 1) + (lane & 15);      // this lane's feature of a pair
    const int pn = o.act2 == 5 ? o.pair_n : o.split, pld = o.act2 == 5 ? o.ld_pair : o.ld1;
    TO* pout = (TO*)(o.act2 == 5 ? o.pair_out : o.out1) + pf;
    const bool low = lane < 16, live = pf < pn;
    auto go = [&](auto pair) {
      each([&](const uint32_t (&v)[16], int t, int rows) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          // lanes < 16 hold gates, the others ups: exchange so that a lane < 16 gets token j's pair and lane + 16 token j + 8's
          const float give = __uint_as_float(low ? v[j + 8] : v[j]);
          const float got = __shfl_xor_sync(0xffffffffu, give, 16);
          const float g = low ? __uint_as_float(v[j]) : got, up = low ? got : __uint_as_float(v[j + 8]);
          const int row = low ? j : j + 8;
          if (live && row < rows) pout[(size_t)(t + row) * pld] = from_f<TO>(pair(g, up));
        }
      });
    };
    if (o.act_kind == 0) go([](float g, float u) { return silu_f(g) * u; });
    else if (o.act_kind == 1) go([](float g, float u) { return gelu_tanh_f(g) * u; });
    else go([&](float g, float u) { return gated_pair_f(o.act_kind, g, u, o.act_limit); });
    return;
  }
  if (o.resid) {
    float* col = o.resid + n;
    const size_t ld = (size_t)o.ldr;
    const bool post = o.post_w != nullptr, next = o.next_w != nullptr;
    const float pw = post && in ? o.post_w[n] : 0.0f, pb = post && in ? o.post_b[n] : 0.0f, pl = post && in ? o.post_ls[n] : 0.0f;
    const float nw = next && in ? o.next_w[n] : 0.0f, nb = next && in ? o.next_b[n] : 0.0f;
    auto go = [&](auto sublayer, auto leave) {
      each([&](const uint32_t (&v)[16], int t, int rows) {
        if (!in) return;
        float* p = col + t * ld;
        float x[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) x[j] = j < rows ? p[j * ld] : 0.0f;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (j >= rows) continue;
          const float y = x[j] + sublayer(__uint_as_float(v[j]) * o.alpha + bias);
          p[j * ld] = y;
          leave((t + j) * ld + n, y);
        }
      });
    };
    auto plain = [](float c) { return c; };
    auto normed = [&](float c) { return pl * fmaf(tanhf(o.post_alpha * c), pw, pb); };
    auto nothing = [](size_t, float) {};
    auto half = [&](size_t at, float y) { ((bf16*)o.next_out)[at] = __float2bfloat16_rn(fmaf(tanhf(o.next_alpha * y), nw, nb)); };
    auto full = [&](size_t at, float y) { ((float*)o.next_out)[at] = fmaf(tanhf(o.next_alpha * y), nw, nb); };
    if (!post && !next) go(plain, nothing);
    else if (post && !next) go(normed, nothing);
    else if (post && !o.next_f32) go(normed, half);
    else if (post) go(normed, full);
    else if (!o.next_f32) go(plain, half);
    else go(plain, full);
    return;
  }
  const int pitch = second ? o.ld2 : o.ld1;
  char* dst = second ? (char*)o.out2 + (size_t)(n - o.split) * (wide ? 4 : 2) : (char*)o.out1 + (size_t)n * sizeof(TO);
  auto go = [&](auto value) {
    each([&](const uint32_t (&v)[16], int t, int rows) {
      if (!in) return;
      if (wide) {
        float* p = (float*)dst + (size_t)t * pitch;
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (j < rows) p[(size_t)j * pitch] = value(__uint_as_float(v[j]) * o.alpha + bias);
      } else {
        bf16* p = (bf16*)dst + (size_t)t * pitch;
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (j < rows) p[(size_t)j * pitch] = __float2bfloat16_rn(value(__uint_as_float(v[j]) * o.alpha + bias));
      }
    });
  };
  const bool square = o.act2 == 1 && second;
  if (o.act2 == 1) go([&](float c) { const float r = fmaxf(c, 0.0f); return square ? r * r : c; });
  else if (o.act2 == 3) go([&](float c) { return act_f(o.act_kind, c); });
  else if (o.act2 == 4) go([&](float c) { return expf(o.act_limit * log_sigmoid_f(c)); });
  else go([](float c) { return c; });
}

template <typename TO>
struct HyEpilogue {
  GemmOut o;
  __device__ __forceinline__ void operator()(uint32_t taddr, int n, int t0, int cols, int T, int N, int lane) const {
    tc_store_columns<TO>(o, taddr, n, t0, cols, T, N, lane);
  }
};

// ---- products of fp32 rows with bf16 weights (step sizes) ------------------------------------------------------------------------
// An fp32 number is the sum of three bf16 numbers, its upper, middle and lower eight bits, so the product of fp32 rows is one of bf16 rows
// [lower | middle | upper], three times as long, with the weights side by side three times: every product of two numbers is exact as it
// was, and the sums are the tensor cores' fp32 sums (the upper parts come last, so that what is cut off a sum is cut off few large ones).  Those lose
// more with every block of k than sums of fp32 additions do, so up to K 128 only.  Against 64 bits, of the result's norm, gemm_simt_kernel -> this:
// operands of both signs K 16 7.5e-8 -> 5.0e-8, K 64 1.4e-7 -> 7.7e-8, K 128 2.1e-7 -> 1.3e-7, K 256 2.8e-7 -> 2.3e-7, K 512 4.0e-7 -> 4.8e-7; of one
// sign, where the cut goes the same way every time, K 64 1.2e-7 -> 9.0e-8, K 128 1.7e-7 -> 1.8e-7, K 256 2.4e-7 -> 3.7e-7, K 512 3.3e-7 -> 8.7e-7.
// us, gemm_simt_kernel and both kernels here: N 4096, K 128, T 100 10.7 11.7, T 300 18.5 11.8, T 512 36.2 12.2, T 2048 88.3 18.4; N 2048, K 128, T 200 10.6
// 11.5, T 512 16.4 12.0; N 2048, K 64, T 200 6.4 10.3, T 300 10.5 10.5, T 512 11.8 10.6, T 2048 35.6 12.6.  From 512 rows on nothing is slower.  Not
// where every result goes through functions (decays, 2048 x 2048 and K 16: 36 us either way): that is what takes the time there.
constexpr int HY_SPLIT_ROWS = 512, HY_SPLIT_K = 128;
inline int split_cols(int K) { return (K + 63) / 64 * 64; }    // of each part
// a [T, lda] (K columns) -> o [T][3][KP], zeros beyond K.  What is no number, and infinities, stay whole in the upper part.
__global__ void __launch_bounds__(128) split_rows_kernel(const float* __restrict__ a, int lda, int T, int K, int KP, bf16* __restrict__ o) {
  pdl_begin();
  const int per = KP / 2;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < T * per; i += gridDim.x * blockDim.x) {
    const int t = i / per, k = i % per * 2;
    uint32_t part[3] = {};
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float x = k + j < K ? a[(size_t)t * lda + k + j] : 0.0f;
      const uint32_t u = __float_as_uint(x);
      const bool whole = (u & 0x7f800000u) == 0x7f800000u;
      const float hi = whole ? __bfloat162float(__float2bfloat16_rn(x)) : __uint_as_float(u & 0xffff0000u), r = whole ? 0.0f : x - hi;
      const float mid = __uint_as_float(__float_as_uint(r) & 0xffff0000u), lo = r - mid;
      part[0] |= (__float_as_uint(lo) >> 16) << (16 * j);      // lo has no more than eight bits left
      part[1] |= (__float_as_uint(mid) >> 16) << (16 * j);
      part[2] |= (__float_as_uint(hi) >> 16) << (16 * j);
    }
    uint32_t* row = reinterpret_cast<uint32_t*>(o + (size_t)t * 3 * KP + k);
    row[0] = part[0]; row[KP / 2] = part[1]; row[KP] = part[2];
  }
}

// Host-side packer: row-major [N, K] floats -> bf16 tiles [ceil(N/128)][ceil(K/64)] of 128 x 64 in the swizzled layout.
inline void pack_tiles(const float* w, int N, int K, std::vector<uint16_t>& out) {
  const int NT = (N + 127) / 128, KT = (K + 63) / 64;
  out.assign((size_t)NT * KT * 128 * 64, 0);
  for (int n = 0; n < N; ++n)
    for (int k = 0; k < K; ++k) {
      const size_t tile = (size_t)(n / 128) * KT + k / 64;
      const uint32_t off = jf::sw128_offset((uint32_t)(n % 128), (uint32_t)(k % 64));
      __nv_bfloat16 b = __float2bfloat16_rn(w[(size_t)n * K + k]);
      uint16_t bits;
      memcpy(&bits, &b, 2);
      out[tile * 8192 + off / 2] = bits;
    }
}

}  // namespace hy
