// hy_few.cuh — bf16 products of up to eight rows (decode steps): C[t, n] = sum_k A[t, k] W[n, k], fp32 accumulation, dense and by expert
// (libjf_hybrid.so).
//
// What such a product takes is its weights' way through the chip once, so a warp takes 16 features and keeps eight 16-byte loads per lane in
// flight, two batches at a time; the first batch of its first tile travels while the kernel before this one ends (weights do not depend on
// it).  The products run as mma.m16n8k16 with the weights as the 16-row operand and the eight rows as the columns: tcgen05 would want the weights in
// shared memory, in tiles of 128 features, and has nothing to win at 8 columns.  Which k stands where inside a block of 32 is free as long as
// both operands agree, so a lane's 16 bytes of a weight row are its operands of two products as they come.
// Few features: ksplit warps share a tile and their sums are added in part order.
// Behind a small kernel, weights from HBM, us, a column per warp on the fp32 units (gemm_rows_kernel) -> this: eight rows, N 32000, K 1024 59.5 -> 15.9
// (one row 22.9 -> 15.3); N 10496, K 1024 23.1 -> 11.0 (10.1 -> 9.6); N 2112, K 2048 17.1 -> 7.3; N 1024, K 7168 41.4 -> 12.7; four rows of
// N 4096, K 2048 15.0 -> 8.7.  The floor of the first is 10.0; what is left is the start of two kernels, about 4 us.
#pragma once
#include "hy_kernels.cuh"

namespace hy {

constexpr int FEW_ROWS = 8, FEW_BATCH = 4;                     // rows of a product; blocks of 32 k per batch of loads

__device__ __forceinline__ uint4 few_load(const bf16* p, bool in) {
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  if (in) asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void few_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// elements from row to row of the staged rows: blocks of 32 k, and rows that eight lanes read at once start 64 bytes apart modulo 128
__host__ __device__ constexpr int few_stride(int K) { const int kp = (K + 31) / 32 * 32; return kp % 64 == 0 ? kp + 32 : kp; }
__host__ __device__ constexpr size_t few_smem(int K) { return (size_t)FEW_ROWS * few_stride(K) * 2; }

struct FewBatch { uint4 lo[FEW_BATCH], hi[FEW_BATCH]; };       // features g and g + 8 of a tile
// Blocks s .. of 32 k; row_lo, row_hi: this lane's weight rows at its first k (NULL: none).
__device__ __forceinline__ void few_fetch(FewBatch& w, const bf16* row_lo, const bf16* row_hi, int s, int end, int k0, int K) {
#pragma unroll
  for (int u = 0; u < FEW_BATCH; ++u) {
    const bool in = s + u < end && (s + u) * 32 + k0 < K;
    w.lo[u] = few_load(row_lo + (s + u) * 32, in && row_lo);
    w.hi[u] = few_load(row_hi + (s + u) * 32, in && row_hi);
  }
}
// The tensor cores cut what their sums lose off, so a sum that goes through all of k there is further from 64 bits than one of fp32
// additions (N 32000, K 1024: 3.8e-7 of its norm against 6.5e-8).  Here every product begins
// at zero and joins one of eight fp32 sums: 6.6e-8 to 6.9e-8 there, and within 6 % of the fp32 kernel's (mostly below) at thirteen other sizes.
struct FewSums {
  float c[2 * FEW_BATCH][4] = {};
  __device__ __forceinline__ float total(int i) const {
    return ((c[0][i] + c[1][i]) + (c[2][i] + c[3][i])) + ((c[4][i] + c[5][i]) + (c[6][i] + c[7][i]));
  }
};
__device__ __forceinline__ void few_products(FewSums& sums, const FewBatch& w, const bf16* x, int s, int end) {
#pragma unroll
  for (int u = 0; u < FEW_BATCH; ++u) {
    if (s + u >= end) break;
    const uint4 b = *reinterpret_cast<const uint4*>(x + (s + u) * 32);
    float c[4] = {}, d[4] = {};
    few_mma(c, w.lo[u].x, w.hi[u].x, w.lo[u].y, w.hi[u].y, b.x, b.y);
    few_mma(d, w.lo[u].z, w.hi[u].z, w.lo[u].w, w.hi[u].w, b.z, b.w);
#pragma unroll
    for (int i = 0; i < 4; ++i) { sums.c[2 * u][i] += c[i]; sums.c[2 * u + 1][i] += d[i]; }
  }
}
// Row r of the operand, at rows[r] (NULL: zeros), into shared memory; K is a multiple of 8.
template <typename Row>
__device__ __forceinline__ void few_stage(bf16* xs, int K, Row row) {
  const int stride = few_stride(K), nc = (K + 31) / 32 * 4;
  for (int i = threadIdx.x; i < FEW_ROWS * nc; i += blockDim.x) {
    const int r = i / nc, k = i % nc * 8;
    const bf16* src = row(r);
    *reinterpret_cast<uint4*>(xs + r * stride + k) = src && k < K ? *reinterpret_cast<const uint4*>(src + k) : make_uint4(0u, 0u, 0u, 0u);
  }
}
// Sums of a tile's ksplit warps, in the first of them.  parts [warps][4][32]; ends with a barrier.
__device__ __forceinline__ void few_add_parts(float (&c)[4], float* parts, int ksplit, int warp, int lane) {
#pragma unroll
  for (int i = 0; i < 4; ++i) parts[(warp * 4 + i) * 32 + lane] = c[i];
  for (int half = ksplit >> 1; half > 0; half >>= 1) {          // in halves: as few roundings on the way as there are doublings
    __syncthreads();
    const int at = warp % ksplit;
    if (at < half) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        c[i] += parts[((warp + half) * 4 + i) * 32 + lane];
        parts[(warp * 4 + i) * 32 + lane] = c[i];
      }
    }
  }
  __syncthreads();
}

// Rows of A and W begin on 16 bytes, K is a multiple of 8 (few_takes).  grid.x blocks of WARPS / ksplit tiles walk the features.
template <typename TO, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 16 / WARPS) gemm_few_kernel(const bf16* __restrict__ A, int lda, const bf16* __restrict__ W, int ldw, int T, int N, int K,
                                                          int ksplit, GemmOut o) {
  extern __shared__ __align__(16) unsigned char hy_smem[];
  __shared__ float parts[WARPS * 4 * 32];
  bf16* xs = reinterpret_cast<bf16*>(hy_smem);
  pdl_trigger();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, k0 = (lane & 3) * 8;
  const int per = WARPS / ksplit, steps = (K + 31) / 32, each = (steps + ksplit - 1) / ksplit;
  const int s0 = warp % ksplit * each, s1 = min(steps, s0 + each), tiles = (N + 15) / 16;
  auto fetch = [&](FewBatch& w, int tile, int s) {
    const int n = tile * 16 + g;
    few_fetch(w, n < N ? W + (size_t)n * ldw + k0 : nullptr, n + 8 < N ? W + (size_t)(n + 8) * ldw + k0 : nullptr, s, s1, k0, K);
  };
  FewBatch w;
  int tile = blockIdx.x * per + warp / ksplit;
  fetch(w, tile, s0);
  pdl_wait();
  few_stage(xs, K, [&](int r) { return r < T ? A + (size_t)r * lda : nullptr; });
  __syncthreads();
  const bf16* x = xs + g * few_stride(K) + k0;
  for (int base = blockIdx.x * per; base < tiles; base += gridDim.x * per) {
    FewSums sums;
    const int next = tile + gridDim.x * per;
    for (int s = s0; s < s1; s += FEW_BATCH) {
      FewBatch n;
      if (s + FEW_BATCH < s1) fetch(n, tile, s + FEW_BATCH);
      else fetch(n, next, s0);
      few_products(sums, w, x, s, s1);
      w = n;
    }
    float c[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] = sums.total(i);
    if (ksplit > 1) few_add_parts(c, parts, ksplit, warp, lane);
    if (warp % ksplit == 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int n = tile * 16 + g + (i >> 1) * 8, t = (lane & 3) * 2 + (i & 1);
        if (t < T && n < N) gemm_store<TO>(o, t, n, c[i]);
      }
    }
    tile = next;
  }
}

// The routed form: block row e takes the choices of expert e, found among the step's, A row = token (per_token) or pair, output row = pair, as
// expert_rows_kernel.  They are at most eight, because a step here has at most eight tokens and a token's choices are distinct, whatever its scores (see
// lowest_free); walking an expert's pairs eight at a time instead cost decode steps up to 1 %.  GLU: a tile is 8 gate rows and the 8 up rows N further on.
template <typename TO, bool GLU>
__global__ void __launch_bounds__(256, 2) expert_few_kernel(const bf16* __restrict__ A, int lda, const int* __restrict__ ids, int pairs, int top, int per_token,
                                                            const bf16* __restrict__ W, size_t w_stride, int N, int K, int ksplit, TO* __restrict__ out,
                                                            int ldo, int act, float limit) {
  extern __shared__ __align__(16) unsigned char hy_smem[];
  __shared__ float parts[8 * 4 * 32];
  __shared__ int mine[FEW_ROWS], count;
  bf16* xs = reinterpret_cast<bf16*>(hy_smem);
  pdl_begin();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, k0 = (lane & 3) * 8;
  if (warp == 0) {
    int n = 0;
    for (int i0 = 0; i0 < pairs; i0 += 32) {
      const bool hit = i0 + lane < pairs && ids[i0 + lane] == (int)blockIdx.y;
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      const int at = n + __popc(m & ((1u << lane) - 1));
      if (hit && at < FEW_ROWS) mine[at] = i0 + lane;
      n += __popc(m);
    }
    if (lane == 0) count = min(n, FEW_ROWS);
  }
  __syncthreads();
  const int rows = count;
  if (rows == 0) return;
  constexpr int TN = GLU ? 8 : 16;
  const int per = 8 / ksplit, steps = (K + 31) / 32, each = (steps + ksplit - 1) / ksplit;
  const int s0 = warp % ksplit * each, s1 = min(steps, s0 + each), tiles = (N + TN - 1) / TN;
  const bf16* We = W + (size_t)blockIdx.y * w_stride;
  auto fetch = [&](FewBatch& w, int tile, int s) {
    const int n = tile * TN + g;
    const bf16* lo = n < N ? We + (size_t)n * K + k0 : nullptr;
    const bf16* hi = GLU ? (lo ? lo + (size_t)N * K : nullptr) : n + 8 < N ? We + (size_t)(n + 8) * K + k0 : nullptr;
    few_fetch(w, lo, hi, s, s1, k0, K);
  };
  FewBatch w;
  int tile = blockIdx.x * per + warp / ksplit;
  fetch(w, tile, s0);
  few_stage(xs, K, [&](int r) { return r < rows ? A + (size_t)(per_token ? mine[r] / top : mine[r]) * lda : nullptr; });
  __syncthreads();
  const bf16* x = xs + g * few_stride(K) + k0;
  for (int base = blockIdx.x * per; base < tiles; base += gridDim.x * per) {
    FewSums sums;
    const int next = tile + gridDim.x * per;
    for (int s = s0; s < s1; s += FEW_BATCH) {
      FewBatch n;
      if (s + FEW_BATCH < s1) fetch(n, tile, s + FEW_BATCH);
      else fetch(n, next, s0);
      few_products(sums, w, x, s, s1);
      w = n;
    }
    float c[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] = sums.total(i);
    if (ksplit > 1) few_add_parts(c, parts, ksplit, warp, lane);
    if (warp % ksplit == 0) {
#pragma unroll
      for (int i = 0; i < (GLU ? 2 : 4); ++i) {
        const int n = tile * TN + g + (i >> 1) * 8, t = (lane & 3) * 2 + (i & 1);
        if (t >= rows || n >= N) continue;
        const float v = GLU ? gated_pair_f(act, c[i], c[i + 2], limit) : act >= 0 ? act_f(act, c[i]) : c[i];
        out[(size_t)mine[t] * ldo + n] = from_f<TO>(v);
      }
    }
    tile = next;
  }
}

// ---- host ----------------------------------------------------------------------------------------------------------------------------
// Whether a product of T rows may run here: rows of both operands on 16 bytes, operand rows that fit an SM.
inline bool few_takes(const void* A, int lda, const void* W, size_t ldw, int T, int K) {
  return T <= FEW_ROWS && K % 8 == 0 && lda % 8 == 0 && ldw % 8 == 0 && few_smem(K) <= 200 * 1024 &&
         ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) == 0;
}
// One or two rows over few weights stay with a column per warp (gemm_rows_kernel): a block starts sooner there.  Behind a small kernel, weights from HBM,
// us, that kernel and this one, at N x K:
//   one row     2048 x 2048 5.7 5.6   1024 x 4096 6.1 7.2   3072 x 2048 8.5 7.1   1024 x 7168 9.6 10.1   4096 x 2048 9.2 7.4   32000 x 256 12.2 5.8
//   two rows    256 x 4096 3.8 7.5    2048 x 1024 3.7 5.3   512 x 7168 6.7 10.4   1024 x 4096 7.4 7.6   2048 x 2048 7.3 6.1   1024 x 7168 12.2 10.7
//   four rows   512 x 512 3.4 4.5     1024 x 1024 5.2 5.4   256 x 4096 6.7 7.7    2048 x 1024 5.6 5.4   1024 x 2048 5.6 5.8   2048 x 2048 9.8 6.2
//   five rows   512 x 512 4.8 4.6     256 x 4096 10.1 7.9   2048 x 2048 15.4 6.4
// Two requests of 24 tokens, every product here -> by this rule: 9.07 -> 8.77 ms and, with experts, 10.63 -> 10.25.  With four, behind longer kernels than that
// small one, weights that travel ahead make up for the start: the other kernel below two million weights 9.64 ms, every product here 9.53 (11.57 and 11.47); with
// three 9.11 and 9.14 (11.38 and 11.32).
inline bool few_pays(int T, int N, int K) {
  const long long weights = (long long)N * K;
  return T == 1 ? N >= 2048 && weights >= 6000000 : T > 2 || (N >= 1024 && weights >= 4000000);
}
// Warps per tile: as many as bring the SMs a block and a half each, four blocks of 32 k at least for each.  Where a tile for every SM is too many already,
// blocks are 16 warps on one tile (eight rows, N 1024, K 4096: 11.6 -> 9.2 us; K 7168: 16.8 -> 12.7).
inline int few_ksplit(long long tiles, int K, int most = 8) {
  int s = K >= 512 ? 2 : 1;                                    // two: half the additions behind one another
  while (s < most && tiles * s < 148 * 12 && (K + 31) / 32 >= s * 2 * FEW_BATCH) s *= 2;
  return s;
}
inline bool few_wide(int tiles, int K) { return tiles <= 148 && few_ksplit(tiles, K, 16) == 16; }

}  // namespace hy
