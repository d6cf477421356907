// jf_step.cuh — a forward over in-flight rows as one kernel per stage: the persistent kernel's arithmetic, bit for bit, on launches that
// fill the SMs.
//
// The persistent kernel has four worker warps per SM for everything that is no product, because its roles share one block's
// registers.  At 230 rows of the 7B shape that is what a forward waits for (us a layer, of 270: SwiGLU epilogue 24, output and down
// epilogues 16, reduce + norm tails 42, attention 40, merge of its chunks 21, rotary stage 21).  Here every stage has the blocks that its
// rows need, launches overlap (pdl_trigger), and a product's weight tiles travel while the stage before it still runs.  A layer at 32 / 72 / 128 / 230
// rows of one sequence so: 100 / 107 / 121 / 146 us (72 of them the weights' at HBM's rate).
//
// Same sums in the same order: k-splits and their order, 64-key chunks of the attention and their merge, the row statistic by tiles
// of 128 columns, every rounding to bf16.  A forward so leaves the same bits whichever of the two runs it, and the choice between
// them (step_pays) is free.
#pragma once
#include "jf_kernel.cuh"
#include "jf_wide.cuh"

namespace jf {

// ---- products ------------------------------------------------------------------------------------------------------------------------
// Weight tiles of 128 features are the A operand, all rows (up to 256) the B operand, as in jf_gemm.cuh: D^T [128 features x rows] in
// tensor memory.  Bound by the weights' stream from HBM; beyond about 128 rows also by what a block takes in of the activations (its whole
// range of k) and by the epilogue behind a block's only tile.  Warp 0 brings weights and has the first stages under way before the
// kernel before this one ends, warp 2 the activations, warp 1 issues the products, groups of four warps store.
// us, back to back, at 16 / 128 / 230 rows: N 3584, K 18944 23.5 / 25.7 / 30.2 (136 MB);  gate and up of N 18944, K 3584
// 43.8 / 45.6 / 51 (272 MB).  Pairs of SMs that share the activations (cta_group::2) gave the same sums and were no faster at any row
// count (gate and up at 230 rows 61.5 against 58.5 before the epilogue was mended): what an SM takes in is not the bound.
enum StepEpilogue : int { STEP_PARTIAL = 0, STEP_SWIGLU = 1, STEP_SWIGLU_TAGGED = 2, STEP_HEAD = 3 };
constexpr int STEP_MAX_STAGES = 8, STEP_MAX_GROUPS = 4, STEP_WARP0 = 3, STEP_MAX_THREADS = 32 * (STEP_WARP0 + 4 * STEP_MAX_GROUPS);

struct StepGemm {
  const __nv_bfloat16 *W, *X;
  void* out;                       // PARTIAL: float [row][split][N]; SWIGLU: the next product's operand; SWIGLU_TAGGED: u64; HEAD: fp32 logits or null
  unsigned long long* keys;        // HEAD: argmax keys of the rows
  int n_tiles, k_chunks, splits, M, N, x_row0, xrows_cap;
  int row_stride, split_stride, out_rows_cap;
  unsigned int tag;
  int m_tiles, mt_rows;            // tiles of rows (at most 256 each, multiples of 16)
  int cols, bufs;                  // tensor memory columns of one accumulator, accumulators in turn
  int stages, slot, xslot, ks;     // ring: bytes of a stage and of one chunk's activations in it, chunks of k per stage
  int groups;                      // epilogue groups of four warps
  // what L2 is asked for behind the last weights: bytes of every tile of a later product's weights
  const __nv_bfloat16* ahead; int ahead_tiles; size_t ahead_stride; uint32_t ahead_bytes;
};

struct StepSmem {
  uint64_t full[STEP_MAX_STAGES], empty[STEP_MAX_STAGES], acc_full[2], acc_empty[2];
  uint32_t tmem_base, failed;
};

__device__ __forceinline__ bool step_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool step_wait(uint32_t bar, uint32_t parity, StepSmem* sm, int* err) {
  if (step_try(bar, parity)) return true;
  for (uint32_t i = 0; i < TC_SPIN_LIMIT; ++i) {
    if (*reinterpret_cast<volatile uint32_t*>(&sm->failed)) return false;
    if (step_try(bar, parity)) return true;
  }
  sm->failed = 1;
  atomicExch(err, 1);
  return false;
}
// plain bytes to an address of the shared window
__device__ __forceinline__ void step_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void step_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void step_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar, uint64_t policy) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar), "l"(policy) : "memory");
}

// The largest of 32 lanes for each of 16 rows in 16 exchanges instead of 80: at every step a lane hands over the rows that its partner
// keeps.  Lane l ends with row step_row(l).
__device__ __forceinline__ int step_row(int lane) { return ((lane >> 4) & 1) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1); }
__device__ __forceinline__ unsigned long long step_max16(unsigned long long (&k)[16], int lane) {
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const int half = 8 >> s, o = 16 >> s;
    const bool high = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i >= half) break;
      const unsigned long long keep = high ? k[i + half] : k[i], give = high ? k[i] : k[i + half];
      const unsigned long long got = __shfl_xor_sync(0xffffffffu, give, o);
      k[i] = got > keep ? got : keep;
    }
  }
  const unsigned long long got = __shfl_xor_sync(0xffffffffu, k[0], 1);
  return got > k[0] ? got : k[0];
}

template <int EPI>
__global__ void __launch_bounds__(STEP_MAX_THREADS, 1) step_gemm_kernel(const __grid_constant__ StepGemm g, int* err) {
  extern __shared__ __align__(16) unsigned char step_smem[];
  constexpr bool DUAL = EPI == STEP_SWIGLU || EPI == STEP_SWIGLU_TAGGED;
  constexpr int PARTS = DUAL ? 2 : 1;                         // weight tiles per chunk of k
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(step_smem) + 1023) & ~(uintptr_t)1023);
  StepSmem* sm = reinterpret_cast<StepSmem*>(base + (size_t)g.stages * g.slot);
  unsigned long long* best = reinterpret_cast<unsigned long long*>(sm + 1);                 // HEAD: [4 quarters][256 rows]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int items = g.n_tiles * g.splits * g.m_tiles;
  const uint32_t tm_cols = (uint32_t)(g.cols * PARTS * g.bufs);
  const uint32_t ring = smem_u32(base), ring_end = ring + g.stages * g.slot, full = smem_u32(sm->full), empty = smem_u32(sm->empty);
  const int ks = DUAL ? 1 : g.ks;                             // chunks of k per stage
  auto rows_of = [&](int mt) { return min(g.mt_rows, g.M - mt * g.mt_rows); };
  auto place = [&](int item, int& n_tile, int& split, int& mt, int& k0, int& k1) {
    mt = item % g.m_tiles;
    const int u = item / g.m_tiles;
    n_tile = u / g.splits; split = u - n_tile * g.splits;
    k0 = split_k0(split, g.splits, g.k_chunks); k1 = split_k1(split, g.splits, g.k_chunks);
  };
  if (threadIdx.x == 0) {
    for (int i = 0; i < g.stages; ++i) { mbar_init(&sm->full[i], 2); mbar_init(&sm->empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&sm->acc_full[i], 1); mbar_init(&sm->acc_empty[i], g.groups * 4); }
    sm->failed = 0;
    fence_mbar_init();
  }
  // What a stage costs the threads that fill it and the one that issues its products has to stay below what its bytes cost HBM (two
  // weight tiles pass an SM in 700 ns): running addresses instead of divisions, two tiles to a stage and one barrier for both operands.
  // N 3584, K 18944, 16 rows, back to back: 34.5 us with one thread, one tile to a stage and divisions; 26.2 with running
  // addresses; 23.5 so.
  const uint64_t policy = l2_policy_evict_first();            // weights are read once a forward
  const size_t up = (size_t)g.n_tiles * g.k_chunks * (kTileN * kTileK);
  auto load_w = [&](uint32_t dst, const __nv_bfloat16* w, int chunks, uint32_t bar) {
    step_expect(bar, (uint32_t)(chunks * PARTS) * kWTileBytes);
    step_bulk(dst, w, (uint32_t)chunks * kWTileBytes, bar, policy);
    if (DUAL) step_bulk(dst + kWTileBytes, w + up, kWTileBytes, bar, policy);
  };
  int ahead = 0;                                              // stages of the first item whose weights are under way
  if (threadIdx.x == 0) {
    int n_tile, split, mt, k0, k1;
    place(blockIdx.x, n_tile, split, mt, k0, k1);
    const __nv_bfloat16* w = g.W + ((size_t)n_tile * g.k_chunks + k0) * (kTileN * kTileK);
    for (int k = k0; k < k1 && ahead < g.stages; k += ks, ++ahead)
      load_w(ring + ahead * g.slot, w + (size_t)(k - k0) * (kTileN * kTileK), min(ks, k1 - k), full + ahead * 8);
  }
  if (warp == 1) tmem_alloc(&sm->tmem_base, tm_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_trigger();                                             // this block owns its columns (see pdl_trigger)
  if (warp != 0) pdl_wait();
  if (warp == 0) {
    if (lane == 0) {                                          // weights: nothing that a kernel before this one writes
      uint32_t dst = ring, bar = 0, parity = 1u;
      bool ok = true;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        int n_tile, split, mt, k0, k1;
        place(item, n_tile, split, mt, k0, k1);
        const __nv_bfloat16* w = g.W + ((size_t)n_tile * g.k_chunks + k0) * (kTileN * kTileK);
        for (int k = k0; k < k1; k += ks) {
          if (ahead > 0) --ahead;
          else {
            ok = step_wait(empty + bar, parity, sm, err);
            if (!ok) break;
            load_w(dst, w, min(ks, k1 - k), full + bar);
          }
          w += ks * (kTileN * kTileK);
          dst += g.slot; bar += 8;
          if (dst == ring_end) { dst = ring; bar = 0; parity ^= 1u; }
        }
      }
      for (int i = blockIdx.x; i < g.ahead_tiles && ok; i += gridDim.x) bulk_prefetch_l2(g.ahead + (size_t)i * g.ahead_stride, g.ahead_bytes);
      if (!ok) for (int i = 0; i < 1000; ++i) __nanosleep(1000);      // copies in flight land before the block leaves
    }
    __syncwarp();
  } else if (warp == 2) {
    if (lane == 0) {                                          // activations
      uint32_t dst = ring + 2 * kWTileBytes, bar = 0, parity = 1u;
      if (!DUAL && ks == 1) dst -= kWTileBytes;
      const uint32_t first = dst;
      const size_t chunk = (size_t)g.xrows_cap * kTileK;
      bool ok = true;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        int n_tile, split, mt, k0, k1;
        place(item, n_tile, split, mt, k0, k1);
        const uint32_t bytes = (uint32_t)round_up16(rows_of(mt)) * 128u;
        const __nv_bfloat16* x = g.X + (size_t)k0 * chunk + (size_t)(g.x_row0 + mt * g.mt_rows) * kTileK;
        for (int k = k0; k < k1; k += ks) {
          ok = step_wait(empty + bar, parity, sm, err);
          if (!ok) break;
          const bool two = !DUAL && ks == 2 && k + 1 < k1;
          step_expect(full + bar, two ? 2 * bytes : bytes);
          step_bulk(dst, x, bytes, full + bar);
          if (two) step_bulk(dst + g.xslot, x + chunk, bytes, full + bar);
          x += ks * chunk;
          dst += g.slot; bar += 8;
          if (bar == (uint32_t)g.stages * 8u) { dst = first; bar = 0; parity ^= 1u; }
        }
      }
      if (!ok) for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      const uint64_t dw0 = umma_desc_sw128(ring), xoff = (uint64_t)((DUAL || ks == 2 ? 2 : 1) * kWTileBytes / 16);
      uint64_t dw = dw0;
      uint32_t bar = 0, parity = 0u;
      int i = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x, ++i) {
        int n_tile, split, mt, k0, k1;
        place(item, n_tile, split, mt, k0, k1);
        const int b = i % g.bufs;
        const uint32_t idesc = umma_idesc_bf16(128, (uint32_t)round_up16(rows_of(mt)));
        const uint32_t d = sm->tmem_base + (uint32_t)(b * g.cols * PARTS);
        ok = step_wait(smem_u32(&sm->acc_empty[b]), ((i / g.bufs) & 1) ^ 1, sm, err);
        tc_fence_after();
        for (int k = k0; k < k1 && ok; k += ks) {
          ok = step_wait(full + bar, parity, sm, err);
          if (!ok) break;
          tc_fence_after();
          const uint64_t dx = dw + xoff;
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {                    // 32 bytes further on in each operand; addresses in descriptors count 16 bytes
            umma_bf16(d, dw + kk * 2, dx + kk * 2, idesc, (k > k0 || kk > 0) ? 1u : 0u);
            if (DUAL) umma_bf16(d + g.cols, dw + kWTileBytes / 16 + kk * 2, dx + kk * 2, idesc, (k > k0 || kk > 0) ? 1u : 0u);
          }
          if (!DUAL && ks == 2 && k + 1 < k1) {
            const uint64_t dx2 = dx + ((uint32_t)g.xslot >> 4);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) umma_bf16(d, dw + kWTileBytes / 16 + kk * 2, dx2 + kk * 2, idesc, 1u);
          }
          umma_commit(&sm->empty[bar >> 3]);
          dw += (uint32_t)g.slot >> 4; bar += 8;
          if (bar == (uint32_t)g.stages * 8u) { dw = dw0; bar = 0; parity ^= 1u; }
        }
        if (ok) umma_commit(&sm->acc_full[b]);
      }
    }
    __syncwarp();
  } else if (warp >= STEP_WARP0) {
    const int q = warp & 3, grp = (warp - STEP_WARP0) >> 2, G = g.groups;        // quarter of the lanes that this warp may read; the groups take the rows in turn
    if (EPI == STEP_HEAD) {
      for (int m = lane; m < g.M; m += 32)
        if ((m >> 4) % G == grp) best[q * 256 + m] = 0ull;
      __syncwarp();
    }
    int i = 0;
    for (int item = blockIdx.x; item < items; item += gridDim.x, ++i) {
      int n_tile, split, mt, k0, k1;
      place(item, n_tile, split, mt, k0, k1);
      const int b = i % g.bufs, m0 = mt * g.mt_rows, mlive = rows_of(mt);
      const int n = n_tile * kTileN + q * 32 + lane;
      const bool nvalid = n < g.N;
      if (!step_wait(smem_u32(&sm->acc_full[b]), (i / g.bufs) & 1, sm, err)) break;
      tc_fence_after();
      __syncwarp();
      const uint32_t taddr = sm->tmem_base + (uint32_t)(b * g.cols * PARTS) + ((uint32_t)(q * 32) << 16);
      for (int c0 = grp * 16; c0 < mlive; c0 += 16 * G) {
        const int r0 = g.x_row0 + m0 + c0, rows = min(16, mlive - c0);
        uint32_t v[16], up[16];
        tmem_ld16(taddr + c0, v);
        if (DUAL) tmem_ld16(taddr + g.cols + c0, up);
        tmem_ld_wait();
        if (EPI == STEP_PARTIAL) {
          float* out = reinterpret_cast<float*>(g.out) + (size_t)r0 * g.row_stride + (size_t)split * g.split_stride + n;
#pragma unroll
          for (int j = 0; j < 16; ++j)
            st_pred_f32(out + (size_t)j * g.row_stride, __uint_as_float(v[j]), nvalid && j < rows);
        } else if (EPI == STEP_SWIGLU_TAGGED) {
          unsigned long long* out = reinterpret_cast<unsigned long long*>(g.out) + (size_t)r0 * g.row_stride + (size_t)split * g.split_stride + n;
          const unsigned long long tg = (unsigned long long)g.tag << 32;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            st_pred_u64(out + (size_t)j * g.row_stride, tg | v[j], nvalid && j < rows);
            st_pred_u64(out + (size_t)j * g.row_stride + g.N, tg | up[j], nvalid && j < rows);
          }
        } else if (EPI == STEP_SWIGLU) {                       // rounding points: gemm_epilogue
          uint8_t* dst = reinterpret_cast<uint8_t*>(g.out) + ((size_t)(n >> 6) * g.out_rows_cap + r0) * 128 + (n & 7) * 2;      // r0: a multiple of 16
          const uint32_t chunk = (n & 63) >> 3;
          float gate[16], res[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) { gate[j] = bf16_round(__uint_as_float(v[j])); res[j] = bf16_round(__uint_as_float(up[j])); }
          swiglu_rows(gate, res);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const __nv_bfloat16 o = __float2bfloat16_rn(res[j]);
            st_pred_u16(dst + j * 128 + ((chunk ^ (j & 7)) << 4), *reinterpret_cast<const unsigned short*>(&o), nvalid && j < rows);
          }
        } else {
          if (g.out) {
            float* out = reinterpret_cast<float*>(g.out) + (size_t)(m0 + c0) * g.row_stride + n;
#pragma unroll
            for (int j = 0; j < 16; ++j) st_pred_f32(out + (size_t)j * g.row_stride, __uint_as_float(v[j]), nvalid && j < rows);
          }
          unsigned long long key[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) key[j] = nvalid ? argmax_key(bf16_round(__uint_as_float(v[j])), n) : 0ull;
          const unsigned long long mine = step_max16(key, lane);
          const int m = c0 + step_row(lane);
          if ((lane & 1) == 0 && m < mlive && mine > best[q * 256 + m]) best[q * 256 + m] = mine;
          __syncwarp();
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm->acc_empty[b]);
    }
    if (EPI == STEP_HEAD) {
      __syncwarp();
      for (int m = lane; m < g.M; m += 32) {
        const unsigned long long k = (m >> 4) % G == grp ? best[q * 256 + m] : 0ull;
        if (k != 0ull) atomicMax(&g.keys[g.x_row0 + m], k);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(sm->tmem_base, tm_cols);
}

// ---- row kernels ---------------------------------------------------------------------------------------------------------------------
// What rows_norm_impl does to one row: (embedding | the k-splits' sum, added to the residual row) -> hidden, then the RMS norm into the
// next product's operand.  One block per row, 8 columns per thread; the statistic by tiles of 128 columns, in the same trees.
struct StepNorm {
  const int* tok; const __nv_bfloat16* embed; int vocab;
  const float* part; int part_stride;                         // floats between rows; splits are h apart
  __nv_bfloat16* hidden; const __nv_bfloat16* w; int h; float eps;
  uint8_t* xn; int rows_cap;
};
template <int SPLITS>
__global__ void __launch_bounds__(1024) step_norm_kernel(const StepNorm a) {
  __shared__ float tile_ss[kMaxHTiles];
  if (SPLITS > 0) pdl_trigger();
  const int t = blockIdx.x, v = threadIdx.x, nvec = a.h >> 3, nt_h = (a.h + 127) >> 7, l16 = threadIdx.x & 15;
  __nv_bfloat16* hrow = a.hidden + (size_t)t * a.h;
  float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  uint4 wraw = make_uint4(0u, 0u, 0u, 0u);
  if (v < nvec) wraw = __ldg(reinterpret_cast<const uint4*>(a.w) + v);
  pdl_wait();
  if (SPLITS == 0) pdl_trigger();                             // the commits ahead of this forward are in their pages (step_attention_kernel)
  if (v < nvec) {
    if (SPLITS == 0) {
      int tk = a.tok[t];
      tk = tk < 0 ? 0 : (tk >= a.vocab ? a.vocab - 1 : tk);
      unpack8(__ldg(reinterpret_cast<const uint4*>(a.embed + (size_t)tk * a.h) + v), x);
    } else {
      const uint4 rr = reinterpret_cast<const uint4*>(hrow)[v];
      const float4* p = reinterpret_cast<const float4*>(a.part + (size_t)t * a.part_stride) + v * 2;
      const size_t stride = (size_t)a.h >> 2;
      float4 pa[SPLITS > 0 ? SPLITS : 1], pb[SPLITS > 0 ? SPLITS : 1];
#pragma unroll
      for (int s = 0; s < SPLITS; ++s) { pa[s] = p[s * stride]; pb[s] = p[s * stride + 1]; }
      float sr[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, r[8];
#pragma unroll
      for (int s = 0; s < SPLITS; ++s) {
        sr[0] += pa[s].x; sr[1] += pa[s].y; sr[2] += pa[s].z; sr[3] += pa[s].w;
        sr[4] += pb[s].x; sr[5] += pb[s].y; sr[6] += pb[s].z; sr[7] += pb[s].w;
      }
      unpack8(rr, r);
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = bf16_round(r[j] + bf16_round(sr[j]));
    }
    reinterpret_cast<uint4*>(hrow)[v] = pack8(x);
  }
  const float ss = halfwarp_tree(sumsq8(x));                  // lanes past the row's end bring zeros
  if (l16 == 0 && (v >> 4) < nt_h) tile_ss[v >> 4] = ss;
  __syncthreads();
  float p = 0.f;
  for (int s = l16; s < nt_h; s += 16) p += tile_ss[s];
  const float total = halfwarp_tree(p);
  if (v < nvec) {
    const float rstd = 1.0f / sqrtf(total / (float)a.h + a.eps);
    float wt[8], o[8];
    unpack8(wraw, wt);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = wt[j] * bf16_round(x[j] * rstd);
    *reinterpret_cast<uint4*>(a.xn + ((size_t)(v >> 3) * a.rows_cap + t) * 128 + (((v & 7) ^ (t & 7)) << 4)) = pack8(o);
  }
}

// Split gate/up: sums of the splits in order, silu(gate) * up into the down projection's operand (gu_swiglu_tail_impl).  8 features per thread, whose
// quotients do not wait for one another (swiglu_rows) and whose sums, read once, pass L1 by: 24 layers of the 0.5B shape, us, at 8 / 32 / 240 rows with division
// 1109 / 1369 / -, without 1043 / 1174 / 1913, past L1 1017 / 1092 / 1788.  By the last of a tile's k-splits to arrive instead, a launch less but few
// blocks: 1015 / 1156 / 2249.
template <int SPLITS>
__global__ void __launch_bounds__(128) step_swiglu_kernel(const unsigned long long* __restrict__ tgu, int N, int T, uint8_t* __restrict__ xact, int rows_cap) {
  pdl_trigger();
  pdl_wait();
  const int n0 = (blockIdx.x * 128 + threadIdx.x) * 8, t = blockIdx.y;
  if (n0 >= N) return;
  const unsigned long long* p = tgu + (size_t)t * SPLITS * 2 * N + n0;
  float sum[2][8];
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    ulonglong2 wd[SPLITS][4];
#pragma unroll
    for (int s = 0; s < SPLITS; ++s)
#pragma unroll
      for (int k = 0; k < 4; ++k) wd[s][k] = __ldcg(reinterpret_cast<const ulonglong2*>(p + ((size_t)s * 2 + g) * N + 2 * k));
#pragma unroll
    for (int k = 0; k < 8; ++k) sum[g][k] = 0.f;
#pragma unroll
    for (int s = 0; s < SPLITS; ++s)
#pragma unroll
      for (int k = 0; k < 4; ++k) { sum[g][2 * k] += tagged_val(wd[s][k].x); sum[g][2 * k + 1] += tagged_val(wd[s][k].y); }
#pragma unroll
    for (int k = 0; k < 8; ++k) sum[g][k] = bf16_round(sum[g][k]);
  }
  swiglu_rows(sum[0], sum[1]);
  *reinterpret_cast<uint4*>(xact + (size_t)(n0 >> 6) * rows_cap * 128 + sw128_offset((uint32_t)t, (uint32_t)(n0 & 63))) = pack8(sum[1]);
}

// What qkv_rope_impl does, one (row, head slot) per warp.
struct StepRope {
  const float* part; int row_stride, split_stride;
  const float* bias; const int* row_pos; const __nv_bfloat16 *cosb, *sinb;
  __nv_bfloat16 *qbuf, *k, *v;
  int T, n_q, n_kv, d, max_pos;
};
template <int SPLITS, int PPL>
__global__ void __launch_bounds__(256) step_rope_kernel(const StepRope a) {
  pdl_trigger();
  const int slots = a.n_q + 2 * a.n_kv, half = a.d >> 1, lane = threadIdx.x & 31;
  const int item = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (item >= a.T * slots) return;
  const int t = item / slots, slot = item - t * slots, e0 = lane * PPL;
  int pos = a.row_pos[t];                                     // of the plan: there before the forward's first kernel began
  pos = pos < 0 ? 0 : (pos >= a.max_pos ? a.max_pos - 1 : pos);
  float bl[PPL], bh[PPL], cs[PPL], sn[PPL];
#pragma unroll
  for (int j = 0; j < PPL; ++j) {
    bl[j] = __ldg(a.bias + slot * a.d + e0 + j); bh[j] = __ldg(a.bias + slot * a.d + half + e0 + j);
    cs[j] = __bfloat162float(__ldg(a.cosb + (size_t)pos * half + e0 + j)); sn[j] = __bfloat162float(__ldg(a.sinb + (size_t)pos * half + e0 + j));
  }
  pdl_wait();
  const float* p = a.part + (size_t)t * a.row_stride + slot * a.d + e0;
  float vl[SPLITS][PPL], vh[SPLITS][PPL];
#pragma unroll
  for (int s = 0; s < SPLITS; ++s) {
    if constexpr (PPL == 2) {
      const float2 l2 = *reinterpret_cast<const float2*>(p + (size_t)s * a.split_stride), h2 = *reinterpret_cast<const float2*>(p + (size_t)s * a.split_stride + half);
      vl[s][0] = l2.x; vl[s][PPL - 1] = l2.y; vh[s][0] = h2.x; vh[s][PPL - 1] = h2.y;
    } else {
      vl[s][0] = p[(size_t)s * a.split_stride];
      vh[s][0] = p[(size_t)s * a.split_stride + half];
    }
  }
  __nv_bfloat16* dst = slot < a.n_q ? a.qbuf + ((size_t)t * a.n_q + slot) * a.d
                                    : (slot < a.n_q + a.n_kv ? a.k + ((size_t)t * a.n_kv + slot - a.n_q) * a.d : a.v + ((size_t)t * a.n_kv + slot - a.n_q - a.n_kv) * a.d);
  float outl[PPL], outh[PPL];
#pragma unroll
  for (int j = 0; j < PPL; ++j) {
    float lo = 0.f, hi = 0.f;
#pragma unroll
    for (int s = 0; s < SPLITS; ++s) { lo += vl[s][j]; hi += vh[s][j]; }
    float l = bf16_round(lo + bl[j]), hv = bf16_round(hi + bh[j]);
    if (slot < a.n_q + a.n_kv) {
      const float nlo = bf16_round(bf16_round(l * cs[j]) - bf16_round(hv * sn[j]));
      const float nhi = bf16_round(bf16_round(hv * cs[j]) + bf16_round(l * sn[j]));
      l = nlo; hv = nhi;
    }
    outl[j] = l; outh[j] = hv;
  }
  if constexpr (PPL == 2) {
    *reinterpret_cast<uint32_t*>(dst + e0) = pack_bf16x2(outl[0], outl[PPL - 1]);
    *reinterpret_cast<uint32_t*>(dst + half + e0) = pack_bf16x2(outh[0], outh[PPL - 1]);
  } else {
    dst[e0] = __float2bfloat16_rn(outl[0]);
    dst[half + e0] = __float2bfloat16_rn(outh[0]);
  }
}

// ---- attention -----------------------------------------------------------------------------------------------------------------------
// The persistent kernel's unit (attention_unit) and merge (attn_combine_impl), one unit per block of four warps.  ONE_SUB: chunks of 64 keys, whose
// output starts at zero instead of being scaled: three blocks per SM without spills.  Eight sequences of the 7B shape (200 rows, 768 units) 15.9 -> 13.2 us
// against the general form; four blocks per SM (128 registers) 13.7, five (96) 14.0: bound by mma.sync and the fragments' loads, not by latency.
struct StepCtx {
  ModelDims md;
  int attn_chunk, max_pages_per_seq, num_pages, T_cap, xrows_cap;
  const int* block_tables;
  __nv_bfloat16 *kv_cache, *kv_scratch, *qbuf, *xa;
  float *attn_o, *attn_ml;
  const int2* row_attn;
};
struct StepWorker {
  uint8_t* smem;
  __device__ __forceinline__ int cta() const { return (int)blockIdx.x; }
  __device__ __forceinline__ int nctas() const { return (int)gridDim.x; }
  __device__ __forceinline__ int wtid() const { return (int)threadIdx.x; }
  __device__ __forceinline__ int wwarp() const { return (int)(threadIdx.x >> 5); }
  __device__ __forceinline__ int lane() const { return (int)(threadIdx.x & 31); }
  __device__ __forceinline__ uint8_t* attn_smem() const { return smem; }
  __device__ __forceinline__ const PlanCache* plan() const { return nullptr; }
};
__device__ __forceinline__ void prof_mark(const StepCtx&, const StepWorker&, int) {}

template <int D, bool ONE_SUB>
__global__ void __launch_bounds__(128, 3) step_attention_kernel(const __grid_constant__ StepCtx c, const Group* __restrict__ groups, int G, int layer, int plan_hs, int hs) {
  extern __shared__ __align__(16) uint8_t step_attn_smem[];
  pdl_trigger();
  const StepWorker w{step_attn_smem};
  const int u = blockIdx.x, lane = threadIdx.x & 31;
  // the plan was there before the forward's first kernel began; units of the plan are for plan_hs
  Group grp = {};
  for (int g0 = 0; g0 < G; g0 += 32) {                         // the last group whose first unit is not behind u
    const int4* p = reinterpret_cast<const int4*>(groups + min(g0 + lane, G - 1));
    const int4 a = p[0], b = p[1];
    const unsigned m = __ballot_sync(0xffffffffu, g0 + lane < G && b.z / plan_hs * hs <= u);
    if (m == 0u) break;
    const int l = 31 - __clz(m);
    grp.row0 = __shfl_sync(0xffffffffu, a.x, l); grp.len = __shfl_sync(0xffffffffu, a.y, l);
    grp.seq = __shfl_sync(0xffffffffu, a.z, l); grp.ctx = __shfl_sync(0xffffffffu, a.w, l);
    grp.nchunks = __shfl_sync(0xffffffffu, b.x, l); grp.qsplit = __shfl_sync(0xffffffffu, b.y, l);
    grp.unit0 = __shfl_sync(0xffffffffu, b.z, l); grp.slot0 = __shfl_sync(0xffffffffu, b.w, l);
  }
  int local = u - grp.unit0 / plan_hs * hs;
  const int kvh = local % c.md.n_kv; local /= c.md.n_kv;
  const int h = local % hs; local /= hs;
  const int chunk = local % grp.nchunks, k0 = chunk * c.attn_chunk;
  // Committed keys and values travel while the rotary stage ends: their pages were written before this forward, or by its commit
  // kernel, which was over when the first norm let later kernels start.
  if (k0 < grp.ctx) {
    const int page = c.block_tables[(size_t)grp.seq * c.max_pages_per_seq + k0 / kPage], rows = min(kAttnSub, grp.ctx - k0);
    for (int i = threadIdx.x; i < 2 * kAttnSub * (D / 8); i += 128) {
      const int kv = i / (kAttnSub * (D / 8)), r = i / (D / 8) % kAttnSub, v = i % (D / 8);
      if (r < rows)
        cp_async_16(reinterpret_cast<__nv_bfloat16*>(step_attn_smem) + (kv * kAttnSub + r) * (D + 8) + v * 8,
                    c.kv_cache + kv_cache_offset(c.md, c.num_pages, layer, kv, page, kvh, k0 % kPage) + (size_t)r * D + v * 8, 16);
    }
    cp_async_commit();
  }
  pdl_wait();
  attention_unit<D, true, ONE_SUB>(c, w, layer, grp, kvh, chunk, local / grp.nchunks, h, true, hs);
}

// attn_combine's merge of up to 32 chunks with a row's statistics and first eight chunks in flight at once, one (row, head) per warp.
template <int VPL>
__global__ void __launch_bounds__(256) step_combine_kernel(const __grid_constant__ StepCtx c, int T) {
  pdl_trigger();
  const int item = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31, D = c.md.d, n_q = c.md.n_q;
  if (item >= T * n_q) return;
  const int t = item / n_q, head = item - t * n_q;
  const int2 ra = c.row_attn[t];                              // of the plan: there before the forward's first kernel began
  const size_t base = (size_t)ra.x * n_q + head, ostride = (size_t)n_q * D;
  const float* ob = c.attn_o + base * D + lane * VPL;
  pdl_wait();
  if (ra.y >= 32) { attn_merge_long(c, t, head, base, ra.y, lane, VPL, D); return; }
  float2 ml = make_float2(-INFINITY, 0.f);
  if (lane <= ra.y) ml = *reinterpret_cast<const float2*>(c.attn_ml + (base + (size_t)lane * n_q) * 2);
  float v[8][VPL];
  auto load = [&](int c0) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float* op = ob + (size_t)min(c0 + u, ra.y) * ostride;
      if constexpr (VPL == 4) { const float4 x = *reinterpret_cast<const float4*>(op); v[u][0] = x.x; v[u][1] = x.y; v[u][VPL - 2] = x.z; v[u][VPL - 1] = x.w; }
      else { const float2 x = *reinterpret_cast<const float2*>(op); v[u][0] = x.x; v[u][1] = x.y; }
    }
  };
  load(0);
  float mx = ml.x;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const float wl = (ml.x == -INFINITY) ? 0.f : __expf(ml.x - mx), ll = wl * ml.y;
  float acc[4] = {0.f, 0.f, 0.f, 0.f}, l = 0.f;
  for (int c0 = 0; c0 <= ra.y; c0 += 8) {
    if (c0) load(c0);
#pragma unroll
    for (int u = 0; u < 8; ++u) {                              // chunk order
      float wgt = __shfl_sync(0xffffffffu, wl, (c0 + u) & 31), lc = __shfl_sync(0xffffffffu, ll, (c0 + u) & 31);
      if (c0 + u > ra.y) { wgt = 0.f; lc = 0.f; }
      l += lc;
#pragma unroll
      for (int j = 0; j < VPL; ++j) acc[j] += wgt * v[u][j];
    }
  }
  combine_store(c, t, head, lane, VPL, D, acc, l);
}

// ---- commits, results ------------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) step_commit_kernel(ModelDims md, const CommitEntry* __restrict__ commits, const int* __restrict__ tables, int max_pages,
                                                          int num_pages, int T_cap, const __nv_bfloat16* __restrict__ scratch, __nv_bfloat16* __restrict__ cache) {
  pdl_trigger();
  pdl_wait();
  const CommitEntry e = commits[blockIdx.x];
  const int layer = blockIdx.y >> 1, kv = blockIdx.y & 1, vpr = md.d >> 3;
  const int page = tables[(size_t)e.seq * max_pages + e.pos / kPage];
  for (int i = threadIdx.x; i < md.n_kv * vpr; i += blockDim.x) {
    const int kvh = i / vpr, v = i - kvh * vpr;
    reinterpret_cast<uint4*>(cache + kv_cache_offset(md, num_pages, layer, kv, page, kvh, e.pos % kPage))[v] =
        reinterpret_cast<const uint4*>(scratch + kv_scratch_offset(md, T_cap, layer, kv, e.src_row, kvh))[v];
  }
}
// planned forwards: tokens of the keys; the keys are clean for the next forward
__global__ void __launch_bounds__(256) step_greedy_kernel(unsigned long long* __restrict__ keys, int row0, int rows, int* __restrict__ greedy) {
  pdl_trigger();
  pdl_wait();
  const int t = row0 + blockIdx.x * 256 + threadIdx.x;
  if (t >= row0 + rows) return;
  greedy[t] = argmax_key_index(keys[t]);
  keys[t] = 0ull;
}

// The policy stage of a Jacobi run (policy_stage_jacobi) in a block with the persistent kernel's worker warps and shared-memory map.
constexpr size_t kPolicySmem = kSmemCtxOff + sizeof(DevCtx);
__global__ void __launch_bounds__(kNumThreads, 1) step_policy_kernel(const DevCtx* __restrict__ ctxp, bool first, int max_forwards) {
  uint4* dst = reinterpret_cast<uint4*>(jf_smem_base + kSmemCtxOff);
  for (int i = threadIdx.x; i < (int)(sizeof(DevCtx) / 16); i += blockDim.x) dst[i] = reinterpret_cast<const uint4*>(ctxp)[i];
  WorkerShared* ws = reinterpret_cast<WorkerShared*>(jf_smem_base + kSmemWsOff);
  if (threadIdx.x == 0) *ws = WorkerShared{};
  __syncthreads();
  const int warp = threadIdx.x >> 5;
  if (warp >= kWarpWorker0 && warp < kWarpWorker0 + 4) policy_stage_jacobi(*reinterpret_cast<const DevCtx*>(dst), ws, first, max_forwards);
}

// ---- host ----------------------------------------------------------------------------------------------------------------------------
struct StepPlan {
  int T, G, hsplit, units, max_len;                           // rows, groups, the plan's head split and attention units, the longest group
  int n_commit;                                               // commits of the forward before, ahead of this one
  int n_lm, parity, want_logits;
  const int *lm_row0, *lm_rows;
  unsigned int tag;
};

constexpr int kStepAhead = 4, kStepAheadFrom = 12, kStepAheadRows = 96;      // see step_forward
constexpr size_t kStepAheadBytes = 24 << 20;
inline size_t step_smem_bytes(const StepGemm& g, bool head) {
  return (size_t)g.stages * g.slot + sizeof(StepSmem) + (head ? 4 * 256 * 8 : 0) + 1024;
}

inline cudaError_t step_opt_in(int smem) {
  auto opt = [smem](auto kernel) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); };
  cudaError_t e = opt(step_gemm_kernel<STEP_PARTIAL>);
  if (e == cudaSuccess) e = opt(step_gemm_kernel<STEP_SWIGLU>);
  if (e == cudaSuccess) e = opt(step_gemm_kernel<STEP_SWIGLU_TAGGED>);
  if (e == cudaSuccess) e = opt(step_gemm_kernel<STEP_HEAD>);
  return e;
}

template <int EPI>
inline void step_product(WideStream& w, StepGemm g, int ctas, int smem_max, int* err) {
  constexpr bool DUAL = EPI == STEP_SWIGLU || EPI == STEP_SWIGLU_TAGGED, HEAD = EPI == STEP_HEAD;
  g.m_tiles = (g.M + 255) / 256;
  g.mt_rows = round_up16((g.M + g.m_tiles - 1) / g.m_tiles);
  g.m_tiles = (g.M + g.mt_rows - 1) / g.mt_rows;
  for (g.cols = 32; g.cols < g.mt_rows;) g.cols <<= 1;
  const int items = g.n_tiles * g.splits * g.m_tiles, grid = std::min(items, ctas);
  g.bufs = items > grid && g.cols * (DUAL ? 4 : 2) <= 512 ? 2 : 1;
  // Epilogue groups: one per 16 rows up to two, four where that measured faster.  A 7B forward (12 to 60 chunks of k a block), us, with two -> four: 24 rows
  // 2998 -> 2999, 33 rows 3023 -> 2995, 64 rows of ten layers 1235 -> 1219, 96 rows 3323 -> 3318, 100 rows 3452 -> 3435, 112 rows the same, 128 rows 3600 -> 3591
  // (3423 -> 3450 in another run): from 96 to 128 rows it makes no difference.  With few chunks a block of 600 threads starts later than it is done: the 0.5B shape's layers (5 to 10
  // chunks), 33 rows 1111 -> 1119, 64 rows 1197 -> 1352, 128 rows 1545 -> 1644.  Eleven stands between the two shapes; nothing in between was measured.  The head's tiles (14 and 56 chunks)
  // take as long with either, at 24 to 128 rows of both shapes.
  const int each = (g.k_chunks + g.splits - 1) / g.splits;
  g.groups = g.mt_rows > 128 || (g.mt_rows > 32 && g.mt_rows <= 96 && each >= 11) ? 4 : g.mt_rows > 16 ? 2 : 1;
  g.xslot = (g.mt_rows * 128 + 1023) & ~1023;
  g.stages = 0;
  const int room = smem_max - (int)step_smem_bytes(g, HEAD);
  g.ks = !DUAL && 4 * (2 * kWTileBytes + 2 * g.xslot) <= room ? 2 : 1;      // four stages of two chunks, or more of one
  g.slot = (DUAL ? 2 : g.ks) * kWTileBytes + g.ks * g.xslot;
  const int steps = ((g.k_chunks + g.splits - 1) / g.splits + g.ks - 1) / g.ks * ((items + grid - 1) / grid);
  g.stages = std::min(std::min(STEP_MAX_STAGES, steps), room / g.slot);
  w.launch(step_gemm_kernel<EPI>, grid, 32 * (STEP_WARP0 + 4 * g.groups), step_smem_bytes(g, HEAD), g, err);
}

inline void step_norm(WideStream& w, const DevCtx& c, int T, int splits, const float* part, const __nv_bfloat16* weight) {
  const StepNorm a{c.tok, c.embed, c.md.vocab_embed, part, c.part_splits * c.md.h, c.hidden, weight, c.md.h, c.md.eps, reinterpret_cast<uint8_t*>(c.xn), c.xrows_cap};
  const int threads = ((c.md.h >> 3) + 31) & ~31;
  switch (splits) {
    case 0: w.launch(step_norm_kernel<0>, T, threads, 0, a); break;
    case 1: w.launch(step_norm_kernel<1>, T, threads, 0, a); break;
    case 2: w.launch(step_norm_kernel<2>, T, threads, 0, a); break;
    case 3: w.launch(step_norm_kernel<3>, T, threads, 0, a); break;
    case 4: w.launch(step_norm_kernel<4>, T, threads, 0, a); break;
    case 5: w.launch(step_norm_kernel<5>, T, threads, 0, a); break;
    case 6: w.launch(step_norm_kernel<6>, T, threads, 0, a); break;
    case 7: w.launch(step_norm_kernel<7>, T, threads, 0, a); break;
    default: w.launch(step_norm_kernel<8>, T, threads, 0, a); break;
  }
}
template <int PPL>
inline void step_rope(WideStream& w, const StepRope& a, int splits) {
  const int blocks = (a.T * (a.n_q + 2 * a.n_kv) + 7) / 8;
  switch (splits) {
    case 1: w.launch(step_rope_kernel<1, PPL>, blocks, 256, 0, a); break;
    case 2: w.launch(step_rope_kernel<2, PPL>, blocks, 256, 0, a); break;
    case 3: w.launch(step_rope_kernel<3, PPL>, blocks, 256, 0, a); break;
    case 4: w.launch(step_rope_kernel<4, PPL>, blocks, 256, 0, a); break;
    case 5: w.launch(step_rope_kernel<5, PPL>, blocks, 256, 0, a); break;
    case 6: w.launch(step_rope_kernel<6, PPL>, blocks, 256, 0, a); break;
    case 7: w.launch(step_rope_kernel<7, PPL>, blocks, 256, 0, a); break;
    default: w.launch(step_rope_kernel<8, PPL>, blocks, 256, 0, a); break;
  }
}

inline void step_commit(WideStream& w, const DevCtx& c, int n_commit) {
  if (n_commit > 0)
    w.launch(step_commit_kernel, dim3(n_commit, 2 * c.md.layers), 128, 0, c.md, c.commits, c.block_tables, c.max_pages_per_seq, c.num_pages, c.T_cap, c.kv_scratch, c.kv_cache);
}

// The whole forward on w's stream; the plan's arrays are on the device already.  Argmax keys of the rows are left in half `parity`.
inline void step_forward(WideStream& w, const DevCtx& c, const StepPlan& p, int ctas, int smem_max, int* err) {
  const ModelDims& md = c.md;
  const int T = p.T, kc_h = md.h >> 6, kc_q = md.q_dim >> 6, kc_i = md.inter >> 6;
  const int nt_qkv = (md.qkv_dim + 127) >> 7, nt_h = (md.h + 127) >> 7, nt_i = (md.inter + 127) >> 7, nt_v = (md.vocab + 127) >> 7;
  auto product = [&](const __nv_bfloat16* W, const __nv_bfloat16* X, void* out, int n_tiles, int k_chunks, int splits, int N) {
    StepGemm g = {};
    g.W = W; g.X = X; g.out = out; g.n_tiles = n_tiles; g.k_chunks = k_chunks; g.splits = splits; g.M = T; g.N = N; g.xrows_cap = c.xrows_cap;
    g.out_rows_cap = c.xrows_cap;
    return g;
  };
  // HBM has nothing to do while the rotary stage, attention and its merge run, and again while the output projection ends: the weights of
  // gate and up that come behind the stages which their own kernel fills early are asked for from L2 then, by the products of queries and
  // outputs (`nth` 0 and 1), kStepAhead chunks of every tile each.  One 7B sequence in blocks of 32 100.2 -> 97.8 ms.  Four chunks from the twelfth on, twice; two
  // 98.0, six 98.0, from the sixth 98.2.  By the attention kernel instead, whose own keys come from HBM, 98.6 with four and 102.5 with twelve.
  // Where weights are what a layer waits for; with more rows it hides less of a layer.  A 7B forward, us, without -> with: 24 rows 3100 -> 3028, 64 rows 3188 -> 3163,
  // 96 rows 3366 -> 3356, where the line is; beyond it no more than at it is won or lost: 100 rows 3508 -> 3482, 128 rows 3645 -> 3635 (3421 -> 3460 in another run),
  // 160 rows 3870 -> 3843.
  auto ahead = [&](StepGemm& g, const LayerW& L, int nth) {
    const int from = kStepAheadFrom + nth * kStepAhead;
    if (T > kStepAheadRows || c.splits_gu > 1 || from + kStepAhead > kc_h || (size_t)2 * nt_i * kStepAhead * kWTileBytes > kStepAheadBytes) return;
    g.ahead = L.wgu + (size_t)from * (kTileN * kTileK); g.ahead_tiles = 2 * nt_i; g.ahead_stride = (size_t)kc_h * (kTileN * kTileK);
    g.ahead_bytes = kStepAhead * kWTileBytes;
  };
  auto partial = [&](const __nv_bfloat16* W, const __nv_bfloat16* X, float* out, int n_tiles, int k_chunks, int splits, int N, const LayerW* L = nullptr, int nth = 0) {
    StepGemm g = product(W, X, out, n_tiles, k_chunks, splits, N);
    if (L) ahead(g, *L, nth);
    g.row_stride = c.part_splits * N; g.split_stride = N;
    step_product<STEP_PARTIAL>(w, g, ctas, smem_max, err);
  };
  const StepCtx sc{md, c.attn_chunk, c.max_pages_per_seq, c.num_pages, c.T_cap, c.xrows_cap, c.block_tables, c.kv_cache, c.kv_scratch, c.qbuf, c.xa,
                   c.attn_o, c.attn_ml, c.row_attn};
  // heads of a unit: one round of four 16-row tiles per block, however long the longest group is (attention_unit's ONE_ROUND)
  const int row_tiles = (std::min(p.max_len, kQTokPerUnit) + 15) / 16, hs = (md.n_rep + 4 / row_tiles - 1) / (4 / row_tiles), units = p.units / p.hsplit * hs;
  const size_t attn_smem = (size_t)2 * kAttnSub * (md.d + 8) * 2;
  const int combine = (T * md.n_q + 7) / 8;
  w.mark(SID_NONE);
  step_commit(w, c, p.n_commit);
  step_norm(w, c, T, 0, nullptr, c.layer[0].ln1);
  w.mark(SID_EMBED);
  for (int l = 0; l < md.layers && !w.failed; ++l) {
    const LayerW& L = c.layer[l];
    partial(L.wqkv, c.xn, c.part, nt_qkv, kc_h, c.splits_qkv, md.qkv_dim, &L, 0);
    w.mark(SID_QKV);
    const StepRope r{c.part, c.part_splits * c.part_n, c.part_n, L.bqkv, c.row_pos, c.rope_cos, c.rope_sin, c.qbuf,
                     c.kv_scratch + kv_scratch_offset(md, c.T_cap, l, 0, 0, 0), c.kv_scratch + kv_scratch_offset(md, c.T_cap, l, 1, 0, 0),
                     T, md.n_q, md.n_kv, md.d, md.max_pos};
    if (md.d == 128) step_rope<2>(w, r, c.splits_qkv); else step_rope<1>(w, r, c.splits_qkv);
    w.mark(SID_ROPE);
    auto attention = [&](auto kernel) { w.launch(kernel, units, 128, attn_smem, sc, c.groups, p.G, l, p.hsplit, hs); };
    if (md.d == 128) { if (c.attn_chunk == kAttnSub) attention(step_attention_kernel<128, true>); else attention(step_attention_kernel<128, false>); }
    else { if (c.attn_chunk == kAttnSub) attention(step_attention_kernel<64, true>); else attention(step_attention_kernel<64, false>); }
    w.mark(SID_ATTN);
    if (md.d == 128) w.launch(step_combine_kernel<4>, combine, 256, 0, sc, T); else w.launch(step_combine_kernel<2>, combine, 256, 0, sc, T);
    w.mark(SID_COMBINE);
    partial(L.wo, c.xa, c.part_rs[0], nt_h, kc_q, c.splits_o, md.h, &L, 1);
    w.mark(SID_O);
    step_norm(w, c, T, c.splits_o, c.part_rs[0], L.ln2);
    w.mark(SID_O_NORM);
    if (c.splits_gu > 1) {
      StepGemm g = product(L.wgu, c.xn, c.tgu, nt_i, kc_h, c.splits_gu, md.inter);
      g.tag = p.tag; g.row_stride = c.splits_gu * 2 * md.inter; g.split_stride = 2 * md.inter;
      step_product<STEP_SWIGLU_TAGGED>(w, g, ctas, smem_max, err);
      const dim3 grid((md.inter / 8 + 127) / 128, T);
      switch (c.splits_gu) {
        case 2: w.launch(step_swiglu_kernel<2>, grid, 128, 0, c.tgu, md.inter, T, reinterpret_cast<uint8_t*>(c.xact), c.xrows_cap); break;
        case 3: w.launch(step_swiglu_kernel<3>, grid, 128, 0, c.tgu, md.inter, T, reinterpret_cast<uint8_t*>(c.xact), c.xrows_cap); break;
        default: w.launch(step_swiglu_kernel<4>, grid, 128, 0, c.tgu, md.inter, T, reinterpret_cast<uint8_t*>(c.xact), c.xrows_cap); break;
      }
    } else {
      step_product<STEP_SWIGLU>(w, product(L.wgu, c.xn, c.xact, nt_i, kc_h, 1, md.inter), ctas, smem_max, err);
    }
    w.mark(SID_GU);
    partial(L.wd, c.xact, c.part_rs[1], nt_h, kc_i, c.splits_down, md.h);
    w.mark(SID_DOWN);
    step_norm(w, c, T, c.splits_down, c.part_rs[1], l + 1 < md.layers ? c.layer[l + 1].ln1 : c.final_norm);
    w.mark(SID_DOWN_NORM);
  }
  for (int i = 0; i < p.n_lm; ++i) {
    StepGemm g = product(c.lm_head, c.xn, i == 0 && p.want_logits ? c.logits : nullptr, nt_v, kc_h, 1, md.vocab);
    g.M = p.lm_rows[i]; g.x_row0 = p.lm_row0[i]; g.row_stride = md.vocab;
    g.keys = c.argmax_keys + (size_t)p.parity * c.T_cap;
    step_product<STEP_HEAD>(w, g, ctas, smem_max, err);
  }
  w.mark(SID_LM);
}

}  // namespace jf
