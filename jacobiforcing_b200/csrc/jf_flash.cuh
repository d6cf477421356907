// jf_flash.cuh — softmax attention of prompt-sized steps on the 5th-generation tensor cores, shared by both engines.
//
// A block serves 128 rows, a row being a (head, token) pair of one key head of one request, and walks the key tiles of 128 that
// its rows see.  S = Q K^T and O += P V run as tcgen05.mma with the accumulators in tensor memory; one thread per row reads its
// scores from there, and the weights go back to tensor memory as the second product's first operand (bf16, or with SPLIT as a
// bf16 head plus a bf16 remainder and two products, so that a weight keeps about 16 bits of its mantissa).  The scores of tile
// j + 1 are made while the softmax of tile j runs.  The accumulated output is rescaled only when a row's maximum has grown by
// more than a factor of 2^8 (any reference point is as good as the maximum as long as nothing overflows; all sums are fp32).
// Keys and values travel by TMA, from pages of 256 tokens or from rows made for the step.
//
// Warp 0: producer (one lane).  Warp 1: owns tensor memory, one lane issues the products.  Warps 2-5: softmax, one thread per row.
// Tensor memory: scores 2 x 128 columns, output 128, weights 64 + 64 (remainder).  Every wait on an mbarrier is bounded (see tp_wait): on
// a timeout the kernel raises the error flag, stops waiting, lets its copies land and frees its tensor memory.  The allocation of tensor
// memory waits without a limit; jf_pair.cuh says why it ends.
#pragma once
#include "jf_pair.cuh"

namespace jf {

constexpr int FL_THREADS = 192;
constexpr int FL_KEYS = 128;

// Rows pair0 .. pair0 + 127 (at most heads * len) of key head `kvh`: pair p is token row0 + p % len (position pos0 + p % len) of head
// head0 + p / len.  The key of position j is in the pages of the table at `table`, or (table < 0) row own_row0 + j of the maps, columns of
// key head `kvh`.
struct FlashUnit { int row0, len, pair0, pairs, head0, kvh, pos0, own_row0, table; };

struct FlashArgs {
  const FlashUnit* units;
  const __nv_bfloat16* q; size_t ldq; int q_head;        // head h's query at column h * q_head
  const int* page_table; int kv_heads;                   // pages: row ((page * kv_heads + kvh) * 256 + slot) of the maps
  float scale; int window;                               // window > 0: only keys j with i - j < window
  const __nv_bfloat16* sink;                             // [heads] a logit without key and value (NULL: none)
  const __nv_bfloat16* gate; size_t ldg;                 // output times sigmoid(gate[row, head * DV + d]) (NULL: none)
  __nv_bfloat16* out; size_t ldo;                        // row-major [row, head * DV + d], or (packed_rows > 0) [chunk of 64][packed_rows][64] swizzled
  int packed_rows;
  int* err;
};

struct FlSmem {
  uint64_t k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], s_free[2], q_full, p_full, o_done;
  uint32_t tmem_base, failed;
};
__host__ __device__ constexpr size_t fl_smem_bytes(int dk, int dv) {
  return (size_t)(dk / 64) * 16384 * 3 + (size_t)(dv / 64) * 16384 * 2 + sizeof(FlSmem) + 1024;
}

__device__ __forceinline__ bool fl_wait(uint64_t* bar, uint32_t parity, FlSmem* sm, int* err) {
  if (sm->failed) return false;
  for (uint32_t i = 0; i < TC_SPIN_LIMIT; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  sm->failed = 1;
  atomicExch(err, 1);
  return false;
}
__device__ __forceinline__ void fl_load(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar)) : "memory");
}

// The key tiles of a unit, aligned to absolute positions.
struct FlTiles {
  int lo, n;                                             // first position of the first tile (a multiple of 128), tiles
  __device__ FlTiles(const FlashUnit& u, int window) {
    const int rows = min(128, u.pairs - u.pair0), a = u.pair0 % u.len, b = a + rows - 1;
    const int first_tok = b < u.len ? a : 0, last_tok = b < u.len ? b : u.len - 1;
    lo = (window > 0 ? max(0, u.pos0 + first_tok - window + 1) : 0) / FL_KEYS * FL_KEYS;
    n = (u.pos0 + last_tok - lo) / FL_KEYS + 1;
  }
};

template <int DK, int DV, bool SPLIT>
__global__ void __launch_bounds__(FL_THREADS, 1)
flash_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap, FlashArgs a) {
  extern __shared__ __align__(16) unsigned char tp_smem[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tp_smem) + 1023) & ~(uintptr_t)1023);
  constexpr int KC = DK / 64, VC = DV / 64, CHUNK = 16384;
  unsigned char* sq = base;
  unsigned char* sk = sq + KC * CHUNK;                     // [2]
  unsigned char* sv = sk + 2 * KC * CHUNK;                 // [2]
  FlSmem* sm = reinterpret_cast<FlSmem*>(sv + 2 * VC * CHUNK);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sm->k_full[i], 1); mbar_init(&sm->k_empty[i], 1); mbar_init(&sm->v_full[i], 1); mbar_init(&sm->v_empty[i], 1);
      mbar_init(&sm->s_full[i], 1); mbar_init(&sm->s_free[i], 4);
    }
    mbar_init(&sm->q_full, 128); mbar_init(&sm->p_full, 4); mbar_init(&sm->o_done, 1);
    sm->failed = 0;
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc(&sm->tmem_base, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_trigger();                                           // this block owns its columns
  pdl_wait();
  const FlashUnit u = a.units[blockIdx.x];
  const FlTiles tiles(u, a.window);
  const uint32_t tm = sm->tmem_base;

  if (warp == 0) {
    if (lane == 0) {
      bool ok = true;
      for (int j = 0; j < tiles.n && ok; ++j) {
        const int s = j & 1;
        const uint32_t ph = ((j >> 1) & 1) ^ 1;
        const int p = tiles.lo + j * FL_KEYS;
        const bool paged = u.table >= 0;
        const int row = paged ? (a.page_table[u.table + p / 256] * a.kv_heads + u.kvh) * 256 + p % 256 : u.own_row0 + p;
        const int xk = paged ? 0 : u.kvh * DK, xv = paged ? 0 : u.kvh * DV;
        ok = fl_wait(&sm->k_empty[s], ph, sm, a.err);
        if (!ok) break;
        mbar_expect_tx(&sm->k_full[s], KC * CHUNK);
#pragma unroll
        for (int c = 0; c < KC; ++c) fl_load(sk + (s * KC + c) * CHUNK, &kmap, xk + c * 64, row, &sm->k_full[s]);
        ok = fl_wait(&sm->v_empty[s], ph, sm, a.err);
        if (!ok) break;
        mbar_expect_tx(&sm->v_full[s], VC * CHUNK);
#pragma unroll
        for (int c = 0; c < VC; ++c) fl_load(sv + (s * VC + c) * CHUNK, &vmap, xv + c * 64, row, &sm->v_full[s]);
      }
      if (!ok) for (int i = 0; i < 1000; ++i) __nanosleep(1000);    // copies in flight land before the block leaves
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t is = umma_idesc_bf16(128, FL_KEYS), io = umma_idesc_bf16_bmn(128, DV);
      const uint32_t aq = smem_u32(sq), ak = smem_u32(sk), av = smem_u32(sv);
      bool ok = fl_wait(&sm->q_full, 0, sm, a.err);
      auto output = [&](int j) {                              // O += P V of tile j
        const int s = j & 1;
        ok = ok && fl_wait(&sm->p_full, j & 1, sm, a.err) && fl_wait(&sm->v_full[s], (j >> 1) & 1, sm, a.err);
        if (!ok) return;
        tc_fence_after();
#pragma unroll
        for (int part = 0; part < (SPLIT ? 2 : 1); ++part)
#pragma unroll
          for (int kk = 0; kk < FL_KEYS / 16; ++kk)
            umma_bf16_ts(tm + 256, tm + 384 + part * 64 + kk * 8, umma_desc_sw128_mn(av + s * VC * CHUNK + kk * 2048, CHUNK, 1024), io,
                         (j > 0 || part > 0 || kk > 0) ? 1u : 0u);
        umma_commit(&sm->v_empty[s]);
        umma_commit(&sm->o_done);
      };
      for (int j = 0; j < tiles.n && ok; ++j) {
        const int s = j & 1;
        ok = fl_wait(&sm->k_full[s], (j >> 1) & 1, sm, a.err) && fl_wait(&sm->s_free[s], ((j >> 1) & 1) ^ 1, sm, a.err);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < DK / 16; ++kk)
          umma_bf16(tm + s * 128, umma_desc_sw128(aq + (kk >> 2) * CHUNK + (kk & 3) * 32), umma_desc_sw128(ak + (s * KC + (kk >> 2)) * CHUNK + (kk & 3) * 32),
                    is, kk > 0 ? 1u : 0u);
        umma_commit(&sm->k_empty[s]);
        umma_commit(&sm->s_full[s]);
        if (j > 0) output(j - 1);
      }
      if (ok) output(tiles.n - 1);
    }
    __syncwarp();
  } else {
    const int q4 = warp & 3, r = q4 * 32 + lane;                // this thread's row: lane r of tensor memory
    const uint32_t tl = tm + ((uint32_t)(q4 * 32) << 16);
    const int p = min(u.pair0 + r, u.pairs - 1);                // rows beyond the last repeat it and are not stored
    const bool live = u.pair0 + r < u.pairs;
    const int tok = p % u.len, head = u.head0 + p / u.len, pos = u.pos0 + tok;
    const size_t row = (size_t)(u.row0 + tok);
    {                                                           // query row -> swizzled shared memory
      const uint4* src = reinterpret_cast<const uint4*>(a.q + row * a.ldq + (size_t)head * a.q_head);
#pragma unroll
      for (int c = 0; c < DK / 8; ++c)
        *reinterpret_cast<uint4*>(sq + (c >> 3) * CHUNK + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = src[c];
      fence_proxy_async_smem();
      mbar_arrive(&sm->q_full);
    }
    const float c2 = a.scale * 1.4426950408889634f;             // scores in units of log 2
    const int first = a.window > 0 ? max(0, pos - a.window + 1) : 0;
    float m = -INFINITY, l = 0.0f;                              // reference point and sum of the weights so far
    bool ok = true;
    for (int j = 0; j < tiles.n; ++j) {
      const int s = j & 1;
      const int k0 = tiles.lo + j * FL_KEYS;
      ok = fl_wait(&sm->s_full[s], (j >> 1) & 1, sm, a.err);
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
      uint32_t x[128];                                          // the scores
#pragma unroll
      for (int c = 0; c < 8; ++c) tmem_ld16(tl + s * 128 + c * 16, *reinterpret_cast<uint32_t(*)[16]>(&x[c * 16]));
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm->s_free[s]);
      const int end = min(pos + 1, k0 + FL_KEYS);               // keys [first, end) of this tile
      if (first > k0 || end < k0 + FL_KEYS) {
#pragma unroll
        for (int k = 0; k < 128; ++k)
          if (k0 + k < first || k0 + k >= end) x[k] = 0xff800000u;                // minus infinity
      }
      float t0 = -INFINITY, t1 = -INFINITY, t2 = -INFINITY, t3 = -INFINITY;
#pragma unroll
      for (int k = 0; k < 128; k += 4) {
        t0 = fmaxf(t0, __uint_as_float(x[k])); t1 = fmaxf(t1, __uint_as_float(x[k + 1]));
        t2 = fmaxf(t2, __uint_as_float(x[k + 2])); t3 = fmaxf(t3, __uint_as_float(x[k + 3]));
      }
      const float top = fmaxf(fmaxf(t0, t1), fmaxf(t2, t3)) * c2;
      float grow = 1.0f;
      const bool moves = top > m + 8.0f || (m == -INFINITY && top > -INFINITY);
      if (moves) { grow = exp2f(m - top); m = top; l *= grow; }
      const float ref = m == -INFINITY ? 0.0f : m;
      uint32_t hi[64], lo[SPLIT ? 64 : 1];
      float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
      for (int k = 0; k < 128; k += 2) {
        const float e0 = exp2f(fmaf(__uint_as_float(x[k]), c2, -ref)), e1 = exp2f(fmaf(__uint_as_float(x[k + 1]), c2, -ref));
        s0 += e0; s1 += e1;
        const uint32_t h = pack_bf16x2(e0, e1);
        hi[k >> 1] = h;
        if constexpr (SPLIT) lo[k >> 1] = pack_bf16x2(e0 - __uint_as_float(h << 16), e1 - __uint_as_float(h & 0xffff0000u));
      }
      l += s0 + s1;
      if (j > 0) {                                              // the product of the tile before has read the weights and written the output
        ok = fl_wait(&sm->o_done, (j - 1) & 1, sm, a.err);
        if (!__all_sync(0xffffffffu, ok)) break;
        tc_fence_after();
        if (__any_sync(0xffffffffu, moves)) {
#pragma unroll
          for (int c = 0; c < DV / 16; ++c) {
            uint32_t o[16];
            tmem_ld16(tl + 256 + c * 16, o);
            tmem_ld_wait();
#pragma unroll
            for (int k = 0; k < 16; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * grow);
            tmem_st16(tl + 256 + c * 16, o);
          }
        }
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        tmem_st16(tl + 384 + c * 16, *reinterpret_cast<uint32_t(*)[16]>(&hi[c * 16]));
        if constexpr (SPLIT) tmem_st16(tl + 448 + c * 16, *reinterpret_cast<uint32_t(*)[16]>(&lo[c * 16]));
      }
      tmem_st_wait();
      if (k0 + FL_KEYS > u.pos0 + u.len) {                      // value rows behind the last key: a weight of zero does not silence what is no number
        ok = fl_wait(&sm->v_full[s], (j >> 1) & 1, sm, a.err);
        if (!__all_sync(0xffffffffu, ok)) break;
        if (k0 + r >= u.pos0 + u.len) {
#pragma unroll
          for (int c = 0; c < VC * 8; ++c) *reinterpret_cast<uint4*>(sv + (s * VC + (c >> 3)) * CHUNK + r * 128 + (c & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
        }
        fence_proxy_async_smem();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm->p_full);
    }
    ok = ok && fl_wait(&sm->o_done, (tiles.n - 1) & 1, sm, a.err);
    if (__all_sync(0xffffffffu, ok)) {
      tc_fence_after();
      if (a.sink) l += exp2f(__bfloat162float(a.sink[head]) * 1.4426950408889634f - m);
      const float inv = 1.0f / l;
#pragma unroll
      for (int c = 0; c < DV / 16; ++c) {
        uint32_t o[16];
        tmem_ld16(tl + 256 + c * 16, o);
        tmem_ld_wait();
        if (!live) continue;
        float y[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) y[k] = __uint_as_float(o[k]) * inv;
        if (a.gate) {
          const __nv_bfloat16* g = a.gate + row * a.ldg + (size_t)head * DV + c * 16;
#pragma unroll
          for (int k = 0; k < 16; ++k) y[k] *= 1.0f / (1.0f + expf(-__bfloat162float(g[k])));
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint4 w = make_uint4(pack_bf16x2(y[8 * h], y[8 * h + 1]), pack_bf16x2(y[8 * h + 2], y[8 * h + 3]), pack_bf16x2(y[8 * h + 4], y[8 * h + 5]),
                                     pack_bf16x2(y[8 * h + 6], y[8 * h + 7]));
          const int f = head * DV + c * 16 + h * 8;
          if (a.packed_rows)
            *reinterpret_cast<uint4*>(reinterpret_cast<unsigned char*>(a.out) + (size_t)(f >> 6) * a.packed_rows * 128 + sw128_offset((uint32_t)row, (uint32_t)(f & 63))) = w;
          else *reinterpret_cast<uint4*>(a.out + row * a.ldo + f) = w;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tm, 512);
}

}  // namespace jf
