// jf_flash.cuh — softmax attention of prompt-sized steps on the 5th-generation tensor cores, shared by both engines.
//
// A block serves 128 rows, a row being a (head, token) pair of one key head of one request, and walks the key tiles of 128 that
// its rows see.  S = Q K^T and O += P V run as tcgen05.mma with the accumulators in tensor memory; two threads per row read its
// scores from there, and the weights go back over the scores as the second product's first operand (bf16, or with SPLIT as a
// bf16 head plus a bf16 remainder and two products, so that a weight keeps about 16 bits of its mantissa).  The accumulated output is
// rescaled only when a row's maximum has grown by more than a factor of 2^8 (any reference point is as good as the maximum as long as
// nothing overflows; all sums are fp32).
// What a key tile takes is a chain: scores, softmax, output, each behind a barrier; the products are a quarter of it.  So half of an SM's shared memory
// and tensor memory is all that a block takes (heads of up to 128), and the other block's chain fills its gaps; two threads per row halve the
// softmax.  What showed in cycle counts per key tile of a block: 3700 in all, 2250 of them softmax with one thread per row and all 128 scores in
// registers at once (code that comes by once per tile is fetched once per tile: 450 for the largest score, up to 2800 with a mask), 300 to 580 for
// every wait that was over already (with its slow path in line), 8000 in front of the first scores (query rows read by a lane each).
// 1000 tokens of 28 heads of 128 over four key heads, us: one block of one thread per row and SM 37, two tiles of rows in a block with their chains
// overlapped by its warps 29 to 31, this 27; 1531 tokens behind 2048, 16 heads of 128 + 64, weights split: 152, 119, 112.
// Keys and values travel by TMA, from pages of 256 tokens or from rows made for the step.
//
// Warp 0: producer (one lane).  Warp 1: owns tensor memory, one lane issues the products.  Warps 2-9: softmax, two threads per row.
// Tensor memory: scores 128 columns (then, in the place of every 32 scores, 16 columns of weights and 16 of remainders), output 128.  Products with
// unlike accumulators are not promised to run one behind the other, so the next scores are issued once the product that reads the weights in their
// place is over (its commit, which also gives the values' stage back).  An mbarrier that a product is committed to stands for all products
// issued before it: once scores are there, the output holds everything before.
// Every wait on an mbarrier is bounded (see tp_wait): on a timeout the kernel raises the error flag, stops waiting, lets its copies land
// and frees its tensor memory.  The allocation of tensor memory waits without a limit; jf_pair.cuh says why it ends.
#pragma once
#include "jf_pair.cuh"

namespace jf {

constexpr int FL_THREADS = 320;
constexpr int FL_KEYS = 128;
constexpr int FL_ROWS = 128;                             // rows of a unit

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
  // beyond what every caller has (zeros: none of it)
  int chunk;                                             // position i sees no keys before i / chunk * chunk (instead of a window)
  float temp_coef; int temp_every;                       // scores times 1 + coef ln(floor((i + 1) / every) + 1) as well
  const float* slope;                                    // [heads] slope (i - j) is taken off a score (kernels with BIAS)
  const float* sink_f;                                   // the sinks as fp32
  const float* head_gate; size_t ld_head;                // output times sigmoid(head_gate[row, head])
  int scaled; float out_scale;                           // scaled: output times out_scale
  __device__ __forceinline__ int first(int pos) const { return chunk > 0 ? pos / chunk * chunk : window > 0 ? max(0, pos - window + 1) : 0; }
};

constexpr int FL_MAX_STAGES = 2;
struct FlSmem {
  uint64_t k_full[FL_MAX_STAGES], k_empty[FL_MAX_STAGES], v_full[FL_MAX_STAGES], v_empty[FL_MAX_STAGES], s_full, q_full, p_full, o_done;
  uint32_t tmem_base, failed;
  float part[2][FL_ROWS];                                // per half of the keys and row: largest score, at the end sum of weights
};
// Stages of key and value tiles.  One: a tile's keys are read long before the next one's scores are wanted, its values before the next one's
// weights are made, so that a second stage hides nothing, and two blocks fit an SM.
__host__ __device__ constexpr int fl_stages(int dk) { return dk > 128 ? 2 : 1; }
__host__ __device__ constexpr size_t fl_smem_bytes(int dk, int dv) {
  return (size_t)(dk / 64) * 16384 * (1 + fl_stages(dk)) + (size_t)(dv / 64) * 16384 * fl_stages(dk) + sizeof(FlSmem);
}

// Out of line: what follows a wait that is over already is fetched with it.
__device__ __noinline__ bool fl_wait_on(uint64_t* bar, uint32_t parity, FlSmem* sm, int* err) {
  for (uint32_t i = 0; i < TC_SPIN_LIMIT; ++i) {
    if (sm->failed) return false;
    if (mbar_try_wait(bar, parity)) return true;
  }
  sm->failed = 1;
  atomicExch(err, 1);
  return false;
}
__device__ __forceinline__ bool fl_wait(uint64_t* bar, uint32_t parity, FlSmem* sm, int* err) {
  if (mbar_try_wait(bar, parity)) return true;
  return fl_wait_on(bar, parity, sm, err);
}
__device__ __forceinline__ void fl_load(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar)) : "memory");
}

// The key tiles of a unit, aligned to absolute positions: first one's number, how many.
struct FlTiles {
  int lo, n;
  __device__ FlTiles(const FlashUnit& u, const FlashArgs& a) {
    const int rows = min(FL_ROWS, u.pairs - u.pair0), i = u.pair0 % u.len, b = i + rows - 1;
    const int first_tok = b < u.len ? i : 0, last_tok = b < u.len ? b : u.len - 1;
    lo = a.first(u.pos0 + first_tok) / FL_KEYS;
    n = (u.pos0 + last_tok) / FL_KEYS + 1 - lo;
  }
};
// 2^y in units of the last place of ex2.approx; what would be subnormal is zero
__device__ __forceinline__ float fl_exp2(float y) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y)); return r; }

template <int DK, int DV, bool SPLIT, bool BIAS = false, int BLOCKS = fl_stages(DK) == 1 ? 2 : 1>
__global__ void __launch_bounds__(FL_THREADS, BLOCKS)
flash_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap, FlashArgs a) {
  extern __shared__ __align__(1024) unsigned char fl_smem[];
  constexpr int KC = DK / 64, VC = DV / 64, ST = fl_stages(DK), CHUNK = 16384, COLUMNS = 256;
  unsigned char* sq = fl_smem;
  unsigned char* sk = sq + KC * CHUNK;                     // [ST]
  unsigned char* sv = sk + ST * KC * CHUNK;                // [ST]
  FlSmem* sm = reinterpret_cast<FlSmem*>(sv + ST * VC * CHUNK);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < ST; ++i) {
      mbar_init(&sm->k_full[i], 1); mbar_init(&sm->k_empty[i], 1); mbar_init(&sm->v_full[i], 1); mbar_init(&sm->v_empty[i], 1);
    }
    mbar_init(&sm->s_full, 1); mbar_init(&sm->q_full, 256); mbar_init(&sm->p_full, 8); mbar_init(&sm->o_done, 1);
    sm->failed = 0;
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc(&sm->tmem_base, COLUMNS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_trigger();                                           // this block owns its columns
  pdl_wait();
  const FlashUnit u = a.units[blockIdx.x];
  const FlTiles t(u, a);
  const uint32_t tm = sm->tmem_base;

  if (warp == 0) {
    if (lane == 0) {
      bool ok = true;
      for (int i = 0; i < t.n && ok; ++i) {
        const int s = i % ST, p = (t.lo + i) * FL_KEYS;
        const uint32_t ph = ((i / ST) & 1) ^ 1;
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
      const uint64_t dq = umma_desc_sw128(smem_u32(sq)), dk = umma_desc_sw128(smem_u32(sk)), dv = umma_desc_sw128_mn(smem_u32(sv), CHUNK, 1024);
      bool ok = fl_wait(&sm->q_full, 0, sm, a.err);
#pragma unroll 1
      for (int i = -1; i < t.n && ok; ++i) {                 // O += P V of tile i, then S of tile i + 1
        if (i >= 0) {
          const int s = i % ST;
          ok = fl_wait(&sm->p_full, i & 1, sm, a.err) && fl_wait(&sm->v_full[s], (i / ST) & 1, sm, a.err);
          if (!ok) break;
          tc_fence_after();
          const uint64_t d = dv + (uint64_t)(s * VC * CHUNK >> 4);
#pragma unroll 1
          for (int part = 0; part < (SPLIT ? 2 : 1); ++part)
#pragma unroll
            for (int kk = 0; kk < FL_KEYS / 16; ++kk)
              umma_bf16_ts(tm + 128, tm + part * 16 + (kk >> 1) * 32 + (kk & 1) * 8, d + (uint64_t)(kk * 2048 >> 4), io, (kk > 0 || part > 0 || i > 0) ? 1u : 0u);
          umma_commit(&sm->v_empty[s]);
        }
        if (i + 1 < t.n) {
          const int s = (i + 1) % ST;
          ok = fl_wait(&sm->k_full[s], ((i + 1) / ST) & 1, sm, a.err) && (i < 0 || fl_wait(&sm->v_empty[i % ST], (i / ST) & 1, sm, a.err));
          if (!ok) break;
          tc_fence_after();
          const uint64_t k = dk + (uint64_t)(s * KC * CHUNK >> 4);
#pragma unroll
          for (int kk = 0; kk < DK / 16; ++kk) {
            constexpr int UP = CHUNK >> 4;
            umma_bf16(tm, dq + (uint64_t)((kk >> 2) * UP + (kk & 3) * 2), k + (uint64_t)((kk >> 2) * UP + (kk & 3) * 2), is, kk > 0 ? 1u : 0u);
          }
          umma_commit(&sm->s_full);
          umma_commit(&sm->k_empty[s]);
        } else {
          umma_commit(&sm->o_done);
        }
      }
    }
    __syncwarp();
  } else {
    // this thread's half of every 128 keys (and of the output's columns) and row: lane r of tensor memory
    const int half = warp >= 6, q4 = warp & 3, r = q4 * 32 + lane;
    {
      const uint32_t ts = tm + ((uint32_t)(q4 * 32) << 16), to = ts + 128;
      const int p = min(u.pair0 + r, u.pairs - 1);              // rows beyond the last repeat it and are not stored
      const bool live = u.pair0 + r < u.pairs;
      const int tok = p % u.len, head = u.head0 + p / u.len, pos = u.pos0 + tok;
      const size_t row = (size_t)(u.row0 + tok);
      // Query rows into swizzled shared memory, and results out of it, 16 bytes per lane along the rows: with a row per lane every access touched 32
      // lines, 4.6 us before the first scores and as much behind the last.
      auto at = [&](int rr, int c) { return reinterpret_cast<uint4*>(sq + (c >> 3) * CHUNK + rr * 128 + (((c & 7) ^ (rr & 7)) << 4)); };
      {
        const size_t own = row * a.ldq + (size_t)head * a.q_head;
#pragma unroll 4
        for (int i = half; i < DK / 8; i += 2) {
          const int idx = i * 32 + lane, rr = idx / (DK / 8), c = idx % (DK / 8);
          const size_t from = __shfl_sync(0xffffffffu, (unsigned long long)own, rr);
          *at(q4 * 32 + rr, c) = reinterpret_cast<const uint4*>(a.q + from)[c];
        }
        fence_proxy_async_smem();
        mbar_arrive(&sm->q_full);
      }
      float c2 = a.scale * 1.4426950408889634f;                 // scores in units of log 2
      if (a.temp_every > 0) c2 *= 1.0f + a.temp_coef * logf(floorf((float)(pos + 1) / (float)a.temp_every) + 1.0f);
      const float sl = BIAS ? a.slope[head] * 1.4426950408889634f : 0.0f;
      const int first = a.first(pos);
      float m = -INFINITY, l = 0.0f;                            // reference point and sum of the weights so far
      bool ok = true;
      for (int i = 0; i < t.n; ++i) {
        const int k0 = (t.lo + i) * FL_KEYS;
        ok = __all_sync(0xffffffffu, ok && fl_wait(&sm->s_full, i & 1, sm, a.err));
        if (!ok) { named_bar_sync(1, 256); continue; }      // the warps meet as often whatever fails
        tc_fence_after();
        const int stop = min(pos + 1, k0 + FL_KEYS);            // keys [first, stop) of this tile
        const bool some = __any_sync(0xffffffffu, first > k0 || stop < k0 + FL_KEYS);
        auto piece = [&](int c, uint32_t (&v)[32]) {            // the scores of keys 32 c .. of this tile
          tmem_ld16(ts + c * 32, *reinterpret_cast<uint32_t(*)[16]>(&v[0]));
          tmem_ld16(ts + c * 32 + 16, *reinterpret_cast<uint32_t(*)[16]>(&v[16]));
          tmem_ld_wait();
        };
        float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
#pragma unroll 1
        for (int c = 2 * half; c < 2 * half + 2; ++c) {
          uint32_t v[32];
          piece(c, v);
          if (some) {                                           // what a row does not see becomes minus infinity, there as well
            const int a0 = max(0, min(32, first - k0 - c * 32)), a1 = max(0, min(32, stop - k0 - c * 32));
            const uint32_t seen = a1 > a0 ? (0xffffffffu >> (32 - (a1 - a0))) << a0 : 0u;
#pragma unroll
            for (int k = 0; k < 32; ++k) v[k] = seen & (1u << k) ? v[k] : 0xff800000u;
            tmem_st16(ts + c * 32, *reinterpret_cast<uint32_t(*)[16]>(&v[0]));
            tmem_st16(ts + c * 32 + 16, *reinterpret_cast<uint32_t(*)[16]>(&v[16]));
          }
          if constexpr (BIAS) {                                 // what is compared are the scores as they enter the exponential
            const float from = sl * (float)(k0 + c * 32 - pos);
#pragma unroll
            for (int k = 0; k < 32; ++k) v[k] = __float_as_uint(fmaf(__uint_as_float(v[k]), c2, fmaf(sl, (float)k, from)));
          }
#pragma unroll
          for (int k = 0; k < 32; k += 4) {
            m0 = fmaxf(m0, __uint_as_float(v[k])); m1 = fmaxf(m1, __uint_as_float(v[k + 1]));
            m2 = fmaxf(m2, __uint_as_float(v[k + 2])); m3 = fmaxf(m3, __uint_as_float(v[k + 3]));
          }
        }
        if (some) tmem_st_wait();
        m0 = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
        sm->part[half][r] = m0;
        named_bar_sync(1, 256);
        const float top = fmaxf(m0, sm->part[half ^ 1][r]) * (BIAS ? 1.0f : c2);
        const bool moves = top > m + 8.0f || (m == -INFINITY && top > -INFINITY);
        float grow = 1.0f;
        if (moves) { grow = fl_exp2(m - top); m = top; l *= grow; }
        const float ref = m == -INFINITY ? 0.0f : m;
        float s0 = 0.0f, s1 = 0.0f;
#pragma unroll 1
        for (int c = 2 * half; c < 2 * half + 2; ++c) {         // their weights in their place: 16 columns, and 16 of the remainders
          uint32_t v[32], hi[16], rest[SPLIT ? 16 : 1];
          piece(c, v);
          const float from = BIAS ? fmaf(sl, (float)(k0 + c * 32 - pos), -ref) : -ref;
#pragma unroll
          for (int k = 0; k < 32; k += 2) {
            const float e0 = fl_exp2(fmaf(__uint_as_float(v[k]), c2, BIAS ? fmaf(sl, (float)k, from) : from));
            const float e1 = fl_exp2(fmaf(__uint_as_float(v[k + 1]), c2, BIAS ? fmaf(sl, (float)(k + 1), from) : from));
            s0 += e0; s1 += e1;
            const uint32_t h = pack_bf16x2(e0, e1);
            hi[k >> 1] = h;
            if constexpr (SPLIT) rest[k >> 1] = pack_bf16x2(e0 - __uint_as_float(h << 16), e1 - __uint_as_float(h & 0xffff0000u));
          }
          tmem_st16(ts + c * 32, hi);
          if constexpr (SPLIT) tmem_st16(ts + c * 32 + 16, rest);
        }
        l += s0 + s1;
        if (i > 0 && __any_sync(0xffffffffu, moves)) {       // the output holds the tiles before (see above)
#pragma unroll
          for (int c0 = 0; c0 < DV / 32; ++c0) {
            const int c = half * (DV / 32) + c0;
            uint32_t o[16];
            tmem_ld16(to + c * 16, o);
            tmem_ld_wait();
#pragma unroll
            for (int k = 0; k < 16; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * grow);
            tmem_st16(to + c * 16, o);
          }
        }
        tmem_st_wait();
        if (half == 0 && k0 + FL_KEYS > u.pos0 + u.len) {   // value rows behind the last key: a weight of zero does not silence what is no number
          const int s = i % ST;
          ok = __all_sync(0xffffffffu, fl_wait(&sm->v_full[s], (i / ST) & 1, sm, a.err));
          if (!ok) continue;
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
      ok = __all_sync(0xffffffffu, ok && fl_wait(&sm->o_done, 0, sm, a.err));
      tc_fence_after();
      sm->part[half][r] = l;
      named_bar_sync(1, 256);
      if (ok) {
        l += sm->part[half ^ 1][r];
        if (a.sink) l += exp2f(__bfloat162float(a.sink[head]) * 1.4426950408889634f - m);
        if (a.sink_f) l += exp2f(a.sink_f[head] * 1.4426950408889634f - m);
        float inv = 1.0f / l;
        if (a.scaled) inv *= a.out_scale;
        if (a.head_gate) inv *= 1.0f / (1.0f + expf(-a.head_gate[row * a.ld_head + head]));
        const __nv_bfloat16* gate = a.gate ? a.gate + row * a.ldg + (size_t)head * DV : nullptr;
#pragma unroll 1
        for (int c = half * (DV / 32); c < (half + 1) * (DV / 32); ++c) {      // over the queries: the last scores are made
          uint32_t o[16];
          tmem_ld16(to + c * 16, o);
          tmem_ld_wait();
          float y[16];
#pragma unroll
          for (int k = 0; k < 16; ++k) y[k] = __uint_as_float(o[k]) * inv;
          if (gate) {
#pragma unroll
            for (int k = 0; k < 16; ++k) y[k] *= 1.0f / (1.0f + expf(-__bfloat162float(gate[c * 16 + k])));
          }
#pragma unroll
          for (int h = 0; h < 2; ++h)
            *at(r, c * 2 + h) = make_uint4(pack_bf16x2(y[8 * h], y[8 * h + 1]), pack_bf16x2(y[8 * h + 2], y[8 * h + 3]), pack_bf16x2(y[8 * h + 4], y[8 * h + 5]),
                                           pack_bf16x2(y[8 * h + 6], y[8 * h + 7]));
        }
      }
      named_bar_sync(1, 256);
      if (ok) {
#pragma unroll 4
        for (int i = half; i < DV / 8; i += 2) {
          const int idx = i * 32 + lane, rr = idx / (DV / 8), c = idx % (DV / 8);
          const int orow = __shfl_sync(0xffffffffu, u.row0 + tok, rr), ohead = __shfl_sync(0xffffffffu, live ? head : -1, rr);
          if (ohead < 0) continue;
          const int f = ohead * DV + c * 8;
          const uint4 w = *at(q4 * 32 + rr, c);
          if (a.packed_rows)
            *reinterpret_cast<uint4*>(reinterpret_cast<unsigned char*>(a.out) + (size_t)(f >> 6) * a.packed_rows * 128 + sw128_offset((uint32_t)orow, (uint32_t)(f & 63))) = w;
          else *reinterpret_cast<uint4*>(a.out + (size_t)orow * a.ldo + f) = w;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tm, COLUMNS);
}

}  // namespace jf
