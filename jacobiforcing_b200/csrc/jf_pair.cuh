// jf_pair.cuh — tcgen05 matrix product of prompt-sized steps on pairs of SMs, shared by both engines (bf16 operands, fp32
// accumulation in tensor memory):  C[t, n] = sum_k X[t, k] W[n, k].
//
// A cluster of two CTAs works on one tile of 256 features x BT tokens: each holds the weight rows of its 128 features and half of the
// token rows in shared memory, and one thread of the first issues tcgen05.mma.cta_group::2, which reads both halves from both
// SMs and leaves 128 features in each SM's tensor memory.  An SM so takes in 32 KiB per 64 k for 128 x 256 products instead of
// 48 KiB; what an SM takes in was what bounded a kernel of 128 x 256 tiles on one SM with its activation rows copied by threads.
// Both operands travel by TMA: weight tiles lie in HBM in the K-major SWIZZLE_128B layout already (an unswizzled map of 128-byte
// rows), activation rows are row-major and swizzled on the way in (rows and columns beyond the operand read as zeros).  The kernel
// is persistent: one cluster per pair of SMs walks the tiles, and the epilogue of a tile runs under the products of the next
// (two accumulators).
// Measured cold, TFLOP/s, that kernel -> this one:  N 24576, T 2048, K 2048: 825 -> 1325;  N 2048, T 2048, K 10240: 736 -> 1198;
// N 37888, T 1000, K 3584: 975 -> 1441 (0.87 of the measured cuBLAS burst);  few tiles (N 1024, T 512, K 6144): 68 -> 43 us.
//
// Warp 0:     producer (one lane in each CTA, seven or nine stages; all bytes of a stage count on the first CTA's mbarrier).
// Warp 1:     owns tensor memory; in the first CTA one lane issues the products and commits to both CTAs' mbarriers.
// Warps 2-9:  epilogue (two per quarter of the lanes, one half of the columns each).
// Every wait on an mbarrier is bounded: on a timeout the kernel raises the error flag, stops waiting, lets its copies land and frees
// its tensor memory.  tcgen05.alloc has no such limit; it ends because who holds columns of the SM never waits for this block: the blocks
// of a kernel that may start under this one (see pdl_trigger) start only once every block of this grid owns its columns.
// What leaves with the accumulators is the Epilogue: a functor called by every epilogue warp with (tensor memory address of its lanes
// and columns, this lane's feature n, token of the first column, columns, tokens T, features N, lane).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "jf_ptx.cuh"

namespace jf {

// Programmatic dependent launch: a kernel may start while the one before it still runs and must not touch anything that an
// earlier kernel reads or writes before pdl_wait.  What comes before it (weights, which nothing writes; barriers, tensor memory)
// overlaps the end of the kernel before.
// A kernel that allocates tensor memory triggers behind its allocation and the barrier that follows it, never before: a block of a later
// kernel would otherwise be able to take the columns first and hold them in pdl_wait, which ends with this grid, while a block of this
// grid waits for them in tcgen05.alloc, which has no limit.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

constexpr int TC_WTILE = 128 * 64 * 2;                  // 16 KiB
constexpr uint32_t TC_SPIN_LIMIT = 1u << 22;            // try_wait probes (each blocks for a bounded time itself)
// as many stages as fit: what few tiles with a long k wait for is the latency of their loads
__host__ __device__ constexpr int tp_stages(int bt) { return bt == 256 ? 7 : 9; }
constexpr int TP_MAX_STAGES = 9;
constexpr int TP_THREADS = 320;
constexpr int TP_CLUSTERS = 74;                         // pairs of SMs

struct TpSmem {
  uint64_t full[TP_MAX_STAGES], empty[TP_MAX_STAGES], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  uint32_t failed;
};

__device__ __forceinline__ uint32_t tp_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void tp_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the address of a shared-memory object of this CTA in the first CTA of the pair
__device__ __forceinline__ uint32_t tp_in_first(const void* p) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(p)));
  return a;
}
__device__ __forceinline__ void tp_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool tp_wait(uint64_t* bar, uint32_t parity, TpSmem* sm, int* err) {
  if (sm->failed) return false;
  for (uint32_t i = 0; i < TC_SPIN_LIMIT; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  sm->failed = 1;
  atomicExch(err, 1);
  return false;
}
__device__ __forceinline__ void tp_load(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void tp_load_pairs(void* dst, const CUtensorMap* map, int group, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %2, %2, %3}], [%4];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(0), "r"(group), "r"(bar) : "memory");
}
__device__ __forceinline__ void tp_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrive on the mbarrier at this offset in both CTAs when the products issued so far have completed
__device__ __forceinline__ void tp_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}

// The columns of an epilogue warp, 32 at a time (two loads in flight): store16(sixteen accumulators, first token, how many exist).
template <typename Store>
__device__ __forceinline__ void tp_columns(uint32_t taddr, int t0, int cols, int T, Store store16) {
  for (int c0 = 0; c0 < cols; c0 += 32) {
    if (t0 + c0 >= T) break;
    __syncwarp();                                            // the loads from tensor memory are warp-wide
    uint32_t a[16], b[16];
    tmem_ld16(taddr + c0, a);
    tmem_ld16(taddr + c0 + 16, b);
    tmem_ld_wait();
    store16(a, t0 + c0, min(16, T - t0 - c0));
    if (t0 + c0 + 16 < T) store16(b, t0 + c0 + 16, min(16, T - t0 - c0 - 16));
  }
}

// Grouped mode (routed experts): the tiles of a device-made list, each up to BT consecutive rows of the expert-sorted activation
// rows that belong to one expert; the weight tiles of expert e start e * w_rows map rows further on.  Rows of the next expert
// that a tile reads along are left out by the epilogue.
struct TpGroup { const int* meta; const int* offs; const int* tile_expert; const int* tile_row0; int w_rows; };

// Layout of the operands beyond row-major activations and one weight matrix:
// x_chunk_rows > 0: the activations lie as [K / 64][x_chunk_rows][64], swizzled already (the Jacobi engine's operand layout; the map
// is the unswizzled one of its 128-byte rows); x_row0: the operand's first row (a multiple of 8).
// pairs: gate and up matrices lie one after the other in 128-row tiles, and a tile of the product takes 16 gate and 16 up rows in
// turn, so that a warp of the epilogue holds whole pairs.  The weight map is four-dimensional then (tp_map_pairs) and one copy
// brings a stage; eight copies of 16 rows each held the products back (N 37888, T 1000, K 3584: 279 us against 205).
struct PairLayout { int x_chunk_rows, x_row0, pairs; };

// Few tiles (n parts > 1): every tile's k is cut into `parts` ranges that run on pairs of their own, so that a product of few features and
// tokens still streams its weights through all SMs (N 3584, K 3584 and 18944, 24 rows: 157 us on 14 pairs, 52 us on 70).  Each
// epilogue warp leaves its partial sums in `sums`; the last of a tile's parts to arrive (one counter per tile, CTA and warp) adds all
// of them in the order of the ranges, whoever it is, and goes on to the epilogue.  The counters are zero before and after.
struct PairSplit { int parts; float* sums; int* arrived; };

// One epilogue warp's part: COLS columns of its 32 lanes, `live` of them in use.  Returns whether this warp came last; its tensor memory
// holds the whole sums then.  slot: tile, CTA and warp.
template <int COLS>
__device__ __forceinline__ bool tp_add_parts(uint32_t taddr, const PairSplit& sp, int slot, int part, int live, int lane) {
  float* own = sp.sums + ((size_t)slot * sp.parts + part) * COLS * 32 + lane;
  __syncwarp();
  for (int c = 0; c < live; c += 16) {
    uint32_t v[16];
    tmem_ld16(taddr + c, v);
    tmem_ld_wait();
#pragma unroll
    for (int k = 0; k < 16; ++k) own[(c + k) * 32] = __uint_as_float(v[k]);
  }
  __threadfence();
  __syncwarp();
  int before = 0;
  if (lane == 0) before = atomicAdd(&sp.arrived[slot], 1);
  before = __shfl_sync(0xffffffffu, before, 0);
  if (before != sp.parts - 1) return false;
  __threadfence();
  if (lane == 0) sp.arrived[slot] = 0;
  const float* all = sp.sums + (size_t)slot * sp.parts * COLS * 32 + lane;
  for (int c = 0; c < live; c += 16) {
    float a[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) a[k] = __ldcg(all + (c + k) * 32);
    for (int p = 1; p < sp.parts; ++p) {
#pragma unroll
      for (int k = 0; k < 16; ++k) a[k] += __ldcg(all + ((size_t)p * COLS + c + k) * 32);
    }
    uint32_t v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = __float_as_uint(a[k]);
    tmem_st16(taddr + c, v);
  }
  tmem_st_wait();
  return true;
}

template <class Epilogue, int BT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TP_THREADS, 1)
pair_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, int T, int N, int K, const Epilogue epilogue, int* err,
            TpGroup grp, PairLayout lay, PairSplit split) {
  extern __shared__ __align__(16) unsigned char tp_smem[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tp_smem) + 1023) & ~(uintptr_t)1023);
  constexpr int TP_STAGES = tp_stages(BT), XTILE = BT / 2 * 128, SLOT = TC_WTILE + XTILE;
  TpSmem* sm = reinterpret_cast<TpSmem*>(base + TP_STAGES * SLOT);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = (int)tp_rank();
  const int KT = (K + 63) / 64, nx = (N + 255) / 256, parts = split.parts, step = (gridDim.x >> 1) / parts;
  // this pair's range of k and first tile (parts > 1: one tile per pair)
  const int part = (int)(blockIdx.x >> 1) % parts, first = (int)(blockIdx.x >> 1) / parts, kt0 = part * KT / parts, kt1 = (part + 1) * KT / parts;
  if (threadIdx.x == 0) {
    for (int i = 0; i < TP_STAGES; ++i) { mbar_init(&sm->full[i], 1); mbar_init(&sm->empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&sm->acc_full[i], 1); mbar_init(&sm->acc_empty[i], 16); }
    sm->failed = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm->tmem_base)), "r"((uint32_t)(2 * BT)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tp_cluster_sync();
  tc_fence_after();
  pdl_trigger();                                            // both CTAs own their columns (see pdl_trigger)
  // one stage's weight tile: 128 rows, or 64 gate and 64 up rows
  auto load_w = [&](unsigned char* dst, int x, int kt, int base_row, uint32_t bar) {
    if (!lay.pairs) {
      tp_load(dst, &wmap, 0, base_row + ((2 * x + rank) * KT + kt) * 128, bar);
    } else {
      const int f0 = (2 * x + rank) * 64;
      tp_load_pairs(dst, &wmap, ((f0 >> 7) * KT + kt) * 8 + (f0 & 127) / 16, bar);
    }
  };
  // the weight tiles of the first stages travel while the kernel before this one ends (which tile is the first is known when the
  // tiles are not a list that it makes)
  int ahead = 0;
  if (warp == 0 && lane == 0 && !grp.meta) {
    const int x = first / ((T + BT - 1) / BT);
    for (; ahead < min(TP_STAGES, kt1 - kt0); ++ahead) {
      if (rank == 0) mbar_expect_tx(&sm->full[ahead], 2 * SLOT);
      load_w(base + ahead * SLOT, x, kt0 + ahead, 0, tp_in_first(&sm->full[ahead]));
    }
  }
  pdl_wait();
  const int ny = grp.meta ? grp.meta[0] : (T + BT - 1) / BT, tiles = nx * ny;
  // token tile and feature tile of a tile number: neighbours share the weight rows (grouped: the expert's activation rows)
  auto place = [&](int tile, int& x, int& y) {
    if (grp.meta) { x = tile % nx; y = tile / nx; }
    else { x = tile / ny; y = tile % ny; }
  };

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;
      bool ok = true;
      for (int tile = first; tile < tiles && ok; tile += step) {
        int x, y;
        place(tile, x, y);
        const int t0 = (grp.meta ? grp.tile_row0[y] : y * BT) + rank * (BT / 2);
        const int w0 = grp.meta ? grp.tile_expert[y] * grp.w_rows : 0;
        for (int kt = kt0; kt < kt1; ++kt, ++it) {
          const int s = it % TP_STAGES;
          ok = tp_wait(&sm->empty[s], ((it / TP_STAGES) & 1) ^ 1, sm, err);      // the products that read the slot retired
          if (!ok) break;
          const uint32_t bar = tp_in_first(&sm->full[s]);
          if (it >= ahead) {
            if (rank == 0) mbar_expect_tx(&sm->full[s], 2 * SLOT);
            load_w(base + s * SLOT, x, kt, w0, bar);
          }
          if (lay.x_chunk_rows) tp_load(base + s * SLOT + TC_WTILE, &xmap, 0, kt * lay.x_chunk_rows + lay.x_row0 + t0, bar);
          else tp_load(base + s * SLOT + TC_WTILE, &xmap, kt * 64, t0, bar);
        }
      }
      if (!ok) for (int i = 0; i < 1000; ++i) __nanosleep(1000);    // copies in flight land before the block leaves
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      const uint32_t idesc = umma_idesc_bf16(256, BT);
      int it = 0, i = 0;
      bool ok = true;
      for (int tile = first; tile < tiles && ok; tile += step, ++i) {
        const uint32_t d = sm->tmem_base + (i & 1) * BT;
        ok = tp_wait(&sm->acc_empty[i & 1], ((i >> 1) & 1) ^ 1, sm, err);        // both CTAs have read it
        tc_fence_after();
        for (int kt = kt0; kt < kt1 && ok; ++kt, ++it) {
          const int s = it % TP_STAGES;
          ok = tp_wait(&sm->full[s], (it / TP_STAGES) & 1, sm, err);
          if (!ok) break;
          tc_fence_after();
          const uint32_t sa = smem_u32(base + s * SLOT), sb = sa + TC_WTILE;
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            tp_mma(d, umma_desc_sw128(sa + kk * 32), umma_desc_sw128(sb + kk * 32), idesc, (kt > kt0 || kk > 0) ? 1u : 0u);
          tp_commit(&sm->empty[s]);
        }
        if (ok) tp_commit(&sm->acc_full[i & 1]);
      }
    }
    __syncwarp();
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2;                 // quarter of the lanes that this warp may read, half of the columns
    int i = 0;
    for (int tile = first; tile < tiles; tile += step, ++i) {
      int x, y;
      place(tile, x, y);
      if (!tp_wait(&sm->acc_full[i & 1], (i >> 1) & 1, sm, err)) break;
      tc_fence_after();
      const int t0 = (grp.meta ? grp.tile_row0[y] : y * BT) + half * (BT / 2);
      const int rows = grp.meta ? grp.offs[grp.tile_expert[y] + 1] : T;
      const uint32_t taddr = sm->tmem_base + (i & 1) * BT + half * (BT / 2) + ((uint32_t)(q * 32) << 16);
      bool mine = true;
      if (parts > 1) mine = tp_add_parts<BT / 2>(taddr, split, tile * 16 + rank * 8 + warp - 2, part, min(BT / 2, rows - t0), lane);
      if (mine) epilogue(taddr, x * 256 + rank * 128 + q * 32 + lane, t0, BT / 2, rows, N, lane);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) tp_arrive_cluster(tp_in_first(&sm->acc_empty[i & 1]));
    }
  }
  tc_fence_before();
  __syncthreads();
  tp_cluster_sync();                                                // nothing of the pair still reads or signals this CTA
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(sm->tmem_base), "r"((uint32_t)(2 * BT)) : "memory");
}

constexpr size_t tp_smem_bytes(int bt) { return (size_t)tp_stages(bt) * (TC_WTILE + bt / 2 * 128) + sizeof(TpSmem) + 1024; }

// ---- host: tensor maps ------------------------------------------------------------------------------------------------------------
typedef CUresult (*TpEncode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                             const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline TpEncode tp_encode() {
  static const TpEncode f = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult r;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &r) != cudaSuccess || r != cudaDriverEntryPointSuccess) p = nullptr;
    return (TpEncode)p;
  }();
  return f;
}
// rows x cols bf16 elements, `ld` elements from row to row, in boxes of box_rows x 64
inline bool tp_map(CUtensorMap* m, const void* p, uint64_t rows, uint64_t cols, uint64_t ld, int box_rows, bool swizzle) {
  const TpEncode f = tp_encode();
  if (!f) return false;
  const cuuint64_t dims[2] = {cols, rows}, strides[1] = {ld * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)box_rows}, one[2] = {1, 1};
  return f(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(p), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
           swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Gate and up tiles of 128 rows x 64 (both matrices [n_tiles][KT], the up matrix behind the gate matrix): boxes of four times 16 gate rows
// and the 16 up rows that go with them.
inline bool tp_map_pairs(CUtensorMap* m, const void* p, uint64_t n_tiles, uint64_t KT) {
  const TpEncode f = tp_encode();
  if (!f) return false;
  const cuuint64_t dims[4] = {64, 16, 2, n_tiles * KT * 8}, strides[3] = {128, n_tiles * KT * 16384, 2048};
  const cuuint32_t box[4] = {64, 16, 2, 4}, one[4] = {1, 1, 1, 1};
  return f(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(p), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Token rows per tile: 128 when those tiles fit one wave of the pairs (the wave is over sooner: N 1024, T 2048, K 6144: 45 us against
// 48 with 256 rows), 256 otherwise (N 2048, T 2048, K 2048: 27 us against 35).
inline int tp_tile_rows(int N, int T) { return (long long)((N + 255) / 256) * ((T + 127) / 128) <= TP_CLUSTERS ? 128 : 256; }

// Parts of k per tile: as many as pairs are idle otherwise, at least eight steps of 64 k each.
inline int tp_parts(int tiles, int K) { return std::max(1, std::min(std::min(TP_CLUSTERS / std::max(1, tiles), (K + 63) / 64 / 8), 8)); }
// Floats and counters that a product with parts may need (parts > 1: at most TP_CLUSTERS tiles and parts together).
constexpr size_t TP_SUMS = (size_t)TP_CLUSTERS * 16 * 32 * 128, TP_ARRIVED = (size_t)TP_CLUSTERS * 16;

}  // namespace jf
