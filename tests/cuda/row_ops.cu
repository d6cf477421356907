// row_ops.cu — single kernels of libjf_hybrid.so over the caller's device buffers, launched as the engine launches them (tests/row_ops.py): products of few
// rows, of fp32 rows in three parts and on the fp32 units, the parts themselves, and the selective scan's exponential.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "jf_wide.cuh"
#include "hy_gemm.cuh"
#include "hy_few.cuh"

using namespace hy;

namespace {
GemmOut to_rows(float* out, int N) { return GemmOut{out, N, 1 << 30, nullptr, 0, 0, nullptr, 0, 1.0f}; }
template <typename F>
bool room(F* kernel, size_t smem) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess; }
int done() { return cudaGetLastError() == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess ? 0 : -1; }

__global__ void exp_rates_kernel(const float* dt, const float* a, float* out, int n) {
  for (int i = 2 * (blockIdx.x * blockDim.x + threadIdx.x); i < n; i += 2 * gridDim.x * blockDim.x) {      // a pair of states shares its step; n is even
    const RatePair r(a[i], a[i + 1]);
    const float2 e = exp_rates(finite_step(dt[i]), r);
    out[i] = e.x; out[i + 1] = e.y;
  }
}
__global__ void sigmoid_kernel(const float* z, float* out, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = sigmoid_f(z[i]);
}
// bf16(g / (1 + exp(-g))) * u of eight rows at a time, by swiglu_rows or with IEEE division; n is a multiple of 8
__global__ void swiglu_kernel(const float* gate, const float* up, float* out, int n, bool divide) {
  for (int i = 8 * (blockIdx.x * blockDim.x + threadIdx.x); i < n; i += 8 * gridDim.x * blockDim.x) {
    float g[8], u[8];
    for (int j = 0; j < 8; ++j) { g[j] = gate[i + j]; u[j] = up[i + j]; }
    if (divide) for (int j = 0; j < 8; ++j) u[j] *= jf::bf16_round(g[j] / (1.f + __expf(-g[j])));
    else jf::swiglu_rows(g, u);
    for (int j = 0; j < 8; ++j) out[i + j] = u[j];
  }
}
}  // namespace

extern "C" {
int ops_sigmoid(const float* z, float* out, int n) {
  sigmoid_kernel<<<148, 256>>>(z, out, n);
  return done();
}
int ops_swiglu(const float* gate, const float* up, float* out, int n, int divide) {
  swiglu_kernel<<<148, 128>>>(gate, up, out, n, divide != 0);
  return done();
}
int ops_exp_rates(const float* dt, const float* a, float* out, int n) {
  exp_rates_kernel<<<148, 128>>>(dt, a, out, n);
  return done();
}
// 1: these operands do not run there
int ops_few(const bf16* A, int lda, const bf16* W, int T, int N, int K, float* out, int wait) {
  if (!few_takes(A, lda, W, K, T, K)) return 1;
  const int tiles = (N + 15) / 16, ksplit = few_ksplit(tiles, K), per = 8 / ksplit;
  if (few_wide(tiles, K)) {
    if (!room(gemm_few_kernel<float, 16>, few_smem(K))) return -1;
    gemm_few_kernel<float, 16><<<tiles, 512, few_smem(K)>>>(A, lda, W, K, T, N, K, 16, to_rows(out, N));
  } else {
    if (!room(gemm_few_kernel<float, 8>, few_smem(K))) return -1;
    gemm_few_kernel<float, 8><<<std::min((tiles + per - 1) / per, 148 * 2), 256, few_smem(K)>>>(A, lda, W, K, T, N, K, ksplit, to_rows(out, N));
  }
  return wait ? done() : 0;
}
// the kernel beside it, with a column per warp
int ops_rows(const bf16* A, int lda, const bf16* W, int T, int N, int K, float* out, int wait) {
  const size_t row_bytes = (size_t)(K + 7) / 8 * 16;
  if (T > 8 || row_bytes * 8 > 200 * 1024) return 1;
  int ksplit = 1;
  while (ksplit < 8 && (long long)N * ksplit < 148LL * 32 && K / (ksplit * 2) >= 512) ksplit *= 2;
  const int cpb = 8 / ksplit, blocks = std::min((N + cpb - 1) / cpb, 148 * (T > 4 ? 4 : 16));
  auto go = [&](auto kern, int rows) {
    if (!room(kern, rows * row_bytes)) return;
    kern<<<dim3(blocks, (T + rows - 1) / rows), 256, rows * row_bytes>>>(A, lda, W, K, T, N, K, ksplit, to_rows(out, N));
  };
  if (T == 1) go(gemm_rows_kernel<bf16, bf16, float, 1>, 1);
  else if (T == 2) go(gemm_rows_kernel<bf16, bf16, float, 2>, 2);
  else if (T <= 4) go(gemm_rows_kernel<bf16, bf16, float, 4>, 4);
  else go(gemm_rows_kernel<bf16, bf16, float, 8>, 8);
  return wait ? done() : 0;
}
int ops_split_rows(const float* a, int lda, int T, int K, bf16* o) {
  const int KP = split_cols(K);
  split_rows_kernel<<<std::min((T * (KP / 2) + 127) / 128, 148 * 16), 128>>>(a, lda, T, K, KP, o);
  return done();
}
// Weights [N, K] on the host to the three-part product's tiles on the host; tiles NULL: how many elements.
long long ops_split_tiles(const float* w, int N, int K, uint16_t* tiles) {
  const int KP = split_cols(K);
  const long long n = (long long)((N + 127) / 128) * (3 * KP / 64) * 128 * 64;
  if (!tiles) return n;
  std::vector<float> three((size_t)N * 3 * KP, 0.0f);
  for (int r = 0; r < N; ++r)
    for (int p = 0; p < 3; ++p) std::copy_n(w + (size_t)r * K, K, &three[((size_t)r * 3 + p) * KP]);
  std::vector<uint16_t> t;
  pack_tiles(three.data(), N, 3 * KP, t);
  std::copy(t.begin(), t.end(), tiles);
  return (long long)t.size() == n ? n : -1;
}
// parts [T][3][KP] as ops_split_rows leaves them; err: one int, set to zero by the caller
int ops_split_product(const bf16* parts, int T, int K, const uint16_t* tiles, int N, float* out, int* err) {
  typedef HyEpilogue<float> Epi;
  const int KP = 3 * split_cols(K), nx = (N + 255) / 256, KT = KP / 64, NT = (N + 127) / 128, bt = jf::tp_tile_rows(N, T);
  CUtensorMap xm, wm;
  if (!jf::tp_map(&xm, parts, (uint64_t)T, (uint64_t)KP, (uint64_t)KP, bt / 2, true) || !jf::tp_map(&wm, tiles, (uint64_t)NT * KT * 128, 64, 64, 128, false)) return -1;
  const int n_tiles = nx * ((T + bt - 1) / bt), split = jf::tp_parts(std::min(n_tiles, jf::TP_CLUSTERS + 1), KP);
  static float* sums = nullptr; static int* arrived = nullptr;
  if (!sums && (cudaMalloc((void**)&sums, jf::TP_SUMS * 4) != cudaSuccess || cudaMalloc((void**)&arrived, jf::TP_ARRIVED * 4) != cudaSuccess ||
                cudaMemset(arrived, 0, jf::TP_ARRIVED * 4) != cudaSuccess)) return -1;
  auto kern = bt == 128 ? jf::pair_kernel<Epi, 128> : jf::pair_kernel<Epi, 256>;
  if (!room(kern, jf::tp_smem_bytes(bt))) return -1;
  kern<<<2 * std::min(n_tiles * split, jf::TP_CLUSTERS), jf::TP_THREADS, jf::tp_smem_bytes(bt)>>>(xm, wm, T, N, KP, Epi{to_rows(out, N)}, err, jf::TpGroup{},
                                                                                                   jf::PairLayout{0, 0, 0}, jf::PairSplit{split, sums, arrived});
  return done();
}
int ops_fp32_product(const float* a, int lda, const bf16* W, int T, int N, int K, float* out) {
  if ((long long)((N + 63) / 64) * ((T + 63) / 64) >= 148)
    gemm_simt_kernel<float, bf16, float, 64><<<dim3((N + 63) / 64, (T + 63) / 64), 256>>>(a, lda, W, K, T, N, K, to_rows(out, N));
  else
    gemm_simt_kernel<float, bf16, float, 32><<<dim3((N + 31) / 32, (T + 31) / 32), 256>>>(a, lda, W, K, T, N, K, to_rows(out, N));
  return done();
}
}
