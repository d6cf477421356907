// hy_gla.cuh — gated linear attention with one decay per key channel, retention (one fixed decay per head, rotated queries and
// keys), the gated linear recurrence whose forget gate also sets what is written, the state-space recurrence with one decay per token and
// head, and the row kernels between the sublayers of blocks with plain RMS weights (libjf_hybrid.so).
//
// Per head, S [dim, vdim]:  S <- diag(a) S + k v^T ;  o = S^T q dim^(-1/2)   (the read-out sees the current token's write)
//   out = o / rms(o) * norm_w * silu(g)        (norm over the head's vdim, one weight shared by the heads)
// The decay a = sigmoid(z)^(1 / tau) leaves the decay projection's epilogue as fp32 (gemm_store).  Retention is the same
// recurrence with one number per head for a and with q, k rotated at their position (in fp32, between the projections and the
// recurrence) and no weight in the norm.
//
// The recurrence has no feedback from the read-out and its value columns are independent, so a head is cut into blocks of
// CPB = VC 128 / PARTS columns that run side by side on different SMs, and PARTS lanes share VC columns, each holding DR / PARTS
// of its key rows in registers; what does not depend on the state is made beforehand (linear_rows_kernel).  The norm needs
// whole heads: it follows in a kernel of its own (gla_out_kernel).
#pragma once
#include "hy_kernels.cuh"
#include "hy_delta.cuh"
#include "jf_ptx.cuh"

namespace hy {

// qk [T][H][q dim | k dim] fp32 from linear_rows_kernel, v [T, ldv] (H heads of vdim).  Decays: decay [T, ldd] fp32 (H heads of dim),
// or with GLA_HEAD one number per head, head_decay [H].  With GLA_FORGET the rows hold [q | f] (forget_rows_kernel) and the
// update is S <- f S + (1 - f) v^T, written as v + f (S - v).  o [T, ldo] fp32 (H heads of vdim).  state [slot][H][dim][vdim] fp32.
// grid (H * blocks_per_head, entries), 128 threads.  Lane layout, vec and vvec as in delta_head_kernel.
// With GLA_TOKEN (state-space recurrence with one decay per head) the rows [q | k] = [C | B] are shared by the H / G heads of a
// group, a head's step size dt = softplus(dt_raw + bias) and decay exp(-exp(A_log) dt) are made per token from dt_raw [T, lddt]
// (column h), the value is dt x and the read-out gets D_h x added.
// GLA_TOKEN, 2048 tokens of 32 heads of 64 channels x 128 states: eight lanes with sixteen consecutive states each (staged rows read
// with four-way bank conflicts, one exchange per token) took 766 us, this layout 284 us, 237 with two columns per lane.
// GLA_FORGET, 2048 tokens of 8 heads of 128 x 128: one block per head with a column per thread took 1927 us, this layout 202 us, 187 with the next
// token's rows read ahead.
enum GlaMode : int { GLA_CHANNEL = 0, GLA_HEAD = 1, GLA_FORGET = 2, GLA_TOKEN = 3 };
struct GlaToken { int G; const void* dt_raw; int lddt; const float* dt_bias; const float* A_log; const float* D; };
template <typename AT, int DR, int PARTS, int VC, int MODE>
__global__ void __launch_bounds__(128) gla_kernel(Batch b, const float* __restrict__ qk, const AT* __restrict__ v, int ldv,
                                                  const float* __restrict__ decay, int ldd, const float* __restrict__ head_decay, int H,
                                                  int dim, int vdim, int blocks_per_head, int vec, int vvec, float* __restrict__ state,
                                                  float* __restrict__ o, int ldo, GlaToken tk) {
  pdl_trigger();
  constexpr int TB = lin_tb(DR), RP = DR / PARTS, CW = 32 / PARTS, CPB = lin_cpb(PARTS, VC), VW = CPB < 8 ? 8 : CPB;
  constexpr bool HEAD = MODE == GLA_HEAD;
  constexpr int RW = MODE == GLA_CHANNEL ? 3 * DR : 2 * DR;    // floats of a staged row: q | k (| decays)
  extern __shared__ __align__(16) unsigned char hy_smem[];
  float* sqk = reinterpret_cast<float*>(hy_smem);              // [2][TB][RW]
  AT* sv = reinterpret_cast<AT*>(sqk + 2 * TB * RW);           // [2][TB][VW]
  __shared__ float2 sdt[MODE == GLA_TOKEN ? 2 * TB : 1];       // [2][TB] decay, step size
  const int h = blockIdx.x / blocks_per_head, c0 = (blockIdx.x % blocks_per_head) * CPB, e = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cl = warp * CW + lane % CW, part = lane / CW, col = c0 + cl * VC;
  const int ncol = min(CPB, vdim - c0);
  const int start = b.ent_start[e], cnt = b.ent_start[e + 1] - start, pos0 = b.ent_pos0[e];
  float* st = state + ((size_t)b.ent_slot[e] * H + h) * dim * vdim;
  float2 S[VC][RP / 2];
#pragma unroll
  for (int i = 0; i < RP; i += 2) {
    const int r = 4 * (part + PARTS * (i / 4)) + (i & 3);
#pragma unroll
    for (int c = 0; c < VC; ++c)
      S[c][i / 2] = make_float2((col + c < vdim && r < dim && pos0 > 0) ? st[(size_t)r * vdim + col + c] : 0.0f,
                                (col + c < vdim && r + 1 < dim && pos0 > 0) ? st[(size_t)(r + 1) * vdim + col + c] : 0.0f);
  }
  const float hd = HEAD ? head_decay[h] : 0.0f;
  const int rows_per_token = MODE == GLA_TOKEN ? tk.G : H, row_of = MODE == GLA_TOKEN ? h / (H / tk.G) : h;
  const float rate = MODE == GLA_TOKEN ? expf(tk.A_log[h]) : 0.0f, dt_bias = MODE == GLA_TOKEN ? tk.dt_bias[h] : 0.0f;
  const float skip = MODE == GLA_TOKEN ? tk.D[h] : 0.0f;
  pdl_wait();
  float raw = 0.0f;                                            // raw step size of token tid of the batch in flight
  if (dim < DR)                                                // rows beyond the head's key size stay zero
    for (int i = tid; i < 2 * TB * RW; i += 128) if (i % DR >= dim) sqk[i] = 0.0f;
  auto fetch = [&](int j0, int buf) {
    const int nb = min(TB, cnt - j0);
    const size_t t0 = (size_t)(start + j0);
    float* d = sqk + (size_t)buf * TB * RW;
    const float* src = qk + (t0 * rows_per_token + row_of) * 2 * dim;
    const size_t ld = (size_t)rows_per_token * 2 * dim;
    if (MODE == GLA_TOKEN && tid < nb) raw = to_f(((const AT*)tk.dt_raw)[(t0 + tid) * tk.lddt + h]);
    copy_rows(d, RW, src, ld, nb, dim, vec);
    copy_rows(d + DR, RW, src + dim, ld, nb, dim, vec);
    if (MODE == GLA_CHANNEL) copy_rows(d + 2 * DR, RW, decay + t0 * ldd + h * dim, ldd, nb, dim, vec);
    copy_values(sv + (size_t)buf * TB * VW, VW, v + t0 * ldv + h * vdim + c0, ldv, nb, ncol, vvec);
    jf::cp_async_commit();
  };
  fetch(0, 0);
  constexpr int TG = TB < 8 ? TB : 8;                          // tokens whose read-outs are reduced together
  int buf = 0;
  for (int j0 = 0; j0 < cnt; j0 += TB, buf ^= 1) {
    const int nb = min(TB, cnt - j0);
    if (MODE == GLA_TOKEN && tid < nb) {
      const float dt = softplus_f(raw + dt_bias);
      sdt[buf * TB + tid] = make_float2(expf(-rate * dt), dt);
    }
    jf::cp_async_wait_all();
    __syncthreads();                                           // this batch has landed; the batch before it is finished
    if (j0 + TB < cnt) fetch(j0 + TB, buf ^ 1);
    const float* rb = sqk + (size_t)buf * TB * RW + 4 * part;
    const AT* vb = sv + (size_t)buf * TB * VW + cl * VC;                     // columns beyond the head's last are never stored
    float* po = o + (size_t)(start + j0) * ldo + h * vdim + col;
    auto leave = [&](int tt, int c, float p) {
      if constexpr (MODE == GLA_TOKEN) p = fmaf(skip, to_f(vb[tt * VW + c]), p);
      if (col + c < vdim) po[(size_t)tt * ldo + c] = p;
    };
    // one token's rows in registers; where they are few, the next token's are read before this one's products, which covers their latency
    struct Row { float4 q[RP / 4], k[RP / 4], a[MODE == GLA_CHANNEL ? RP / 4 : 1]; VecN<AT, VC> v; float2 sd; };
    auto read = [&](Row& w, int tt) {
#pragma unroll
      for (int i = 0; i < RP / 4; ++i) {
        w.q[i] = *reinterpret_cast<const float4*>(rb + tt * RW + 4 * PARTS * i);
        w.k[i] = *reinterpret_cast<const float4*>(rb + tt * RW + DR + 4 * PARTS * i);
        if constexpr (MODE == GLA_CHANNEL) w.a[i] = *reinterpret_cast<const float4*>(rb + tt * RW + 2 * DR + 4 * PARTS * i);
      }
      w.v = *reinterpret_cast<const VecN<AT, VC>*>(vb + tt * VW);
      if constexpr (MODE == GLA_TOKEN) w.sd = sdt[buf * TB + tt];
    };
    // one token's update of this lane's key rows and columns; leaves its parts of the read-outs
    auto update = [&](const Row& w, float (&out)[VC]) {
      float2 p[VC], vv[VC];
#pragma unroll
      for (int c = 0; c < VC; ++c) {
        float x = to_f(w.v.v[c]);
        if constexpr (MODE == GLA_TOKEN) x *= w.sd.y;
        vv[c] = make_float2(x, x);
        p[c] = make_float2(0.0f, 0.0f);
      }
      const float td = MODE == GLA_TOKEN ? w.sd.x : hd;
#pragma unroll
      for (int i = 0; i < RP / 4; ++i) {
        const float4 q = w.q[i], k = w.k[i], a = MODE == GLA_CHANNEL ? w.a[MODE == GLA_CHANNEL ? i : 0] : make_float4(td, td, td, td);
#pragma unroll
        for (int c = 0; c < VC; ++c) {
          float2 &R0 = S[c][2 * i], &R1 = S[c][2 * i + 1];
          if constexpr (MODE == GLA_FORGET) {
            const float2 less = make_float2(-vv[c].x, -vv[c].y);
            R0 = fma2(make_float2(k.x, k.y), add2(R0, less), vv[c]);
            R1 = fma2(make_float2(k.z, k.w), add2(R1, less), vv[c]);
          } else {
            R0 = fma2(make_float2(a.x, a.y), R0, mul2(make_float2(k.x, k.y), vv[c]));
            R1 = fma2(make_float2(a.z, a.w), R1, mul2(make_float2(k.z, k.w), vv[c]));
          }
          p[c] = fma2(R0, make_float2(q.x, q.y), p[c]);
          p[c] = fma2(R1, make_float2(q.z, q.w), p[c]);
        }
      }
#pragma unroll
      for (int c = 0; c < VC; ++c) out[c] = p[c].x + p[c].y;
    };
    constexpr bool FLY = RP <= 8;
    static_assert(!FLY || TG % 2 == 0, "a group of tokens leaves the next row where the next group begins");
    Row w[FLY ? 2 : 1];
    if (FLY) read(w[0], 0);
    int tt = 0;
    for (; tt + TG <= nb; tt += TG) {
      // TG tokens without a shuffle between them, then one exchange in which every step halves the tokens a lane keeps
      float p[TG][VC];
#pragma unroll
      for (int u = 0; u < TG; ++u) {
        if constexpr (FLY) read(w[(u + 1) & 1], min(tt + u + 1, nb - 1));
        else read(w[0], tt + u);
        update(w[FLY ? u & 1 : 0], p[u]);
      }
      int n = TG, base = 0;
#pragma unroll
      for (int s = 16; s >= CW; s >>= 1) {
        const bool hi = (lane & s) != 0;
        if (n > 1) {
          n >>= 1;
#pragma unroll
          for (int u = 0; u < TG / 2; ++u) {
            if (u >= n) break;
#pragma unroll
            for (int c = 0; c < VC; ++c) {
              const float other = __shfl_xor_sync(0xffffffffu, hi ? p[u][c] : p[u + n][c], s);
              p[u][c] = (hi ? p[u + n][c] : p[u][c]) + other;
            }
          }
          base += hi ? n : 0;
        } else {
#pragma unroll
          for (int c = 0; c < VC; ++c) p[0][c] += __shfl_xor_sync(0xffffffffu, p[0][c], s);
        }
      }
      constexpr int LEFT = TG > PARTS ? TG / PARTS : 1, SAME = PARTS > TG ? PARTS / TG : 1;     // tokens per lane, lanes per token
      if ((part & (SAME - 1)) == 0) {
#pragma unroll
        for (int u = 0; u < LEFT; ++u)
#pragma unroll
          for (int c = 0; c < VC; ++c) leave(tt + base + u, c, p[u][c]);
      }
    }
    for (; tt < nb; ++tt) {
      float p[VC];
      read(w[0], tt);
      update(w[0], p);
#pragma unroll
      for (int c = 0; c < VC; ++c) {
#pragma unroll
        for (int s = CW; s < 32; s <<= 1) p[c] += __shfl_xor_sync(0xffffffffu, p[c], s);
        if (part == 0) leave(tt, c, p[c]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < RP; i += 2) {
    const int r = 4 * (part + PARTS * (i / 4)) + (i & 3);
#pragma unroll
    for (int c = 0; c < VC; ++c) {
      if (r < dim && col + c < vdim) st[(size_t)r * vdim + col + c] = S[c][i / 2].x;
      if (r + 1 < dim && col + c < vdim) st[(size_t)(r + 1) * vdim + col + c] = S[c][i / 2].y;
    }
  }
}

// Operand rows of the recurrence with a forget gate: [T][H][silu(q) | f], f = lower + (1 - lower) sigmoid(f_raw + f_bias).
template <typename AT, int V>
__global__ void __launch_bounds__(1024) forget_rows_kernel(const AT* __restrict__ in, int ld, int col_q, int col_f,
                                                           const float* __restrict__ f_bias, const float* __restrict__ lower, int H, int dim,
                                                           float* __restrict__ qf) {
  pdl_begin();
  const AT* row = in + (size_t)blockIdx.x * ld;
  float* out = qf + (size_t)blockIdx.x * H * 2 * dim;
  for (int i = threadIdx.x * V; i < H * dim; i += blockDim.x * V) {
    const size_t at = (size_t)(i / dim) * 2 * dim + i % dim;
    float q[V], f[V], lo[V], bias[V];
    load_f(q, row + col_q + i); load_f(f, row + col_f + i); load_f(lo, lower + i); load_f(bias, f_bias + i);
#pragma unroll
    for (int j = 0; j < V; ++j) { q[j] = silu_f(q[j]); f[j] = fmaf(1.0f - lo[j], sigmoid_f(f[j] + bias[j]), lo[j]); }
    store_f(out + at, q);
    store_f(out + at + dim, f);
  }
}

// Norm per head, weight (NULL: none), output gate: out[t, h, :] = o / rms(o) * w * gate * out_scale, gate = silu(g), sigmoid(g) or one.
// One warp per (token, head).
enum OutGate : int { GATE_SILU = 0, GATE_SIGMOID = 1, GATE_NONE = 2 };
template <typename AT, typename GT, int GATE, int V>
__global__ void __launch_bounds__(128) gla_out_kernel(int T, int H, int vdim, const float* __restrict__ o, int ldi,
                                                      const GT* __restrict__ g, int ldg, const float* __restrict__ w, float eps,
                                                      float out_scale, AT* __restrict__ out, int ldo) {
  pdl_begin();
  const int unit = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (unit >= T * H) return;
  const size_t t = unit / H, c0 = (size_t)(unit % H) * vdim;
  const float* orow = o + t * ldi + c0;
  float ss = 0.0f;
  for (int k = lane * V; k < vdim; k += 32 * V) {
    float v[V];
    load_f(v, orow + k);
#pragma unroll
    for (int i = 0; i < V; ++i) ss = fmaf(v[i], v[i], ss);
  }
  const float inv = out_scale / sqrtf(warp_sum(ss) / (float)vdim + eps);
  for (int k = lane * V; k < vdim; k += 32 * V) {
    float v[V], x[V];
    load_f(v, orow + k);
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] *= inv;
    if (w) {
      load_f(x, w + k);
#pragma unroll
      for (int i = 0; i < V; ++i) v[i] *= x[i];
    }
    if constexpr (GATE != GATE_NONE) {
      load_f(x, g + t * ldg + c0 + k);
#pragma unroll
      for (int i = 0; i < V; ++i) v[i] *= GATE == GATE_SILU ? silu_f(x[i]) : sigmoid_f(x[i]);
    }
    store_f(out + t * ldo + c0 + k, v);
  }
}

// ---- one token's row between two sublayers ----------------------------------------------------------------------------------
// x += a sublayer's result: its rows (y), or the mixture of a routed feed-forward (rows), or nothing (both NULL); through an
// RMS norm of its own first when post_w is given.  Then what the next sublayer reads: the RMS norm of the row (norm_w), or
// the row itself (cast_out: the stream's half of the loop projection's operand), in the activation type.
// A choice >= n_experts stands for the sublayer's input: h [T, width] in the activation type, the buffer the norm is then
// written to (a thread reads a channel before it writes it).
struct RowClose {
  const float* rows; int ldr; const int* pair_row; const int* ids; const float* wts; int top, n_experts;
  const void* norm_w; float eps;
  void* cast_out; int ld_cast;
  const float* y; int ldy; const void* post_w;
};

// V channels per thread at a time (V = 4: width and all leading dimensions are multiples of 4).
constexpr int HY_CLOSE_TOP = 64;                               // choices whose rows and weights are staged in shared memory
template <typename AT, typename WT, int V>
__global__ void __launch_bounds__(256) row_close_kernel(RowClose c, int width, float* __restrict__ x, AT* h) {
  pdl_begin();
  typedef VecN<float, V> F;
  extern __shared__ __align__(16) unsigned char hy_smem[];
  float* xs = reinterpret_cast<float*>(hy_smem);               // [width]
  __shared__ float red[33];
  __shared__ int srow[HY_CLOSE_TOP];
  __shared__ float swt[HY_CLOSE_TOP];
  const int t = blockIdx.x;
  const int first = threadIdx.x * V, step = blockDim.x * V;
  const bool adds = c.rows || c.y;
  if (c.rows) {                                                // row of every staged choice, -1: an identity choice
    for (int k = threadIdx.x; k < min(c.top, HY_CLOSE_TOP); k += blockDim.x) {
      const int i = t * c.top + k;
      srow[k] = c.ids[i] >= c.n_experts ? -1 : c.pair_row ? c.pair_row[i] : i;
      swt[k] = c.wts[i];
    }
    __syncthreads();
  }
  float ss = 0.0f;
  auto result = [&](int ch) {
    if (c.y) return *reinterpret_cast<const F*>(c.y + (size_t)t * c.ldy + ch);
    F y{}, own{};
    {
      const VecN<AT, V> hv = *reinterpret_cast<const VecN<AT, V>*>(h + (size_t)t * width + ch);
#pragma unroll
      for (int j = 0; j < V; ++j) own.v[j] = to_f(hv.v[j]);
    }
#pragma unroll 4
    for (int k = 0; k < c.top; ++k) {
      int row; float w;
      if (k < HY_CLOSE_TOP) { row = srow[k]; w = swt[k]; }
      else {
        const int i = t * c.top + k;
        row = c.ids[i] >= c.n_experts ? -1 : c.pair_row ? c.pair_row[i] : i;
        w = c.wts[i];
      }
      const F r = row < 0 ? own : *reinterpret_cast<const F*>(c.rows + (size_t)row * c.ldr + ch);
#pragma unroll
      for (int j = 0; j < V; ++j) y.v[j] = fmaf(w, r.v[j], y.v[j]);
    }
    return y;
  };
  float pinv = 1.0f;
  if (c.post_w) {
    for (int ch = first; ch < width; ch += step) {
      const F y = result(ch);
      *reinterpret_cast<F*>(xs + ch) = y;
#pragma unroll
      for (int j = 0; j < V; ++j) ss = fmaf(y.v[j], y.v[j], ss);
    }
    pinv = 1.0f / sqrtf(block_sum(ss, red) / (float)width + c.eps);
    ss = 0.0f;
  }
  for (int ch = first; ch < width; ch += step) {
    F v = *reinterpret_cast<const F*>(x + (size_t)t * width + ch);
    if (adds) {
      if (c.post_w) {
        const F y = *reinterpret_cast<const F*>(xs + ch);
        const VecN<WT, V> w = *reinterpret_cast<const VecN<WT, V>*>((const WT*)c.post_w + ch);
#pragma unroll
        for (int j = 0; j < V; ++j) v.v[j] += y.v[j] * pinv * to_f(w.v[j]);
      } else {
        const F y = result(ch);
#pragma unroll
        for (int j = 0; j < V; ++j) v.v[j] += y.v[j];
      }
      *reinterpret_cast<F*>(x + (size_t)t * width + ch) = v;
    }
    *reinterpret_cast<F*>(xs + ch) = v;
#pragma unroll
    for (int j = 0; j < V; ++j) ss = fmaf(v.v[j], v.v[j], ss);
  }
  auto out = [&](AT* row, int ch, float f, const WT* w) {
    const F v = *reinterpret_cast<const F*>(xs + ch);
    VecN<AT, V> o;
#pragma unroll
    for (int j = 0; j < V; ++j) o.v[j] = from_f<AT>(w ? v.v[j] * f * to_f(w[ch + j]) : v.v[j]);
    *reinterpret_cast<VecN<AT, V>*>(row + ch) = o;
  };
  if (c.cast_out)
    for (int ch = first; ch < width; ch += step) out((AT*)c.cast_out + (size_t)t * c.ld_cast, ch, 1.0f, nullptr);
  if (!c.norm_w) return;
  const float inv = 1.0f / sqrtf(block_sum(ss, red) / (float)width + c.eps);
  for (int ch = first; ch < width; ch += step) out(h + (size_t)t * width, ch, inv, (const WT*)c.norm_w);
}

// The embedding output x0 into the second half of the loop projection's operand [T, 2 width].
template <typename AT>
__global__ void loop_origin_kernel(const float* __restrict__ x, int width, AT* __restrict__ out) {
  pdl_begin();
  const int t = blockIdx.x;
  for (int c = threadIdx.x; c < width; c += blockDim.x) out[(size_t)t * 2 * width + width + c] = from_f<AT>(x[(size_t)t * width + c]);
}

}  // namespace hy
