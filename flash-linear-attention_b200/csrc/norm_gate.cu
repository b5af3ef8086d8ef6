// Gated RMS norm over the head dimension, forward and backward: the step behind the mixer in fla.layers.GatedDeltaNet
// (fla/layers/gated_deltanet.py:355-357).  Replaces layer_norm_gated_fwd_kernel / layer_norm_gated_bwd_kernel of
// fla/modules/fused_norm_gate.py (36-124, 206-339) in their RMS form without residual:
//     rstd = 1 / sqrt(mean(x^2) + eps);   y = (x rstd weight + bias) act(g),   act(g) = g sigmoid(g) | sigmoid(g)
// Rows are (token, head) vectors of D = 64 .. 512 elements.  Pure HBM streaming: D / 8 lanes own a row, eight consecutive
// elements (16 bytes of bf16) each, so a warp covers 32 / (D / 8) rows per round with full-width accesses.  What counts is the
// loads in flight: one wave of CTAs walks the rows, the next rows are loaded (and kept as loaded, half the registers of
// fp32) before the current ones are worked on, two elements per instruction (f32x2).  262144 rows of 128 in bf16: forward
// 34.5 us (54.8 with each round's loads waited for at once; 31 at copy rate), backward 51.6 (78; 51).  The backward pass holds
// its dweight / dbias sums in registers and leaves ONE partial row per CTA, which a second kernel adds in a fixed order (no
// atomics).
#include "gdn_common.cuh"
#include "rowio.cuh"

namespace gdn {
namespace {

constexpr int NT = 256;   // 8 warps
// CTAs per SM, and row groups a warp works on while as many are being loaded.  Measured at 262144 rows of 128, forward: 3 x 2
// 34.5 us, 4 x 1 35.8, 6 x 1 (spills) 41; backward: 2 x 2 51.6, 3 x 1 53.6, 1 x 3 57, 2 x 1 63.
constexpr int FWD_CTAS = 3, BWD_CTAS = 2, WORK = 2;

// sum over the LPV lanes that share a row (they differ in the low bits of the lane index)
template <int LPV>
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
  for (int o = LPV / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// sum over the 32 / LPV lanes that hold the same columns of different rows
template <int LPV>
__device__ __forceinline__ float col_sum(float v) {
#pragma unroll
  for (int o = LPV; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// what a lane holds of a row, as loaded: NV pieces of eight elements, widened pair by pair where they are used
template <typename T, int NV>
struct RowPart {
  uint4 u[NV][sizeof(T) / 2];
  __device__ __forceinline__ void load(const void* base, int64_t at, int step) {   // pieces `step` elements apart
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
      for (int i = 0; i < (int)sizeof(T) / 2; ++i) u[v][i] = reinterpret_cast<const uint4*>(static_cast<const T*>(base) + at + v * step)[i];
  }
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
      for (int i = 0; i < (int)sizeof(T) / 2; ++i) u[v][i] = make_uint4(0u, 0u, 0u, 0u);
  }
  __device__ __forceinline__ uint64_t pair(int v, int i) const {   // elements 2 i, 2 i + 1 of a piece
    if constexpr (sizeof(T) == 2) {
      const uint32_t w[4] = {u[v][0].x, u[v][0].y, u[v][0].z, u[v][0].w};
      return widen2<T>(w[i]);
    } else {
      const uint4 q = u[v][i >> 1];
      return i & 1 ? pack2(__uint_as_float(q.z), __uint_as_float(q.w)) : pack2(__uint_as_float(q.x), __uint_as_float(q.y));
    }
  }
};

template <typename T>
__device__ __forceinline__ void store_pairs(void* base, int64_t at, const uint64_t (&x)[4]) {
  float y[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 p = unpack2(x[i]);
    y[2 * i] = p.x;
    y[2 * i + 1] = p.y;
  }
  store8<T>(base, at, y);
}

template <int LPV, int NV>
__device__ __forceinline__ void load_param_pairs(const void* p, int dtype, int sub, float absent, uint64_t (&w)[NV][4]) {
#pragma unroll
  for (int v = 0; v < NV; ++v)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int d = (v * LPV + sub) * 8 + 2 * i;
      w[v][i] = p ? pack2(ld_param(p, d, dtype), ld_param(p, d + 1, dtype)) : pack2(absent, absent);
    }
}

// LPV lanes per row, NV pieces of eight elements per lane: D = 8 LPV NV.  A warp works on ROUNDS row groups while the next
// ROUNDS are being loaded.
template <typename T, int LPV, int NV, bool BIAS>
__global__ void __launch_bounds__(NT, sizeof(T) == 2 && NV == 1 ? FWD_CTAS : 2) norm_gate_fwd_kernel(const b200gdn_norm_gate_args a) {
  constexpr int D = 8 * LPV * NV, RW = 32 / LPV, ROUNDS = NV == 1 ? WORK : 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane % LPV, rloc = lane / LPV;
  const bool sig = a.flags & B200GDN_NORM_GATE_SIGMOID;
  uint64_t w[NV][4], b[BIAS ? NV : 1][4];
  load_param_pairs<LPV, NV>(a.weight, a.param_dtype, sub, 1.f, w);
  if constexpr (BIAS) load_param_pairs<LPV, NV>(a.bias, a.param_dtype, sub, 0.f, b);
  const int64_t stride = (int64_t)gridDim.x * (NT / 32) * RW;
  RowPart<T, NV> x[ROUNDS], g[ROUNDS];
  auto fetch = [&](int64_t w0) {
#pragma unroll
    for (int u = 0; u < ROUNDS; ++u) {
      const int64_t r = w0 + u * stride + rloc;
      if (r < a.rows) {
        x[u].load(a.x, r * D + sub * 8, LPV * 8);
        g[u].load(a.g, r * D + sub * 8, LPV * 8);
      } else {
        x[u].zero();
        g[u].zero();
      }
    }
  };
  // the loop bound is the warp's first row, so that every lane takes part in the shuffles of a round
  int64_t w0 = ((int64_t)blockIdx.x * (NT / 32) + warp) * RW;
  fetch(w0);
  while (w0 < a.rows) {
    RowPart<T, NV> xc[ROUNDS], gc[ROUNDS];
#pragma unroll
    for (int u = 0; u < ROUNDS; ++u) {
      xc[u] = x[u];
      gc[u] = g[u];
    }
    const int64_t cur = w0;
    w0 += ROUNDS * stride;
    fetch(w0);
#pragma unroll
    for (int u = 0; u < ROUNDS; ++u) {
      const int64_t r = cur + u * stride + rloc;
      if (cur + u * stride >= a.rows) break;   // warp-uniform
      uint64_t sq = 0ull;
#pragma unroll
      for (int v = 0; v < NV; ++v)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint64_t p = xc[u].pair(v, i);
          sq = fma2(p, p, sq);
        }
      const float2 sp = unpack2(sq);
      const float ss = row_sum<LPV>(sp.x + sp.y);
      const float rstd = 1.f / sqrtf(ss / D + a.eps);
      if (r < a.rows) {
        if (sub == 0 && a.rstd != nullptr) a.rstd[r] = rstd;
        const uint64_t rs2 = pack2(rstd, rstd);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          uint64_t y[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint64_t gp = gc[u].pair(v, i), s = fast_sigmoid2(gp), n = mul2(xc[u].pair(v, i), rs2);
            const uint64_t act = sig ? s : mul2(gp, s);
            y[i] = mul2(BIAS ? fma2(n, w[v][i], b[BIAS ? v : 0][i]) : mul2(n, w[v][i]), act);
          }
          store_pairs<T>(a.y, r * D + (v * LPV + sub) * 8, y);
        }
      }
    }
  }
}

template <typename T, int LPV, int NV, bool BIAS>
__global__ void __launch_bounds__(NT, sizeof(T) == 2 && NV == 1 ? BWD_CTAS : 1) norm_gate_bwd_kernel(const b200gdn_norm_gate_args a) {
  constexpr int D = 8 * LPV * NV, RW = 32 / LPV, ROUNDS = NV == 1 ? WORK : 1;
  __shared__ float part[2][NT / 32][D];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane % LPV, rloc = lane / LPV;
  const bool sig = a.flags & B200GDN_NORM_GATE_SIGMOID;
  uint64_t w[NV][4], b[BIAS ? NV : 1][4], dw[NV][4], db[BIAS ? NV : 1][4];
  load_param_pairs<LPV, NV>(a.weight, a.param_dtype, sub, 1.f, w);
  if constexpr (BIAS) load_param_pairs<LPV, NV>(a.bias, a.param_dtype, sub, 0.f, b);
#pragma unroll
  for (int v = 0; v < NV; ++v)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      dw[v][i] = 0ull;
      if constexpr (BIAS) db[v][i] = 0ull;
    }
  const int64_t stride = (int64_t)gridDim.x * (NT / 32) * RW;
  RowPart<T, NV> x[ROUNDS], g[ROUNDS], dy[ROUNDS];
  float rs[ROUNDS];
  auto fetch = [&](int64_t w0) {
#pragma unroll
    for (int u = 0; u < ROUNDS; ++u) {
      const int64_t r = w0 + u * stride + rloc;
      if (r < a.rows) {
        rs[u] = a.rstd[r];
        x[u].load(a.x, r * D + sub * 8, LPV * 8);
        g[u].load(a.g, r * D + sub * 8, LPV * 8);
        dy[u].load(a.dy, r * D + sub * 8, LPV * 8);
      } else {   // a row past the end adds zeros to every sum
        rs[u] = 0.f;
        x[u].zero();
        g[u].zero();
        dy[u].zero();
      }
    }
  };
  int64_t w0 = ((int64_t)blockIdx.x * (NT / 32) + warp) * RW;
  fetch(w0);
  while (w0 < a.rows) {
    RowPart<T, NV> xc[ROUNDS], gc[ROUNDS], dyc[ROUNDS];
    float rc[ROUNDS];
#pragma unroll
    for (int u = 0; u < ROUNDS; ++u) {
      xc[u] = x[u];
      gc[u] = g[u];
      dyc[u] = dy[u];
      rc[u] = rs[u];
    }
    const int64_t cur = w0;
    w0 += ROUNDS * stride;
    fetch(w0);
#pragma unroll
    for (int u = 0; u < ROUNDS; ++u) {
      const int64_t r = cur + u * stride + rloc;
      if (cur + u * stride >= a.rows) break;   // warp-uniform
      const uint64_t rs2 = pack2(rc[u], rc[u]), one = pack2(1.f, 1.f), minus = pack2(-1.f, -1.f);
      uint64_t dx[NV][4], n[NV][4], dot2 = 0ull;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        uint64_t dg[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint64_t gi = gc[u].pair(v, i), dyi = dyc[u].pair(v, i), s = fast_sigmoid2(gi), q = fma2(s, minus, one);
          const uint64_t act = sig ? s : mul2(gi, s);
          const uint64_t dact = sig ? mul2(s, q) : fma2(act, q, s);   // s (1 - s) | s + g s (1 - s)
          n[v][i] = mul2(xc[u].pair(v, i), rs2);
          const uint64_t y0 = BIAS ? fma2(n[v][i], w[v][i], b[BIAS ? v : 0][i]) : mul2(n[v][i], w[v][i]);
          const uint64_t dy0 = mul2(dyi, act);
          dg[i] = mul2(mul2(dyi, y0), dact);
          dw[v][i] = fma2(dy0, n[v][i], dw[v][i]);
          if constexpr (BIAS) db[v][i] = add2(db[v][i], dy0);
          dx[v][i] = mul2(dy0, w[v][i]);   // gradient w.r.t. the normalised row
          dot2 = fma2(dx[v][i], n[v][i], dot2);
        }
        if (r < a.rows) store_pairs<T>(a.dg, r * D + (v * LPV + sub) * 8, dg);
      }
      const float2 dp = unpack2(dot2);
      const float dot = -row_sum<LPV>(dp.x + dp.y) / D;
      if (r < a.rows) {
        const uint64_t d2 = pack2(dot, dot);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
#pragma unroll
          for (int i = 0; i < 4; ++i) dx[v][i] = mul2(rs2, fma2(n[v][i], d2, dx[v][i]));
          store_pairs<T>(a.dx, r * D + (v * LPV + sub) * 8, dx[v]);
        }
      }
    }
  }
  // one partial row per CTA: the rows of a warp added by shuffles, then the warps' sums in warp order
#pragma unroll
  for (int v = 0; v < NV; ++v)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int d = (v * LPV + sub) * 8 + 2 * i;
      const float2 pw = unpack2(dw[v][i]);
      const float s0 = col_sum<LPV>(pw.x), s1 = col_sum<LPV>(pw.y);
      if (rloc == 0) *reinterpret_cast<float2*>(&part[0][warp][d]) = make_float2(s0, s1);
      if constexpr (BIAS) {
        const float2 pb = unpack2(db[v][i]);
        const float t0 = col_sum<LPV>(pb.x), t1 = col_sum<LPV>(pb.y);
        if (rloc == 0) *reinterpret_cast<float2*>(&part[1][warp][d]) = make_float2(t0, t1);
      }
    }
  __syncthreads();
  for (int idx = threadIdx.x; idx < (BIAS ? 2 : 1) * D; idx += NT) {
    const int which = idx / D, d = idx % D;
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < NT / 32; ++q) s += part[which][q][d];
    a.partials[((int64_t)blockIdx.x * 2 + which) * D + d] = s;
  }
}

// dweight / dbias = sum of the CTAs' partial rows in a fixed order: warp q adds rows q, q + 32, ... for 32 consecutive
// outputs, then the 32 sums are added in warp order
constexpr int RW = 32;
__global__ void __launch_bounds__(32 * RW) norm_gate_param_reduce_kernel(const b200gdn_norm_gate_args a, int n_ctas) {
  __shared__ float part[RW][32];
  const int lane = threadIdx.x & 31, q = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;   // D is a multiple of 32: every lane of a CTA has an output
  const int which = i / a.D, d = i % a.D;
  float s4[4] = {0.f, 0.f, 0.f, 0.f};   // four interleaved running sums, so that the loads overlap
  int c = q;
  for (; c + 3 * RW < n_ctas; c += 4 * RW) {
#pragma unroll
    for (int e = 0; e < 4; ++e) s4[e] += a.partials[((int64_t)(c + e * RW) * 2 + which) * a.D + d];
  }
  for (; c < n_ctas; c += RW) s4[0] += a.partials[((int64_t)c * 2 + which) * a.D + d];
  float s = (s4[0] + s4[1]) + (s4[2] + s4[3]);
  part[q][lane] = s;
  __syncthreads();
  if (q != 0) return;
#pragma unroll
  for (int r = 1; r < RW; ++r) s += part[r][lane];
  if (which == 0) { if (a.dweight) st_param(a.dweight, d, a.param_dtype, s); }
  else if (a.dbias) st_param(a.dbias, d, a.param_dtype, s);
}

template <typename T, int LPV, int NV>
int launch_t(const b200gdn_norm_gate_args& a, cudaStream_t st, bool bwd, int n_ctas) {
  const bool bias = a.bias != nullptr || (bwd && a.dbias != nullptr);
  if (!bwd) {
    if (bias) norm_gate_fwd_kernel<T, LPV, NV, true><<<n_ctas, NT, 0, st>>>(a);
    else norm_gate_fwd_kernel<T, LPV, NV, false><<<n_ctas, NT, 0, st>>>(a);
    return check_launch("norm_gate_fwd");
  }
  if (bias) norm_gate_bwd_kernel<T, LPV, NV, true><<<n_ctas, NT, 0, st>>>(a);
  else norm_gate_bwd_kernel<T, LPV, NV, false><<<n_ctas, NT, 0, st>>>(a);
  if (int e = check_launch("norm_gate_bwd")) return e;
  if (a.dweight != nullptr || a.dbias != nullptr) {
    norm_gate_param_reduce_kernel<<<(bias ? 2 : 1) * a.D / 32, 32 * RW, 0, st>>>(a, n_ctas);
    return check_launch("norm_gate_param_reduce");
  }
  return 0;
}

template <typename T>
int launch_d(const b200gdn_norm_gate_args& a, cudaStream_t st, bool bwd, int n_ctas) {
  switch (a.D) {
    case 64: return launch_t<T, 8, 1>(a, st, bwd, n_ctas);
    case 128: return launch_t<T, 16, 1>(a, st, bwd, n_ctas);
    case 256: return launch_t<T, 32, 1>(a, st, bwd, n_ctas);
    case 512: return launch_t<T, 32, 2>(a, st, bwd, n_ctas);
  }
  return set_error(B200GDN_ERR_UNSUPPORTED, "norm_gate: D=%d (64, 128, 256 and 512 are built)", a.D);
}

}  // namespace

// CTAs of the backward kernel for a row count (one partial row each): as many as fit on the device at once
int norm_gate_grid(int64_t rows) {
  const int64_t want = (rows + NT / 32 - 1) / (NT / 32), most = BWD_CTAS * sm_count();
  return (int)(want < 1 ? 1 : (want > most ? most : want));
}

int launch_norm_gate(const b200gdn_norm_gate_args& a, cudaStream_t st, bool bwd) {
  int n = norm_gate_grid(a.rows);
  if (!bwd) {
    const int64_t want = (a.rows + NT / 32 - 1) / (NT / 32), most = FWD_CTAS * sm_count();
    n = (int)(want < 1 ? 1 : (want > most ? most : want));
  }
  return a.dtype == 0 ? launch_d<__nv_bfloat16>(a, st, bwd, n) : a.dtype == 1 ? launch_d<__half>(a, st, bwd, n) : launch_d<float>(a, st, bwd, n);
}

}  // namespace gdn
