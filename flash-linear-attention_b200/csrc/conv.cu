// Short causal depthwise convolution (+ SiLU) over token-major [rows, D] activations, forward and backward: the step
// in front of the mixer in fla.layers.GatedDeltaNet (fla/layers/gated_deltanet.py:247-300).  Replaces
// causal_conv1d_fwd_kernel / causal_conv1d_bwd_kernel (fla/modules/conv/triton/ops.py) for kernel sizes 2..4:
//     y[t, d] = act( bias[d] + sum_{w < W} weight[d, w] x[t - (W-1) + w, d] ) (+ residual[t, d])
// inside each sequence; inputs before the sequence start come from the cache initial_state[n, d, W - k] = x[-k]
// (k = 1..W-1) or are zero; final_state[n, d, :] holds the last W inputs of the sequence (cache entries shifted in when
// the sequence is shorter than W).
//
// HBM streaming: a thread owns four consecutive channels and walks the tokens of its share with the W-1 previous inputs in
// registers, so x is read once (plus W-1 rows of overlap per share) and y written once.  Channels are handled in pairs by
// two-wide fp32 instructions, loads run four to eight tokens ahead in registers, and groups of four tokens are unrolled so
// that the history is renamed, not moved.  The backward pass recomputes the pre-activation, forms dx with a register ring
// over the W taps (the W-1 tokens after the share are evaluated again for their contribution to its dx), writes the
// gradient of the cache for a sequence's first share, and leaves per-share sums of dweight / dbias that a second kernel
// adds in a fixed order (no atomics: results are bit-reproducible).
// One token per sequence (a decoding step) has a kernel of its own: no walk, the cache as whole words.
// bf16, W = 4, SiLU, [4, 4096, 2048]: forward 27.3 us (4.9 TB/s of x and y; 35.3 with scalar instructions behind a ring of
// asynchronous copies, 32.1 with the activation, the residual and every token's place decided at run time), backward 54.8 us
// (80.9, 61.4) + 4.1 (6.7) for the parameter sums.  What is left to the copy rate is instruction issue (half of the cycles)
// and latency at the warps that the registers allow (an eighth forward or a fifth backward CTA spills: 28.1 and 80.6 us;
// 16-byte accesses with eight channels a thread: 40.9).  A decoding step of 32 users: 2.3 us (4.9).
#include <type_traits>

#include "gdn_common.cuh"
#include "rowio.cuh"

namespace gdn {
namespace {

constexpr int CT = 128;    // threads per CTA
constexpr int C = 4;       // channels per thread
constexpr int GRP = 4;     // tokens per group: one group is computed while one or two are being loaded

// the thread's channels of one token as loaded (8 bytes, 16 for fp32)
template <typename T>
struct Raw {
  static constexpr int N = C * (int)sizeof(T) / 4;   // 32-bit words
  uint32_t w[N];
  __device__ __forceinline__ void load(const void* base, int64_t idx) {
    const T* p = static_cast<const T*>(base) + idx;
    if constexpr (N == 4) *reinterpret_cast<uint4*>(w) = __ldg(reinterpret_cast<const uint4*>(p));
    else *reinterpret_cast<uint2*>(w) = __ldg(reinterpret_cast<const uint2*>(p));
  }
  __device__ __forceinline__ void get(uint64_t (&x)[C / 2]) const {
#pragma unroll
    for (int i = 0; i < C / 2; ++i) {
      if constexpr (sizeof(T) == 2) x[i] = widen2<T>(w[i]);
      else x[i] = pack2(__uint_as_float(w[2 * i]), __uint_as_float(w[2 * i + 1]));
    }
  }
};
template <typename T>
__device__ __forceinline__ void store_pairs(void* base, int64_t idx, const uint64_t (&x)[C / 2]) {
  Raw<T> r;
#pragma unroll
  for (int i = 0; i < C / 2; ++i) {
    if constexpr (sizeof(T) == 2) {
      r.w[i] = narrow2<T>(x[i]);
    } else {
      const float2 f = unpack2(x[i]);
      r.w[2 * i] = __float_as_uint(f.x);
      r.w[2 * i + 1] = __float_as_uint(f.y);
    }
  }
  T* p = static_cast<T*>(base) + idx;
  if constexpr (Raw<T>::N == 4) *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(r.w);
  else *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(r.w);
}

// One CTA's share of a tile: `row` is its first token, `len` its token count, `pos` that token's place in its sequence,
// `after` how many tokens of the sequence follow it (capped at 3, the largest overlap needed).
struct Share {
  int n, row, len, pos, after;
};
__device__ __forceinline__ Share load_share(const b200gdn_conv_args& a, int tile, int sub, int tokens) {
  const int4 m = reinterpret_cast<const int4*>(a.tile_meta)[tile];
  const int ntiles = a.seq_meta[2 * m.x + 1];
  const int start = sub * tokens;
  Share s;
  s.n = m.x;
  s.row = m.y + start;
  s.len = m.z - start < tokens ? m.z - start : tokens;   // <= 0: nothing to do for this CTA
  s.pos = m.w * BT + start;
  const int rest = m.z - start - s.len;                  // tokens of the tile behind this share
  int after = rest;
  if (after < 3 && m.w < ntiles - 1) after += a.tile_meta[4 * (tile + 1) + 2];
  s.after = after < 3 ? (after < 0 ? 0 : after) : 3;
  return s;
}

// x of channels d0.. at place `pos` of sequence n (row0: the row of place 0): a row of x, a cache entry, or zero
template <typename T, int W>
__device__ __forceinline__ void input_at(const b200gdn_conv_args& a, int n, int64_t row0, int pos, int d0, uint64_t (&x)[C / 2]) {
  if (pos >= 0) {
    Raw<T> r;
    r.load(a.x, (row0 + pos) * a.D + d0);
    r.get(x);
  } else {
#pragma unroll
    for (int i = 0; i < C / 2; ++i) {
      float v[2] = {0.f, 0.f};
      if (a.initial_state != nullptr && pos >= -W)
#pragma unroll
        for (int e = 0; e < 2; ++e) v[e] = Io<T>::ld(a.initial_state, ((int64_t)n * a.D + d0 + 2 * i + e) * W + (W + pos));
      x[i] = pack2(v[0], v[1]);
    }
  }
}

template <int W>
struct Taps {
  uint64_t w[W][C / 2], b[C / 2];
  __device__ __forceinline__ void load(const b200gdn_conv_args& a, int d0) {
#pragma unroll
    for (int i = 0; i < C / 2; ++i) {
      const int d = d0 + 2 * i;
#pragma unroll
      for (int j = 0; j < W; ++j)
        w[j][i] = pack2(ld_param(a.weight, (int64_t)d * W + j, a.param_dtype), ld_param(a.weight, (int64_t)(d + 1) * W + j, a.param_dtype));
      b[i] = a.bias ? pack2(ld_param(a.bias, d, a.param_dtype), ld_param(a.bias, d + 1, a.param_dtype)) : 0ull;
    }
  }
  // bias + sum of the taps; hist[j] is x[t - (W-1) + j]
  __device__ __forceinline__ uint64_t pre(const uint64_t (&hist)[W - 1][C / 2], const uint64_t (&cur)[C / 2], int i) const {
    uint64_t acc = fma2(w[W - 1][i], cur[i], b[i]);
#pragma unroll
    for (int j = 0; j < W - 1; ++j) acc = fma2(w[j][i], hist[j][i], acc);
    return acc;
  }
};

template <typename T, int W, bool ACT, bool RES>
__global__ void __launch_bounds__(CT, sizeof(T) == 4 ? 5 : 7) conv_fwd_kernel(const b200gdn_conv_args a, const int tokens) {
  const int d0 = (blockIdx.y * CT + threadIdx.x) * C;
  if (d0 >= a.D) return;
  const Share s = load_share(a, blockIdx.x, blockIdx.z, tokens);
  if (s.len <= 0) return;
  uint64_t hist[W - 1][C / 2];
#pragma unroll
  for (int j = 0; j < W - 1; ++j) input_at<T, W>(a, s.n, s.row - s.pos, s.pos - (W - 1) + j, d0, hist[j]);
  // The last inputs of a sequence are stored by the CTA of its FIRST share: the cache may be updated in place, and its
  // entries are read by the threads of that share alone (as the tokens before it, and below where the sequence is shorter
  // than W), each of which has read what it overwrites.
  if (a.final_state != nullptr && s.pos == 0) {
    const int ntiles = a.seq_meta[2 * s.n + 1], length = (ntiles - 1) * BT + a.tile_meta[4 * (blockIdx.x + ntiles - 1) + 2];
    uint64_t fin[W][C / 2];
#pragma unroll
    for (int j = 0; j < W; ++j) input_at<T, W>(a, s.n, s.row, length - W + j, d0, fin[j]);
#pragma unroll
    for (int i = 0; i < C / 2; ++i)
#pragma unroll
      for (int j = 0; j < W; ++j) {
        const float2 f = unpack2(fin[j][i]);
        Io<T>::st(a.final_state, ((int64_t)s.n * a.D + d0 + 2 * i) * W + j, f.x);
        Io<T>::st(a.final_state, ((int64_t)s.n * a.D + d0 + 2 * i + 1) * W + j, f.y);
      }
  }
  const int64_t base = (int64_t)s.row * a.D + d0;
  const T* const x = static_cast<const T*>(a.x) + base;
  T* const y_out = static_cast<T*>(a.y) + base;
  Raw<T> buf[2][GRP];
  auto fetch = [&](int t0, Raw<T> (&r)[GRP]) {
    const T* p = x + (int64_t)t0 * a.D;
    if (t0 + GRP <= s.len) {
#pragma unroll
      for (int u = 0; u < GRP; ++u, p += a.D) r[u].load(p, 0);
    } else {
#pragma unroll
      for (int u = 0; u < GRP; ++u, p += a.D)
        if (t0 + u < s.len) r[u].load(p, 0);
    }
  };
  fetch(0, buf[0]);
  fetch(GRP, buf[1]);
  Taps<W> k;
  k.load(a, d0);
  auto group = [&](int t0, Raw<T> (&r)[GRP], auto full) {
    T* p = y_out + (int64_t)t0 * a.D;
#pragma unroll
    for (int u = 0; u < GRP; ++u, p += a.D) {
      if (!decltype(full)::value && t0 + u >= s.len) return;
      uint64_t cur[C / 2], y[C / 2];
      r[u].get(cur);
#pragma unroll
      for (int i = 0; i < C / 2; ++i) {
        y[i] = k.pre(hist, cur, i);
        if (ACT) y[i] = mul2(y[i], fast_sigmoid2(y[i]));
      }
      if (RES) {
        Raw<T> q;
        uint64_t res[C / 2];
        q.load(a.residual, base + (int64_t)(t0 + u) * a.D);
        q.get(res);
#pragma unroll
        for (int i = 0; i < C / 2; ++i) y[i] = add2(y[i], res[i]);
      }
      store_pairs<T>(p, 0, y);
#pragma unroll
      for (int j = 0; j < W - 2; ++j)
#pragma unroll
        for (int i = 0; i < C / 2; ++i) hist[j][i] = hist[j + 1][i];
#pragma unroll
      for (int i = 0; i < C / 2; ++i) hist[W - 2][i] = cur[i];
    }
  };
  for (int t0 = 0; t0 < s.len; t0 += 2 * GRP) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int t = t0 + h * GRP;
      if (t + GRP <= s.len) group(t, buf[h], std::true_type{});
      else if (t < s.len) group(t, buf[h], std::false_type{});
      fetch(t + 2 * GRP, buf[h]);
    }
  }
}

// One token per sequence (row n = sequence n): latency of one round of loads.  With W = 4 a thread's 16 cache entries are
// whole 16-byte words.
template <typename T, int W>
__global__ void __launch_bounds__(CT) conv_step_kernel(const b200gdn_conv_args a) {
  const int d0 = (blockIdx.x * CT + threadIdx.x) * C, n = blockIdx.y;
  if (d0 >= a.D) return;
  const int64_t off = (int64_t)n * a.D + d0;
  const bool words = W == 4 && ((reinterpret_cast<uintptr_t>(a.initial_state) | reinterpret_cast<uintptr_t>(a.final_state)) & 15) == 0;
  Raw<T> raw;
  raw.load(a.x, off);
  float c[C * W];   // the cache, channel after channel
#pragma unroll
  for (int i = 0; i < C * W; ++i) c[i] = 0.f;
  if (a.initial_state != nullptr) {
    if (words) {
#pragma unroll
      for (int i = 0; i < C * W / 8; ++i) {
        float z[8];
        load8<T>(a.initial_state, off * W + 8 * i, z);
#pragma unroll
        for (int e = 0; e < 8; ++e) c[8 * i + e] = z[e];
      }
    } else {
#pragma unroll
      for (int i = 0; i < C * W; ++i) c[i] = Io<T>::ld(a.initial_state, off * W + i);
    }
  }
  Taps<W> k;
  k.load(a, d0);
  uint64_t cur[C / 2], y[C / 2], hist[W - 1][C / 2];
  raw.get(cur);
#pragma unroll
  for (int j = 0; j < W - 1; ++j)
#pragma unroll
    for (int i = 0; i < C / 2; ++i) hist[j][i] = pack2(c[2 * i * W + j + 1], c[(2 * i + 1) * W + j + 1]);
#pragma unroll
  for (int i = 0; i < C / 2; ++i) {
    y[i] = k.pre(hist, cur, i);
    if (a.flags & B200GDN_CONV_SILU) y[i] = mul2(y[i], fast_sigmoid2(y[i]));
  }
  if (a.residual) {
    Raw<T> q;
    uint64_t res[C / 2];
    q.load(a.residual, off);
    q.get(res);
#pragma unroll
    for (int i = 0; i < C / 2; ++i) y[i] = add2(y[i], res[i]);
  }
  store_pairs<T>(a.y, off, y);
  if (a.final_state == nullptr) return;
#pragma unroll
  for (int i = 0; i < C; ++i) {   // shift the token in
    const float2 f = unpack2(cur[i / 2]);
#pragma unroll
    for (int j = 0; j < W - 1; ++j) c[i * W + j] = c[i * W + j + 1];
    c[i * W + W - 1] = i & 1 ? f.y : f.x;
  }
  if (words) {
#pragma unroll
    for (int i = 0; i < C * W / 8; ++i) {
      float z[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) z[e] = c[8 * i + e];
      store8<T>(a.final_state, off * W + 8 * i, z);
    }
  } else {
#pragma unroll
    for (int i = 0; i < C * W; ++i) Io<T>::st(a.final_state, off * W + i, c[i]);
  }
}

template <typename T, int W, bool ACT, bool BIAS>
__global__ void __launch_bounds__(CT, sizeof(T) == 4 ? 3 : 4) conv_bwd_kernel(const b200gdn_conv_args a, const int tokens) {
  const int d0 = (blockIdx.y * CT + threadIdx.x) * C;
  if (d0 >= a.D) return;
  const Share s = load_share(a, blockIdx.x, blockIdx.z, tokens);
  // sums of this share: [W + 1][D], taps then bias
  float* const part = a.partials ? a.partials + ((int64_t)blockIdx.x * gridDim.z + blockIdx.z) * (W + 1) * a.D + d0 : nullptr;
  auto put = [&](int j, const uint64_t (&x)[C / 2]) {
    const float2 p = unpack2(x[0]), q = unpack2(x[1]);
    *reinterpret_cast<float4*>(part + (int64_t)j * a.D) = make_float4(p.x, p.y, q.x, q.y);
  };
  if (s.len <= 0) {   // no token in this share: its sums are zeros
    const uint64_t zero[C / 2] = {};
    if (part != nullptr)
      for (int j = 0; j <= W; ++j) put(j, zero);
    return;
  }
  // tokens of the same sequence after this share whose pre-activation gradient reaches its dx
  const int n_tok = s.len + (s.after < W - 1 ? s.after : W - 1);
  const int64_t base = (int64_t)s.row * a.D + d0;
  Raw<T> bx[2][GRP], by[2][GRP];
  auto fetch = [&](int t0, Raw<T> (&rx)[GRP], Raw<T> (&ry)[GRP]) {
    int64_t at = base + (int64_t)t0 * a.D;
    if (t0 + GRP <= n_tok) {
#pragma unroll
      for (int u = 0; u < GRP; ++u, at += a.D) {
        rx[u].load(a.x, at);
        ry[u].load(a.dy, at);
      }
    } else {
#pragma unroll
      for (int u = 0; u < GRP; ++u, at += a.D)
        if (t0 + u < n_tok) {
          rx[u].load(a.x, at);
          ry[u].load(a.dy, at);
        }
    }
  };
  fetch(0, bx[0], by[0]);
  fetch(GRP, bx[1], by[1]);
  Taps<W> k;
  k.load(a, d0);
  uint64_t hist[W - 1][C / 2];
#pragma unroll
  for (int j = 0; j < W - 1; ++j) input_at<T, W>(a, s.n, s.row - s.pos, s.pos - (W - 1) + j, d0, hist[j]);
  uint64_t ring[W - 1][C / 2];   // ring[m]: dx of token (u - 1 - m) so far, u the token being processed
  uint64_t dw[W][C / 2], db[C / 2];
#pragma unroll
  for (int i = 0; i < C / 2; ++i) {
    db[i] = 0ull;
#pragma unroll
    for (int j = 0; j < W; ++j) dw[j][i] = 0ull;
#pragma unroll
    for (int j = 0; j < W - 1; ++j) ring[j][i] = 0ull;
  }
  const bool to_cache = s.pos == 0 && a.dinitial_state != nullptr;
  const int last = n_tok - 1 + (W - 1);   // the extra steps only flush the ring
  const uint64_t one = pack2(1.f, 1.f), mone = pack2(-1.f, -1.f);
  // one step; FULL: the token is known to lie inside the share (it is loaded and counted for the parameters) and not in its
  // first group, so nothing is conditional and the compiler renames the history and ring registers across the unrolled steps of a group
  auto step = [&](int u, const Raw<T>& rx, const Raw<T>& ry, auto full) {
    constexpr bool FULL = decltype(full)::value;
    if (!FULL && u > last) return;
    uint64_t dpre[C / 2];
    if (FULL || u < n_tok) {
      uint64_t cur[C / 2];
      rx.get(cur);
      ry.get(dpre);
#pragma unroll
      for (int i = 0; i < C / 2; ++i) {
        if (ACT) {   // d silu(p) = s (1 + p (1 - s))
          const uint64_t p = k.pre(hist, cur, i), sg = fast_sigmoid2(p);
          dpre[i] = mul2(dpre[i], mul2(sg, fma2(p, fma2(sg, mone, one), one)));
        }
        if (FULL || u < s.len) {   // the parameters' gradients: every token is counted by the share that owns it
          if (BIAS) db[i] = add2(db[i], dpre[i]);
          dw[W - 1][i] = fma2(dpre[i], cur[i], dw[W - 1][i]);
#pragma unroll
          for (int j = 0; j < W - 1; ++j) dw[j][i] = fma2(dpre[i], hist[j][i], dw[j][i]);
        }
#pragma unroll
        for (int j = 0; j < W - 2; ++j) hist[j][i] = hist[j + 1][i];
        hist[W - 2][i] = cur[i];
      }
    } else {
#pragma unroll
      for (int i = 0; i < C / 2; ++i) dpre[i] = 0ull;
    }
    // dpre[u] reaches token u - m through tap W - 1 - m; token u - (W - 1) is complete with it
    uint64_t done[C / 2];
#pragma unroll
    for (int i = 0; i < C / 2; ++i) {
      done[i] = fma2(k.w[0][i], dpre[i], ring[W - 2][i]);
#pragma unroll
      for (int m = W - 2; m > 0; --m) ring[m][i] = fma2(k.w[W - 1 - m][i], dpre[i], ring[m - 1][i]);
      ring[0][i] = mul2(k.w[W - 1][i], dpre[i]);
    }
    const int e = u - (W - 1);
    if (FULL) {
      store_pairs<T>(a.dx, base + (int64_t)e * a.D, done);
    } else if (e >= 0) {
      if (e < s.len) store_pairs<T>(a.dx, base + (int64_t)e * a.D, done);
    } else if (to_cache) {   // an input before the sequence start: gradient of the cache entry x[e] = initial_state[n, d, W + e]
#pragma unroll
      for (int i = 0; i < C / 2; ++i) {
        const float2 f = unpack2(done[i]);
        Io<T>::st(a.dinitial_state, ((int64_t)s.n * a.D + d0 + 2 * i) * W + (W + e), f.x);
        Io<T>::st(a.dinitial_state, ((int64_t)s.n * a.D + d0 + 2 * i + 1) * W + (W + e), f.y);
      }
    }
  };
  for (int t0 = 0; t0 <= last; t0 += 2 * GRP) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int t = t0 + h * GRP;
      if (t >= GRP && t + GRP <= s.len) {
#pragma unroll
        for (int v = 0; v < GRP; ++v) step(t + v, bx[h][v], by[h][v], std::true_type{});
      } else {
#pragma unroll
        for (int v = 0; v < GRP; ++v) step(t + v, bx[h][v], by[h][v], std::false_type{});
      }
      fetch(t + 2 * GRP, bx[h], by[h]);
    }
  }
  if (to_cache) {   // the cache's oldest entry never enters the convolution
#pragma unroll
    for (int c = 0; c < C; ++c) Io<T>::st(a.dinitial_state, ((int64_t)s.n * a.D + d0 + c) * W, 0.f);
  }
  if (part != nullptr) {
#pragma unroll
    for (int j = 0; j < W; ++j) put(j, dw[j]);
    if (BIAS) put(W, db);
  }
}

// dweight[d, w] / dbias[d] = sum over the shares in a fixed order: warp q of a CTA adds shares q, q + 16, ... for 32
// consecutive outputs (four interleaved running sums, so that the loads overlap), then the sixteen sums are added in
// warp order
constexpr int RW = 16;
__global__ void __launch_bounds__(32 * RW) conv_param_reduce_kernel(const b200gdn_conv_args a, const int n) {
  __shared__ float part[RW][32];
  const int lane = threadIdx.x & 31, q = threadIdx.x >> 5;
  const int64_t per_share = (int64_t)a.D * (a.W + 1), n_out = (int64_t)a.D * (a.W + (a.dbias != nullptr));
  const int64_t i = (int64_t)blockIdx.x * 32 + lane;
  float s4[4] = {0.f, 0.f, 0.f, 0.f};
  if (i < n_out) {
    int t = q;
    for (; t + 3 * RW < n; t += 4 * RW) {
#pragma unroll
      for (int e = 0; e < 4; ++e) s4[e] += a.partials[(int64_t)(t + e * RW) * per_share + i];
    }
    for (; t < n; t += RW) s4[0] += a.partials[(int64_t)t * per_share + i];
  }
  float s = (s4[0] + s4[1]) + (s4[2] + s4[3]);
  part[q][lane] = s;
  __syncthreads();
  if (q != 0 || i >= n_out) return;
#pragma unroll
  for (int r = 1; r < RW; ++r) s += part[r][lane];
  const int j = (int)(i / a.D), d = (int)(i % a.D);
  if (j < a.W) st_param(a.dweight, (int64_t)d * a.W + j, a.param_dtype, s);
  else st_param(a.dbias, d, a.param_dtype, s);
}

// Tokens per share: a whole tile of 64 while that still gives the SMs twelve warps each, else 32 (and 16 forward; a
// backward share also costs a row of parameter sums, and the workspace holds two per tile).
int share_tokens(const b200gdn_conv_args& a, int least) {
  int64_t warps = (int64_t)a.n_tiles * ((a.D / C + 31) / 32);
  int tokens = 64;
  for (; tokens > least && warps < 12 * sm_count(); warps *= 2) tokens /= 2;
  return tokens;
}

template <typename T, int W>
int launch_t(const b200gdn_conv_args& a, cudaStream_t st, bool bwd) {
  const unsigned y = (a.D / C + CT - 1) / CT;
  if (!bwd) {
    if (a.rows == a.n_tiles && a.n_seq == a.n_tiles && a.n_seq <= 65535) {   // every sequence is one token
      conv_step_kernel<T, W><<<dim3(y, a.n_seq), CT, 0, st>>>(a);
      return check_launch("conv_step");
    }
    const int tokens = share_tokens(a, 16);
    const dim3 grid(a.n_tiles, y, 64 / tokens);
    const bool act = a.flags & B200GDN_CONV_SILU;
    if (a.residual != nullptr) {
      if (act) conv_fwd_kernel<T, W, true, true><<<grid, CT, 0, st>>>(a, tokens);
      else conv_fwd_kernel<T, W, false, true><<<grid, CT, 0, st>>>(a, tokens);
    } else {
      if (act) conv_fwd_kernel<T, W, true, false><<<grid, CT, 0, st>>>(a, tokens);
      else conv_fwd_kernel<T, W, false, false><<<grid, CT, 0, st>>>(a, tokens);
    }
    return check_launch("conv_fwd");
  }
  const int tokens = share_tokens(a, 32);
  const dim3 grid(a.n_tiles, y, 64 / tokens);
  const bool act = a.flags & B200GDN_CONV_SILU;
  if (a.dbias != nullptr) {
    if (act) conv_bwd_kernel<T, W, true, true><<<grid, CT, 0, st>>>(a, tokens);
    else conv_bwd_kernel<T, W, false, true><<<grid, CT, 0, st>>>(a, tokens);
  } else {
    if (act) conv_bwd_kernel<T, W, true, false><<<grid, CT, 0, st>>>(a, tokens);
    else conv_bwd_kernel<T, W, false, false><<<grid, CT, 0, st>>>(a, tokens);
  }
  if (int e = check_launch("conv_bwd")) return e;
  if (a.partials != nullptr && a.dweight != nullptr) {
    const int64_t n = (int64_t)a.D * (a.W + (a.dbias != nullptr));
    conv_param_reduce_kernel<<<(unsigned)((n + 31) / 32), 32 * RW, 0, st>>>(a, a.n_tiles * (64 / tokens));
    return check_launch("conv_param_reduce");
  }
  return 0;
}

template <typename T>
int launch_w(const b200gdn_conv_args& a, cudaStream_t st, bool bwd) {
  if (a.W == 4) return launch_t<T, 4>(a, st, bwd);
  if (a.W == 3) return launch_t<T, 3>(a, st, bwd);
  if (a.W == 2) return launch_t<T, 2>(a, st, bwd);
  return set_error(B200GDN_ERR_UNSUPPORTED, "conv: kernel size %d (2, 3 and 4 are built)", a.W);
}

}  // namespace

int launch_conv(const b200gdn_conv_args& a, cudaStream_t st, bool bwd) {
  return a.dtype == 0 ? launch_w<__nv_bfloat16>(a, st, bwd) : a.dtype == 1 ? launch_w<__half>(a, st, bwd) : launch_w<float>(a, st, bwd);
}

}  // namespace gdn
