// Token-by-token gated delta rule (decode and short prefill), forward only:
//     S *= exp(g);  r = beta (v - S^T k);  S += k r^T;  o = S^T (scale q)
// Replaces fused_recurrent_gated_delta_rule_fwd_kernel (fla/ops/gated_delta_rule/fused_recurrent.py:30-181),
// including its in-kernel options (q/k L2 norm, -exp(A_log) softplus(g + dt_bias) gate, sigmoid beta,
// V-first state layout).  fp32 arithmetic throughout.  Four kernels:
//   recurrent_step_kernel   one token per sequence, small and middling batches: latency of one pass over the state
//   decode_stream_kernel    one token per sequence, large batches: pure state traffic (read + write K*V fp32)
//   recurrent_few_kernel    a few tokens per sequence: latency of the per-token chain
//   recurrent_pairs_kernel  more tokens per sequence: the same chain for two tokens at a time
#include "gdn_common.cuh"
#include "rowio.cuh"
#include "tc5.cuh"
#include "tma.cuh"

namespace gdn {
namespace {

constexpr int NTHREADS = 128;
constexpr int VS = 32;  // value channels per CTA

__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }

// Slot of the state pool that sequence n uses.  With a pool (state_indices) and a known pool size, an index outside
// [0, n_slots) marks a padding sequence (serving engines use -1): it reads slot 0, its output is meaningless and its
// state is not written back (`*writeback` = false), so no access leaves the pool.
__device__ __forceinline__ int64_t state_slot(const b200gdn_recurrent_args& a, int n, bool* writeback) {
  *writeback = true;
  if (a.state_indices == nullptr) return n;
  const int64_t slot = a.state_indices[n];
  if (a.n_slots > 0 && (slot < 0 || slot >= a.n_slots)) {
    *writeback = false;
    return 0;
  }
  return slot;
}

// RPL consecutive elements (a lane's rows of q or k) as fp32 pairs
template <typename T, int RPL>
__device__ __forceinline__ void load_pairs(const void* base, int64_t idx, bool wide, uint64_t (&x)[RPL / 2]) {
  const T* p = static_cast<const T*>(base) + idx;
  if constexpr (sizeof(T) == 2) {
    if (wide) {
      uint32_t w[RPL / 2];
      if constexpr (RPL >= 8) {
#pragma unroll
        for (int i = 0; i < RPL / 8; ++i) *reinterpret_cast<uint4*>(&w[4 * i]) = reinterpret_cast<const uint4*>(p)[i];
      } else if constexpr (RPL == 4) {
        *reinterpret_cast<uint2*>(w) = *reinterpret_cast<const uint2*>(p);
      } else {
        w[0] = *reinterpret_cast<const uint32_t*>(p);
      }
#pragma unroll
      for (int i = 0; i < RPL / 2; ++i) x[i] = widen2<T>(w[i]);
      return;
    }
  } else if (wide) {
    if constexpr (RPL >= 4) {
#pragma unroll
      for (int i = 0; i < RPL / 4; ++i) {
        const float4 f = reinterpret_cast<const float4*>(p)[i];
        x[2 * i] = pack2(f.x, f.y);
        x[2 * i + 1] = pack2(f.z, f.w);
      }
    } else {
      const float2 f = *reinterpret_cast<const float2*>(p);
      x[0] = pack2(f.x, f.y);
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < RPL / 2; ++i) x[i] = pack2(Io<T>::ld(p, 2 * i), Io<T>::ld(p, 2 * i + 1));
}

// The state of one warp: eight value channels with ALL K rows.  Lane l keeps rows (K/16)(l/2) .. and channels 4 (l%2) .. +3
// of the eight, as pairs of rows.
template <int DK, bool VFIRST>
struct WarpState {
  static constexpr int RPL = DK / 16, RP2 = RPL / 2;
  uint64_t st[RP2][4];   // st[i][j]: rows (r0 + 2 i, r0 + 2 i + 1), channel c0 + j
  __device__ __forceinline__ void load(const float* h, int r0, int c0, int DV) {
    if (h == nullptr) {
#pragma unroll
      for (int i = 0; i < RP2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) st[i][j] = 0ull;
    } else if (!VFIRST) {
#pragma unroll
      for (int i = 0; i < RP2; ++i) {
        const float4 x = *reinterpret_cast<const float4*>(h + (int64_t)(r0 + 2 * i) * DV + c0);
        const float4 y = *reinterpret_cast<const float4*>(h + (int64_t)(r0 + 2 * i + 1) * DV + c0);
        st[i][0] = pack2(x.x, y.x); st[i][1] = pack2(x.y, y.y); st[i][2] = pack2(x.z, y.z); st[i][3] = pack2(x.w, y.w);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < RP2; ++i) st[i][j] = *reinterpret_cast<const uint64_t*>(h + (int64_t)(c0 + j) * DK + r0 + 2 * i);
    }
  }
  __device__ __forceinline__ void store(float* h, int r0, int c0, int DV) const {
#pragma unroll
    for (int i = 0; i < RP2; ++i) {
      const float2 x0 = unpack2(st[i][0]), x1 = unpack2(st[i][1]), x2 = unpack2(st[i][2]), x3 = unpack2(st[i][3]);
      if (!VFIRST) {
        *reinterpret_cast<float4*>(h + (int64_t)(r0 + 2 * i) * DV + c0) = make_float4(x0.x, x1.x, x2.x, x3.x);
        *reinterpret_cast<float4*>(h + (int64_t)(r0 + 2 * i + 1) * DV + c0) = make_float4(x0.y, x1.y, x2.y, x3.y);
      } else {
        *reinterpret_cast<float2*>(h + (int64_t)(c0 + 0) * DK + r0 + 2 * i) = x0;
        *reinterpret_cast<float2*>(h + (int64_t)(c0 + 1) * DK + r0 + 2 * i) = x1;
        *reinterpret_cast<float2*>(h + (int64_t)(c0 + 2) * DK + r0 + 2 * i) = x2;
        *reinterpret_cast<float2*>(h + (int64_t)(c0 + 3) * DK + r0 + 2 * i) = x3;
      }
    }
  }
  // One token.  Both row reductions are taken from the state BEFORE its update,
  //     d = e^g kn S^T k;  r = beta (v - d);  o = e^g qn S^T q + <k,q> r;  S <- e^g S + (kn k) r^T,
  // so one round of shuffles (eight sums over sixteen lanes by recursive halving, eight shuffles) serves both.
  // k2, q2: the lane's rows of k and q as loaded; kn, qn: their factors; kq = <kn k, qn q>; v: the lane's four channels.
  // Returns o of channel c0 + ((lane >> 2) & 3), valid in lanes with bit 4 set.
  __device__ __forceinline__ float step(const uint64_t (&k2)[RP2], const uint64_t (&q2)[RP2], float kn, float qn, float kq, float dec,
                                        float beta, const float (&v)[4], int lane) {
    uint64_t ad[4], aq[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) ad[j] = aq[j] = 0ull;
#pragma unroll
    for (int i = 0; i < RP2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        ad[j] = fma2(st[i][j], k2[i], ad[j]);
        aq[j] = fma2(st[i][j], q2[i], aq[j]);
      }
    // afterwards a lane holds the sum (bit 4: 0 = S^T k, 1 = S^T q) of channel 2 (bit 3) + (bit 2) of its half
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    float x[4], y[2], z;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 d = unpack2(ad[j]), q = unpack2(aq[j]);
      const float sd = d.x + d.y, sq = q.x + q.y;
      x[j] = (b4 ? sq : sd) + __shfl_xor_sync(0xffffffffu, b4 ? sd : sq, 16);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) y[j] = (b3 ? x[2 + j] : x[j]) + __shfl_xor_sync(0xffffffffu, b3 ? x[j] : x[2 + j], 8);
    z = (b2 ? y[1] : y[0]) + __shfl_xor_sync(0xffffffffu, b2 ? y[0] : y[1], 4);
    z += __shfl_xor_sync(0xffffffffu, z, 2);
    z *= dec * (b4 ? qn : kn);
    float r[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) r[j] = beta * (v[j] - __shfl_sync(0xffffffffu, z, 4 * j + (lane & 1)));
    const uint64_t dec2 = pack2(dec, dec);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint64_t rr = pack2(r[j] * kn, r[j] * kn);
#pragma unroll
      for (int i = 0; i < RP2; ++i) st[i][j] = fma2(st[i][j], dec2, mul2(k2[i], rr));
    }
    const float rj = b3 ? (b2 ? r[3] : r[2]) : (b2 ? r[1] : r[0]);
    return z + kq * rj;
  }
};

// e^g and beta of one token with the layer's activations
__device__ __forceinline__ void load_gate_beta(const b200gdn_recurrent_args& a, int64_t row, int hv, float& gg, float& bb) {
  gg = a.g ? ld_param(a.g, row * a.HV + hv, a.gb_dtype) : 0.f;
  bb = ld_param(a.beta, row * a.HV + hv, a.gb_dtype);
}
template <typename Gate>   // the gate's value from its raw one, with the head's parameters
__device__ __forceinline__ void activate(const b200gdn_recurrent_args& a, Gate&& gate, float gg, float bb, float& dec, float& beta) {
  if (a.flags & B200GDN_REC_GATE) gg = gate(gg);
  if (a.flags & B200GDN_REC_BETA_SIGMOID) {
    bb = 1.f / (1.f + expf(-bb));
    if (a.flags & B200GDN_REC_NEG_EIGVAL) bb *= 2.f;
  }
  dec = expf(gg);
  beta = bb;
}
// The parameters are loaded here, where the option is on: as arguments they are loaded ahead of the branch and held, which cost two
// tokens of 16 x 32 heads, K = V = 128 with [V,K] states, 26.4 us for 25.2.
__device__ __forceinline__ void gate_beta(const b200gdn_recurrent_args& a, int64_t row, int hv, float& dec, float& beta) {
  float gg, bb;
  load_gate_beta(a, row, hv, gg, bb);
  auto gate = [&](float x) {
    if (a.dt_bias) x += a.dt_bias[hv];
    return -expf(a.A_log[hv]) * softplus_f(x);
  };
  activate(a, gate, gg, bb, dec, beta);
}

// One token per sequence: a CTA of four warps owns 32 value channels of one (sequence, head).  Every lane loads its own rows
// of q and k from global memory, so the time is one round of loads, one chain, one round of stores.
//  * [V,K] states: a warp has eight channels with all K rows to itself and there is no barrier at all;
//  * [K,V] states: a warp has K/4 rows of all 32 channels, so that a row is moved in whole 128-byte lines (with 32-byte
//    pieces of a row per warp the L1 line rate is the bound: 9.1 against 7.0 us at 15 sequences x 16 heads, K = V = 128), and
//    the four partial sums of S^T k and S^T q meet in shared memory behind ONE barrier (see WarpState::step).
template <int DK, bool VFIRST, typename T>
__global__ void __launch_bounds__(NTHREADS, DK <= 128 ? 7 : 3) recurrent_step_kernel(const b200gdn_recurrent_args a) {
  using W = WarpState<DK, VFIRST>;
  constexpr int RPL = W::RPL, RP2 = W::RP2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int hv = blockIdx.y, n = blockIdx.z, hq = hv / (a.HV / a.H), DV = a.V;
  const bool wide = ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k)) & 15) == 0;
  const int r0 = VFIRST ? (lane >> 1) * RPL : warp * (DK / 4) + (lane >> 3) * RPL;
  const int cl = VFIRST ? warp * 8 + (lane & 1) * 4 : (lane & 7) * 4, c0 = blockIdx.x * VS + cl;
  bool writeback;
  const int64_t slot = state_slot(a, n, &writeback);   // which state of the pool this sequence uses
  const int64_t qk_at = ((int64_t)n * a.H + hq) * DK, v_at = ((int64_t)n * a.HV + hv) * DV;
  uint64_t k2[RP2], q2[RP2];
  load_pairs<T, RPL>(a.k, qk_at + r0, wide, k2);
  load_pairs<T, RPL>(a.q, qk_at + r0, wide, q2);
  float v[4], dec, beta;
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] = Io<T>::ld(a.v, v_at + c0 + j);
  W w;
  w.load(a.h0 ? a.h0 + (slot * a.HV + hv) * DK * DV : nullptr, r0, c0, DV);
  gate_beta(a, n, hv, dec, beta);
  // <k,k>, <q,q>, <k,q> over all K rows.  [V,K]: the lane's rows, summed over the 16 lanes of a channel half
  float sm[3] = {0.f, 0.f, 0.f};
  if constexpr (VFIRST) {
#pragma unroll
    for (int i = 0; i < RP2; ++i) {
      const float2 k = unpack2(k2[i]), q = unpack2(q2[i]);
      sm[0] += k.x * k.x + k.y * k.y;
      sm[1] += q.x * q.x + q.y * q.y;
      sm[2] += k.x * q.x + k.y * q.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < DK / 32; ++i) {
      const float k = Io<T>::ld(a.k, qk_at + i * 32 + lane), q = Io<T>::ld(a.q, qk_at + i * 32 + lane);
      sm[0] += k * k;
      sm[1] += q * q;
      sm[2] += k * q;
    }
  }
#pragma unroll
  for (int e = 0; e < 3; ++e)
#pragma unroll
    for (int o = VFIRST ? 2 : 1; o <= 16; o <<= 1) sm[e] += __shfl_xor_sync(0xffffffffu, sm[e], o);
  const bool l2 = a.flags & B200GDN_REC_L2NORM;
  const float kn = l2 ? rsqrtf(sm[0] + 1e-6f) : 1.f, qn = l2 ? a.scale * rsqrtf(sm[1] + 1e-6f) : a.scale;
  const float kq = sm[2] * kn * qn;
  if constexpr (VFIRST) {
    const float o = w.step(k2, q2, kn, qn, kq, dec, beta, v, lane);
    if ((lane & 18) == 16) Io<T>::st(a.o, v_at + c0 + ((lane >> 2) & 3), o);
  } else {
    __shared__ __align__(16) float red[2][4][VS];
    float d[4], q[4];
    {
      uint64_t ad[4], aq[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) ad[j] = aq[j] = 0ull;
#pragma unroll
      for (int i = 0; i < RP2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          ad[j] = fma2(w.st[i][j], k2[i], ad[j]);
          aq[j] = fma2(w.st[i][j], q2[i], aq[j]);
        }
      // over the four row groups of the warp: bit 4 of the lane picks S^T k or S^T q, bit 3 completes the sum
      const bool b4 = lane & 16;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 x = unpack2(ad[j]), y = unpack2(aq[j]);
        const float sd = x.x + x.y, sq = y.x + y.y;
        d[j] = (b4 ? sq : sd) + __shfl_xor_sync(0xffffffffu, b4 ? sd : sq, 16);
        d[j] += __shfl_xor_sync(0xffffffffu, d[j], 8);
      }
      if ((lane & 8) == 0) *reinterpret_cast<float4*>(&red[lane >> 4][warp][cl]) = make_float4(d[0], d[1], d[2], d[3]);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j) d[j] = q[j] = 0.f;
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const float4 p = *reinterpret_cast<const float4*>(&red[0][x][cl]), s = *reinterpret_cast<const float4*>(&red[1][x][cl]);
      d[0] += p.x; d[1] += p.y; d[2] += p.z; d[3] += p.w;
      q[0] += s.x; q[1] += s.y; q[2] += s.z; q[3] += s.w;
    }
    const uint64_t dec2 = pack2(dec, dec);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float r = beta * (v[j] - dec * kn * d[j]);
      const uint64_t rr = pack2(r * kn, r * kn);
#pragma unroll
      for (int i = 0; i < RP2; ++i) w.st[i][j] = fma2(w.st[i][j], dec2, mul2(k2[i], rr));
      q[j] = dec * qn * q[j] + kq * r;
    }
    if (warp == 0 && lane < 8) {
#pragma unroll
      for (int j = 0; j < 4; ++j) Io<T>::st(a.o, v_at + c0 + j, q[j]);
    }
  }
  if (a.ht != nullptr && writeback) w.store(a.ht + (slot * a.HV + hv) * DK * DV, r0, c0, DV);
}

// A few tokens per sequence: a CTA of four warps owns 32 value channels of one (sequence, head).  q, k and v of TB tokens
// at a time reach shared memory as they are by asynchronous 16-byte copies, one block ahead (two buffers); the norms,
// <k,q>, e^g and beta of a block are formed once by the CTA; then every warp walks the block without a barrier.
// Bound by the latency of the per-token chain (K/32 multiply-adds, five shuffles in sequence, K/32 multiply-adds), about
// 0.26 us a token at K = 64 and 0.45 at K = 128.  128 sequences x 16 heads x 4 tokens, K = V = 128: 75.8 us (110.6 with the
// channels combined through shared memory, five barriers a token).
template <int DK, bool VFIRST, typename T>
__global__ void __launch_bounds__(NTHREADS) recurrent_few_kernel(const b200gdn_recurrent_args a) {
  using W = WarpState<DK, VFIRST>;
  constexpr int TB = 2048 / DK < 32 ? 2048 / DK : 32;   // tokens per block
  constexpr int E16 = 16 / (int)sizeof(T);              // elements of one 16-byte copy
  __shared__ __align__(16) T qs[2][TB * DK];
  __shared__ __align__(16) T ks[2][TB * DK];
  __shared__ __align__(16) T vs[2][TB * VS];
  __shared__ float sk_[TB], sq_[TB], skq[TB], sdec[TB], sbeta[TB];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int v0 = blockIdx.x * VS, hv = blockIdx.y, n = blockIdx.z, hq = hv / (a.HV / a.H), DV = a.V;
  int64_t bos;
  int len;
  if (a.cu_seqlens != nullptr) {
    bos = a.cu_seqlens[n];
    len = a.cu_seqlens[n + 1] - (int)bos;
  } else {
    bos = (int64_t)n * a.T;
    len = a.T;
  }
  const bool wide = ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k) | reinterpret_cast<uintptr_t>(a.v)) & 15) == 0;
  auto fetch = [&](int t0, int buf) {
    const int nt = len - t0 < TB ? len - t0 : TB;
    if (wide) {
      for (int i = tid; i < nt * (DK / E16); i += NTHREADS) {
        const int t = i / (DK / E16), c = (i % (DK / E16)) * E16;
        const int64_t at = ((bos + t0 + t) * a.H + hq) * DK + c;
        cp_async16(&qs[buf][t * DK + c], static_cast<const T*>(a.q) + at);
        cp_async16(&ks[buf][t * DK + c], static_cast<const T*>(a.k) + at);
      }
      for (int i = tid; i < nt * (VS / E16); i += NTHREADS) {
        const int t = i / (VS / E16), c = (i % (VS / E16)) * E16;
        cp_async16(&vs[buf][t * VS + c], static_cast<const T*>(a.v) + ((bos + t0 + t) * a.HV + hv) * DV + v0 + c);
      }
    } else {
      for (int i = tid; i < nt * DK; i += NTHREADS) {
        const int64_t at = ((bos + t0 + i / DK) * a.H + hq) * DK + i % DK;
        qs[buf][i] = static_cast<const T*>(a.q)[at];
        ks[buf][i] = static_cast<const T*>(a.k)[at];
      }
      for (int i = tid; i < nt * VS; i += NTHREADS)
        vs[buf][i] = static_cast<const T*>(a.v)[((bos + t0 + i / VS) * a.HV + hv) * DV + v0 + i % VS];
    }
    cp_async_commit();
  };
  fetch(0, 0);
  bool writeback;
  const int64_t slot = state_slot(a, n, &writeback);   // which state of the pool this sequence uses
  const int half = lane & 1, r0 = (lane >> 1) * W::RPL, cl = warp * 8 + half * 4, c0 = v0 + cl;
  W w;
  w.load(a.h0 ? a.h0 + (slot * a.HV + hv) * DK * DV : nullptr, r0, c0, DV);

  for (int t0 = 0, buf = 0; t0 < len; t0 += TB, buf ^= 1) {
    const int nt = len - t0 < TB ? len - t0 : TB;
    if (tid < nt) gate_beta(a, bos + t0 + tid, hv, sdec[tid], sbeta[tid]);
    cp_async_wait<0>();
    __syncthreads();
    if (t0 + TB < len) fetch(t0 + TB, buf ^ 1);
    // norms and <k,q>: 16 lanes per token, the same rows per lane as in the walk
    for (int t = tid >> 4; t < TB; t += NTHREADS / 16) {   // the same trip count for the lanes of a warp
      const int at = (t < nt ? t : 0) * DK + (lane & 15) * W::RPL;
      uint64_t k2[W::RP2], q2[W::RP2], s2[3] = {0ull, 0ull, 0ull};
      load_pairs<T, W::RPL>(ks[buf], at, true, k2);
      load_pairs<T, W::RPL>(qs[buf], at, true, q2);
#pragma unroll
      for (int i = 0; i < W::RP2; ++i) {
        s2[0] = fma2(k2[i], k2[i], s2[0]);
        s2[1] = fma2(q2[i], q2[i], s2[1]);
        s2[2] = fma2(k2[i], q2[i], s2[2]);
      }
      float sm[3];
#pragma unroll
      for (int e = 0; e < 3; ++e) {
        const float2 f = unpack2(s2[e]);
        sm[e] = f.x + f.y;
#pragma unroll
        for (int o = 1; o <= 8; o <<= 1) sm[e] += __shfl_xor_sync(0xffffffffu, sm[e], o);
      }
      if ((lane & 15) == 0 && t < nt) {
        const bool l2 = a.flags & B200GDN_REC_L2NORM;
        const float kn = l2 ? rsqrtf(sm[0] + 1e-6f) : 1.f, qn = l2 ? a.scale * rsqrtf(sm[1] + 1e-6f) : a.scale;
        sk_[t] = kn;
        sq_[t] = qn;
        skq[t] = sm[2] * kn * qn;
      }
    }
    __syncthreads();
    for (int t = 0; t < nt; ++t) {
      uint64_t k2[W::RP2], q2[W::RP2];
      load_pairs<T, W::RPL>(ks[buf], t * DK + r0, true, k2);
      load_pairs<T, W::RPL>(qs[buf], t * DK + r0, true, q2);
      float v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = Io<T>::ld(vs[buf], t * VS + cl + j);
      const float o = w.step(k2, q2, sk_[t], sq_[t], skq[t], sdec[t], sbeta[t], v, lane);
      if ((lane & 18) == 16) Io<T>::st(a.o, ((bos + t0 + t) * a.HV + hv) * DV + c0 + ((lane >> 2) & 3), o);
    }
    __syncthreads();   // the next block's scalars and the copies after it overwrite what was read here
  }
  if (a.ht != nullptr && writeback) w.store(a.ht + (slot * a.HV + hv) * DK * DV, r0, c0, DV);
}

// ---- several tokens per sequence: tokens in pairs ---------------------------------------------------------------------
constexpr int NT = 2;

// What a token of a pair needs besides its rows; kn k and qn q are the rows with the factors of their norms (and the scale).
struct __align__(16) PairToken {
  float k, q;          // e^g from before the pair to the token, times kn | qn
  float decay, last;   // the same alone; e^g from the token to the pair's end, times kn
  float kk;            // second token: e^g <kn k, kn k of the first>.  First: a factor of the state ahead of the pair, 1 as a rule
  float kq0, kq1;      // <qn q, kn k> with the first token's k (second token: times e^g; first: not used) and the second's
  float beta;
};

// The state of one warp: eight value channels with ALL K rows.  Lane l keeps, of channels 2 (l / 8) and + 1, the rows 32 m + 4 (l % 8)
// .. + 3 as pairs: a row of k is read once for two channels, and a reduction over the rows is three shuffles for both channels of
// S^T k and S^T q together.
template <int DK, bool VFIRST>
struct PairState {
  static constexpr int NM = DK / 32;
  uint64_t st[2 * NM][2];   // st[2 m + e][j]: rows (32 m + 4 (l % 8) + 2 e, + 1), channel c0 + j
  __device__ __forceinline__ void load(const float* h, int s, int c0, int DV) {
#pragma unroll
    for (int m = 0; m < NM; ++m) {
      const int r = 32 * m + 4 * s;
      if (h == nullptr) {
#pragma unroll
        for (int e = 0; e < 2; ++e) st[2 * m + e][0] = st[2 * m + e][1] = 0ull;
      } else if (VFIRST) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float4 x = *reinterpret_cast<const float4*>(h + (int64_t)(c0 + j) * DK + r);
          st[2 * m][j] = pack2(x.x, x.y);
          st[2 * m + 1][j] = pack2(x.z, x.w);
        }
      } else {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float2 x = *reinterpret_cast<const float2*>(h + (int64_t)(r + 2 * e) * DV + c0);
          const float2 y = *reinterpret_cast<const float2*>(h + (int64_t)(r + 2 * e + 1) * DV + c0);
          st[2 * m + e][0] = pack2(x.x, y.x);
          st[2 * m + e][1] = pack2(x.y, y.y);
        }
      }
    }
  }
  __device__ __forceinline__ void store(float* h, int s, int c0, int DV) const {
#pragma unroll
    for (int m = 0; m < NM; ++m) {
      const int r = 32 * m + 4 * s;
      if (VFIRST) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float2 x = unpack2(st[2 * m][j]), y = unpack2(st[2 * m + 1][j]);
          *reinterpret_cast<float4*>(h + (int64_t)(c0 + j) * DK + r) = make_float4(x.x, x.y, y.x, y.y);
        }
      } else {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float2 x = unpack2(st[2 * m + e][0]), y = unpack2(st[2 * m + e][1]);
          *reinterpret_cast<float2*>(h + (int64_t)(r + 2 * e) * DV + c0) = make_float2(x.x, y.x);
          *reinterpret_cast<float2*>(h + (int64_t)(r + 2 * e + 1) * DV + c0) = make_float2(x.y, y.y);
        }
      }
    }
  }
  // Two tokens.  Every reduction is taken from the state before them,
  //     r_t = beta_t (v_t - D kn_t S^T k_t - sum_{s<t} kk_ts r_s);   o_t = D qn_t S^T q_t + sum_{s<=t} kq_ts r_s;
  //     S <- D S + sum_s D(end, s) kn_s k_s r_s^T,
  // so one round of shuffles in sequence serves both.  k, q: this lane's rows of the first token in shared memory; v: the first
  // token's channel of this lane, c0 + ((lane >> 1) & 1).  o: of the same channel, right in lanes with bit 2 set.
  template <typename T>
  __device__ __forceinline__ void pair(const float* k, const float* q, const T* v, const PairToken* c, int lane, float (&o)[NT]) {
    const bool b4 = lane & 4, b2 = lane & 2;
    if (c[0].kk != 1.f) {
      const uint64_t f2 = pack2(c[0].kk, c[0].kk);
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 2 * NM; ++i) st[i][j] = mul2(st[i][j], f2);
    }
    uint64_t k2[NT][2 * NM];
    float z[NT];
#pragma unroll
    for (int u = 0; u < NT; ++u) {
      uint64_t ad[2] = {0ull, 0ull}, aq[2] = {0ull, 0ull};
#pragma unroll
      for (int m = 0; m < NM; ++m) {
        const float4 kf = *reinterpret_cast<const float4*>(k + u * DK + 32 * m), qf = *reinterpret_cast<const float4*>(q + u * DK + 32 * m);
        k2[u][2 * m] = pack2(kf.x, kf.y);
        k2[u][2 * m + 1] = pack2(kf.z, kf.w);
        const uint64_t q0 = pack2(qf.x, qf.y), q1 = pack2(qf.z, qf.w);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          ad[j] = fma2(st[2 * m][j], k2[u][2 * m], ad[j]);
          aq[j] = fma2(st[2 * m][j], q0, aq[j]);
          ad[j] = fma2(st[2 * m + 1][j], k2[u][2 * m + 1], ad[j]);
          aq[j] = fma2(st[2 * m + 1][j], q1, aq[j]);
        }
      }
      // afterwards a lane holds the sum (bit 2: 0 = S^T k, 1 = S^T q) of channel (bit 1) of its two
      float x[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float2 d = unpack2(ad[j]), e = unpack2(aq[j]);
        const float sd = d.x + d.y, sq = e.x + e.y;
        x[j] = (b4 ? sq : sd) + __shfl_xor_sync(0xffffffffu, b4 ? sd : sq, 4);
      }
      z[u] = (b2 ? x[1] : x[0]) + __shfl_xor_sync(0xffffffffu, b2 ? x[0] : x[1], 2);
      z[u] += __shfl_xor_sync(0xffffffffu, z[u], 1);
    }
    // of the lane's channel; right in the lanes that hold S^T k
    const float ra = c[0].beta * (Io<T>::ld(v, 0) - c[0].k * z[0]);
    const float rb = c[1].beta * (Io<T>::ld(v, VS) - (c[1].k * z[1] + c[1].kk * ra));
    const int k_lane = lane & 24;
    const float a0 = __shfl_sync(0xffffffffu, ra, k_lane), a1 = __shfl_sync(0xffffffffu, ra, k_lane | 2);
    const float b0 = __shfl_sync(0xffffffffu, rb, k_lane), b1 = __shfl_sync(0xffffffffu, rb, k_lane | 2);
    const uint64_t dec2 = pack2(c[1].decay, c[1].decay);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float x = (j ? a1 : a0) * c[0].last, y = (j ? b1 : b0) * c[1].last;
      const uint64_t xx = pack2(x, x), yy = pack2(y, y);
#pragma unroll
      for (int i = 0; i < 2 * NM; ++i) st[i][j] = fma2(st[i][j], dec2, fma2(k2[0][i], xx, mul2(k2[1][i], yy)));
    }
    const float oa = b2 ? a1 : a0, ob = b2 ? b1 : b0;
    o[0] = c[0].q * z[0] + c[0].kq0 * oa;
    o[1] = c[1].q * z[1] + (c[1].kq0 * oa + c[1].kq1 * ob);
  }
};

// A CTA of four warps owns 32 value channels of one (sequence, head).  q, k and v of TB tokens at a time reach shared memory as they
// are by asynchronous 16-byte copies, one block ahead (two buffers).  Half a warp then turns the q and k of a pair into fp32 and forms
// what its tokens are to one another (norms, <k,k>, <k,q>, decays; PairToken), once for the CTA, and every warp walks the block pair
// by pair without a barrier.
// Bound by issue and latency at two warps a scheduler: 220 instructions a pair and warp, half of them fma.f32x2 at two cycles, 1000
// cycles a pair, and 1900 a block for its preparation (clock stamps).  A fifth warp that prepares a block ahead took as long as the
// walk (64 tokens 22.9 us for 21.0), groups of four tokens cost more in preparation than they save (22.7 for 19.0).
// 4 sequences x 16 heads x 37 tokens, K = V = 128: 19.0 us (21.1 token by token); 1 x 16 x 64: 21.0 (26.4); 2 x 8 x 64, K = V = 64:
// 15.9 (20.5).
template <int DK, bool VFIRST, typename T>
__global__ void __launch_bounds__(NTHREADS) recurrent_pairs_kernel(const b200gdn_recurrent_args a) {
  constexpr int TB = 2048 / DK < 32 ? 2048 / DK : 32;   // tokens per block
  constexpr int E16 = 16 / (int)sizeof(T);              // elements of one 16-byte copy
  constexpr int RPL = DK / 16, RP2 = RPL / 2;           // rows of q and k per lane while pairs are prepared
  constexpr int PASS = NTHREADS / 16 * NT, NPASS = (TB + PASS - 1) / PASS;   // tokens prepared at once
  constexpr bool WIDEN = sizeof(T) == 2;
  static_assert(TB % NT == 0, "whole pairs");
  __shared__ __align__(16) T qs[2][TB * DK];
  __shared__ __align__(16) T ks[2][TB * DK];
  __shared__ __align__(16) T vs[2][TB * VS];
  __shared__ __align__(16) float qw[WIDEN ? TB * DK : 4], kw[WIDEN ? TB * DK : 4];   // the block in fp32
  __shared__ PairToken tok[TB];
  __shared__ float dots[NTHREADS / 16][8];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int v0 = blockIdx.x * VS, hv = blockIdx.y, n = blockIdx.z, hq = hv / (a.HV / a.H), DV = a.V;
  int64_t bos;
  int len;
  if (a.cu_seqlens != nullptr) {
    bos = a.cu_seqlens[n];
    len = a.cu_seqlens[n + 1] - (int)bos;
  } else {
    bos = (int64_t)n * a.T;
    len = a.T;
  }
  const bool wide = ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k) | reinterpret_cast<uintptr_t>(a.v)) & 15) == 0;
  auto fetch = [&](int t0, int buf) {
    const int nt = len - t0 < TB ? len - t0 : TB;
    if (nt & 1) {   // a last pair that is not full: a token of zeros, which changes nothing
      for (int i = tid; i < DK; i += NTHREADS) qs[buf][nt * DK + i] = ks[buf][nt * DK + i] = T(0.f);
      if (tid < VS) vs[buf][nt * VS + tid] = T(0.f);
    }
    if (wide) {
      for (int i = tid; i < nt * (DK / E16); i += NTHREADS) {
        const int t = i / (DK / E16), c = (i % (DK / E16)) * E16;
        const int64_t at = ((bos + t0 + t) * a.H + hq) * DK + c;
        cp_async16(&qs[buf][t * DK + c], static_cast<const T*>(a.q) + at);
        cp_async16(&ks[buf][t * DK + c], static_cast<const T*>(a.k) + at);
      }
      for (int i = tid; i < nt * (VS / E16); i += NTHREADS) {
        const int t = i / (VS / E16), c = (i % (VS / E16)) * E16;
        cp_async16(&vs[buf][t * VS + c], static_cast<const T*>(a.v) + ((bos + t0 + t) * a.HV + hv) * DV + v0 + c);
      }
    } else {
      for (int i = tid; i < nt * DK; i += NTHREADS) {
        const int64_t at = ((bos + t0 + i / DK) * a.H + hq) * DK + i % DK;
        qs[buf][i] = static_cast<const T*>(a.q)[at];
        ks[buf][i] = static_cast<const T*>(a.k)[at];
      }
      for (int i = tid; i < nt * VS; i += NTHREADS)
        vs[buf][i] = static_cast<const T*>(a.v)[((bos + t0 + i / VS) * a.HV + hv) * DV + v0 + i % VS];
    }
    cp_async_commit();
  };
  // g and beta of the tokens that this lane will prepare the scalars of: lanes 0 and 1 of a half-warp, one token of its pair each
  const int l16 = lane & 15, half = tid >> 4;
  float g_raw[NPASS], b_raw[NPASS];
  auto fetch_gates = [&](int t0) {
#pragma unroll
    for (int p = 0; p < NPASS; ++p) {
      const int t = t0 + p * PASS + half * NT + l16;
      if (l16 < NT && p * PASS + half * NT < TB && t < len) load_gate_beta(a, bos + t, hv, g_raw[p], b_raw[p]);
    }
  };
  const bool gate = a.flags & B200GDN_REC_GATE, l2 = a.flags & B200GDN_REC_L2NORM;
  float A_log = 0.f, dt_bias = 0.f;
  if (gate && l16 < NT) {
    A_log = a.A_log[hv];
    if (a.dt_bias) dt_bias = a.dt_bias[hv];
  }
  fetch_gates(0);
  fetch(0, 0);
  bool writeback;
  const int64_t slot = state_slot(a, n, &writeback);   // which state of the pool this sequence uses
  const int s = lane & 7, cl = warp * 8 + (lane >> 3) * 2, c0 = v0 + cl, ch = (lane >> 1) & 1;
  PairState<DK, VFIRST> w;
  w.load(a.h0 ? a.h0 + (slot * a.HV + hv) * DK * DV : nullptr, s, c0, DV);

  for (int t0 = 0, buf = 0; t0 < len; t0 += TB, buf ^= 1) {
    const int nt = len - t0 < TB ? len - t0 : TB;
    cp_async_wait<0>();
    __syncthreads();   // ... and every warp has walked the block before
    if (t0 + TB < len) fetch(t0 + TB, buf ^ 1);
#pragma unroll
    for (int p = 0; p < NPASS; ++p) {
      const int t = p * PASS + half * NT;   // this half-warp's pair
      if (p * PASS + (half & ~1) * NT >= nt) break;   // (the same for both halves)
      const bool live = t < nt;
      uint64_t k[NT][RP2], q[NT][RP2];
#pragma unroll
      for (int u = 0; u < NT; ++u) {
        const int at = (live ? t + u : u) * DK + l16 * RPL;
        load_pairs<T, RPL>(ks[buf], at, true, k[u]);
        load_pairs<T, RPL>(qs[buf], at, true, q[u]);
        if (WIDEN && live) {
#pragma unroll
          for (int i = 0; i < RP2; ++i) {
            *reinterpret_cast<uint64_t*>(&kw[at + 2 * i]) = k[u][i];
            *reinterpret_cast<uint64_t*>(&qw[at + 2 * i]) = q[u][i];
          }
        }
      }
      uint64_t x2[8] = {};
#pragma unroll
      for (int i = 0; i < RP2; ++i) {
        x2[0] = fma2(k[0][i], k[0][i], x2[0]);
        x2[1] = fma2(k[1][i], k[1][i], x2[1]);
        x2[2] = fma2(q[0][i], q[0][i], x2[2]);
        x2[3] = fma2(q[1][i], q[1][i], x2[3]);
        x2[4] = fma2(k[1][i], k[0][i], x2[4]);
        x2[5] = fma2(q[0][i], k[0][i], x2[5]);
        x2[6] = fma2(q[1][i], k[0][i], x2[6]);
        x2[7] = fma2(q[1][i], k[1][i], x2[7]);
      }
      float x[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float2 f = unpack2(x2[e]);
        x[e] = f.x + f.y;
      }
      // summed over the sixteen lanes by recursive halving: lane l ends with value l / 2
#pragma unroll
      for (int h = 4; h > 0; h >>= 1)
#pragma unroll
        for (int e = 0; e < h; ++e)
          x[e] = (l16 & 2 * h ? x[e + h] : x[e]) + __shfl_xor_sync(0xffffffffu, l16 & 2 * h ? x[e] : x[e + h], 2 * h);
      x[0] += __shfl_xor_sync(0xffffffffu, x[0], 1);
      if (!(l16 & 1)) dots[half][l16 >> 1] = x[0];
      __syncwarp();
      float dec = 1.f, beta = 0.f;   // (a token past the end)
      if (l16 < NT && t + l16 < nt) activate(a, [&](float x) { return -expf(A_log) * softplus_f(x + dt_bias); }, g_raw[p], b_raw[p], dec, beta);
      const float other = __shfl_xor_sync(0xffffffffu, dec, 1);   // of the pair's other token
      if (l16 < NT && live) {
        const float* d = dots[half];
        const float kn0 = l2 ? rsqrtf(d[0] + 1e-6f) : 1.f, kn1 = l2 ? rsqrtf(d[1] + 1e-6f) : 1.f;
        const float qn = l2 ? a.scale * rsqrtf(d[2 + l16] + 1e-6f) : a.scale;
        PairToken g;
        // the state takes the first token's e^g ahead of the pair where the two together are out of fp32's range (zero times an
        // overflowed product is not zero, a large state times one that vanished is not either)
        const float both = dec * other, ahead = both >= 1.17549435e-38f && both < INFINITY ? 1.f : l16 ? other : dec;
        g.decay = ahead == 1.f ? (l16 ? both : dec) : l16 ? dec : 1.f;
        g.k = g.decay * (l16 ? kn1 : kn0);
        g.q = g.decay * qn;
        g.last = l16 ? kn1 : other * kn0;
        g.kk = l16 ? dec * d[4] * kn0 * kn1 : ahead;
        g.kq0 = (l16 ? dec * d[6] : d[5]) * kn0 * qn;
        g.kq1 = d[7] * kn1 * qn;
        g.beta = beta;
        tok[t + l16] = g;
      }
      __syncwarp();   // the next pass writes `dots` again
    }
    __syncthreads();
    fetch_gates(t0 + TB);
    const float* kf = reinterpret_cast<const float*>(WIDEN ? static_cast<const void*>(kw) : ks[buf]);
    const float* qf = reinterpret_cast<const float*>(WIDEN ? static_cast<const void*>(qw) : qs[buf]);
    T* out = static_cast<T*>(a.o) + ((bos + t0) * a.HV + hv) * DV + c0 + ch;
    for (int t = 0; t < nt; t += NT) {
      float o[NT];
      w.template pair<T>(kf + t * DK + 4 * s, qf + t * DK + 4 * s, &vs[buf][t * VS + cl + ch], &tok[t], lane, o);
      if ((lane & 5) == 4) {
        Io<T>::st(out, 0, o[0]);
        if (t + 1 < nt) Io<T>::st(out, (int64_t)a.HV * DV, o[1]);
      }
      out += (int64_t)NT * a.HV * DV;
    }
  }
  if (a.ht != nullptr && writeback) w.store(a.ht + (slot * a.HV + hv) * DK * DV, s, c0, DV);
}

// Single-token decode at large batch as a stream: the step kernel loads a state, computes and stores it, so the memory pipe
// of an SM idles while its CTAs compute.  Here one persistent CTA per SM walks its (sequence, head) items through a ring of
// states in shared memory: a mover thread brings and takes away each 64 KiB state (one contiguous bulk copy each way), three
// warps prepare the tokens (q and k as fp32 with their norms' factors, v, the activated gate scalars) for the same ring, and
// eight consumer warps only compute, shared memory to shared memory.  Bound by HBM (one read and one write of every state).
// 256 sequences x 16 heads, K = V = 128: 91 us, 5.9 TB/s (100 with the tokens fetched and the gates activated by the thread that
// moves the states).  New states stored from registers instead, which leaves the ring to the reads: 92.  Every wait is bounded.
__device__ int g_decode_timeout = 0;

constexpr int kTokenWarps = 3;
template <int DK, int DV>
struct DecodeSmem {
  static constexpr size_t state_bytes = (size_t)DK * DV * 4;
  static constexpr int NS = (int)(192 * 1024 / state_bytes);   // 3 (128 x 128) to 12 (64 x 64) states in the ring
  static constexpr size_t o_k = state_bytes, o_q = o_k + DK * 4, o_v = o_q + DK * 4, o_sc = o_v + DV * 4;
  static constexpr size_t stage = o_sc + 128;
  static constexpr size_t o_red = NS * stage;
  static constexpr size_t red_bytes = 8 * 2 * DV * 4;   // one item's partial sums
  static constexpr size_t o_bar = o_red + 2 * red_bytes;
  static constexpr size_t bytes = o_bar + 2 * NS * 8;
  static_assert(NS < 32 && bytes <= 227 * 1024, "the ring fits, and the mover's block of slots covers it");
  // a token warp's next item is at most one turn of the ring on: its wait for the stage then never sees a phase two back
  static_assert(kTokenWarps <= NS, "one phase of `freed` at a time");
};
constexpr int kStreamThreads = 32 * (8 + 1 + kTokenWarps);   // consumers, mover, token warps

template <int DK, int DV, typename T>
__global__ void __launch_bounds__(kStreamThreads, 1) decode_stream_kernel(const b200gdn_recurrent_args a, const int n_items) {
  using S = DecodeSmem<DK, DV>;
  constexpr int NS = S::NS;
  constexpr int LPR = DV / 4, RPI = 32 / LPR, RW = DK / 8 / RPI;   // lanes to a row, rows to a warp instruction, rows per lane
  extern __shared__ __align__(128) unsigned char dsm[];
  uint64_t* full = reinterpret_cast<uint64_t*>(dsm + S::o_bar);
  uint64_t* freed = full + NS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n_local = (n_items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int G = a.HV / a.H;

  if (tid == 0) {
    for (int s = 0; s < NS; ++s) {
      tc5::mbar_init(&full[s], 2);    // the state and the token
      tc5::mbar_init(&freed[s], 8);   // the consumer warps
    }
    tc5::fence_mbar_init();
  }
  __syncthreads();

  if (warp == 8) {
    // ---- mover: write-back of the item that used the stage last, then the load of the next one.  The states' places are
    // looked up 32 items at a time (a look-up per item would be a memory latency in this thread's chain).
    int64_t cur = 0, prev = 0;
    bool cur_wb = false, prev_wb = false;
    for (int j = 0; j < n_local + NS; ++j) {
      const int s = j % NS, i = j - NS;
      if (j % 32 == 0) {
        prev = cur;
        prev_wb = cur_wb;
        const int item = (int)blockIdx.x + (j + lane) * (int)gridDim.x;
        if (j + lane < n_local) cur = (state_slot(a, item / a.HV, &cur_wb) * a.HV + item % a.HV) * DK * DV;
      }
      const bool same = i / 32 == j / 32;
      const int64_t at_out = __shfl_sync(0xffffffffu, same ? cur : prev, i & 31), at_in = __shfl_sync(0xffffffffu, cur, j & 31);
      const bool writeback = __shfl_sync(0xffffffffu, (int)(same ? cur_wb : prev_wb), i & 31);
      if (i >= 0 && i < n_local) {
        if (!tc5::mbar_wait_warp(&freed[s], (i / NS) & 1)) {
          if (lane == 0) {
            atomicExch(&g_decode_timeout, 1);
            for (int l = i; l < min(j, n_local); ++l) tc5::mbar_wait(&full[l % NS], (l / NS) & 1);   // copies on their way land first
          }
          break;
        }
        if (writeback && lane == 0) {
          asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(a.ht + at_out),
                       "r"(tc5::smem_addr(dsm + (size_t)s * S::stage)), "r"((uint32_t)S::state_bytes)
                       : "memory");
          tma::store_commit();
        }
      }
      if (j < n_local && lane == 0) {
        tma::store_wait_read<0>();   // the stage may be refilled once the copy has read it
        tc5::mbar_expect_tx(&full[s], (uint32_t)S::state_bytes);
        tma::load_1d(dsm + (size_t)s * S::stage, a.h0 + at_in, (uint32_t)S::state_bytes, &full[s]);
      }
    }
    if (lane == 0) tma::store_wait_all<0>();
    return;
  }
  if (warp > 8) {
    // ---- token warps, in turn: k, scale q (with the L2-norm factors), v, decay, beta, <k, q>
    for (int j = warp - 9; j < n_local; j += kTokenWarps) {
      const int s = j % NS, item = (int)blockIdx.x + j * (int)gridDim.x;
      const int n = item / a.HV, hv = item % a.HV, hq = hv / G;
      float k[DK / 32], q[DK / 32], v[DV / 32], dec, beta;
      const int64_t qk_at = ((int64_t)n * a.H + hq) * DK + lane, v_at = ((int64_t)n * a.HV + hv) * DV + lane;
#pragma unroll
      for (int i = 0; i < DK / 32; ++i) {
        k[i] = Io<T>::ld(a.k, qk_at + 32 * i);
        q[i] = Io<T>::ld(a.q, qk_at + 32 * i);
      }
#pragma unroll
      for (int i = 0; i < DV / 32; ++i) v[i] = Io<T>::ld(a.v, v_at + 32 * i);
      gate_beta(a, n, hv, dec, beta);
      float kk = 0.f, qq = 0.f, kq = 0.f;
#pragma unroll
      for (int i = 0; i < DK / 32; ++i) {
        kk += k[i] * k[i];
        qq += q[i] * q[i];
        kq += k[i] * q[i];
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        kk += __shfl_xor_sync(0xffffffffu, kk, o);
        qq += __shfl_xor_sync(0xffffffffu, qq, o);
        kq += __shfl_xor_sync(0xffffffffu, kq, o);
      }
      float kn = 1.f, qn = a.scale;
      if (a.flags & B200GDN_REC_L2NORM) {
        kn = rsqrtf(kk + 1e-6f);
        qn *= rsqrtf(qq + 1e-6f);
      }
      if (j >= NS && !tc5::mbar_wait(&freed[s], ((j / NS) - 1) & 1)) {
        atomicExch(&g_decode_timeout, 1);
        return;
      }
      unsigned char* stg = dsm + (size_t)s * S::stage;
      float *sk = reinterpret_cast<float*>(stg + S::o_k), *sq = reinterpret_cast<float*>(stg + S::o_q);
      float *sv = reinterpret_cast<float*>(stg + S::o_v), *sc = reinterpret_cast<float*>(stg + S::o_sc);
#pragma unroll
      for (int i = 0; i < DK / 32; ++i) {
        sk[lane + 32 * i] = k[i] * kn;
        sq[lane + 32 * i] = q[i] * qn;
      }
#pragma unroll
      for (int i = 0; i < DV / 32; ++i) sv[lane + 32 * i] = v[i];
      if (lane == 0) *reinterpret_cast<float4*>(sc) = make_float4(dec, beta, kq * kn * qn, 0.f);
      __syncwarp();
      if (lane == 0) tc5::mbar_arrive(&full[s]);
    }
    return;
  }

  // ---- consumers: warp w keeps rows [w DK/8, (w+1) DK/8), a lane four columns of every row (128 columns) or of every other
  // one.  As in the step kernel both row reductions are taken from the state before its update, so that one barrier per item
  // serves both.
  const int col = 4 * (lane % LPR), r0 = warp * (DK / 8) + (lane / LPR) * RW;
  for (int j = 0; j < n_local; ++j) {
    const int s = j % NS, item = (int)blockIdx.x + j * (int)gridDim.x;
    unsigned char* stg = dsm + (size_t)s * S::stage;
    float* St = reinterpret_cast<float*>(stg) + r0 * DV + col;
    float (*red)[2][DV] = reinterpret_cast<float (*)[2][DV]>(dsm + S::o_red + (j & 1) * S::red_bytes);
    const uint32_t bad = tc5::mbar_wait(&full[s], (j / NS) & 1) ? 0u : 1u;
    uint64_t st[RW][2], k2[RW], d[2] = {0ull, 0ull}, e[2] = {0ull, 0ull};
#pragma unroll
    for (int i = 0; i < RW; i += 4) {
      const float4 kf = *reinterpret_cast<const float4*>(stg + S::o_k + (r0 + i) * 4);
      const float4 qf = *reinterpret_cast<const float4*>(stg + S::o_q + (r0 + i) * 4);
      const float kv[4] = {kf.x, kf.y, kf.z, kf.w}, qv[4] = {qf.x, qf.y, qf.z, qf.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float4 x = *reinterpret_cast<const float4*>(St + (i + u) * DV);
        st[i + u][0] = pack2(x.x, x.y);
        st[i + u][1] = pack2(x.z, x.w);
        k2[i + u] = pack2(kv[u], kv[u]);
        const uint64_t q2 = pack2(qv[u], qv[u]);
        d[0] = fma2(st[i + u][0], k2[i + u], d[0]);
        d[1] = fma2(st[i + u][1], k2[i + u], d[1]);
        e[0] = fma2(st[i + u][0], q2, e[0]);
        e[1] = fma2(st[i + u][1], q2, e[1]);
      }
    }
    const float4 v = *reinterpret_cast<const float4*>(stg + S::o_v + col * 4);
    const float4 sc = *reinterpret_cast<const float4*>(stg + S::o_sc);   // decay, beta, <k, q>
    {
      const float2 d0 = unpack2(d[0]), d1 = unpack2(d[1]), e0 = unpack2(e[0]), e1 = unpack2(e[1]);
      float4 dv = make_float4(d0.x, d0.y, d1.x, d1.y), ev = make_float4(e0.x, e0.y, e1.x, e1.y);
      if constexpr (RPI == 2) {   // the warp's two rows
        dv.x += __shfl_xor_sync(0xffffffffu, dv.x, 16); dv.y += __shfl_xor_sync(0xffffffffu, dv.y, 16);
        dv.z += __shfl_xor_sync(0xffffffffu, dv.z, 16); dv.w += __shfl_xor_sync(0xffffffffu, dv.w, 16);
        ev.x += __shfl_xor_sync(0xffffffffu, ev.x, 16); ev.y += __shfl_xor_sync(0xffffffffu, ev.y, 16);
        ev.z += __shfl_xor_sync(0xffffffffu, ev.z, 16); ev.w += __shfl_xor_sync(0xffffffffu, ev.w, 16);
      }
      if (lane < LPR) {
        *reinterpret_cast<float4*>(&red[warp][0][col]) = dv;
        *reinterpret_cast<float4*>(&red[warp][1][col]) = ev;
      }
    }
    {
      // the partial sums are complete; the same barrier carries the outcome of the bounded wait, so that all leave together
      // (the loader and the token warps then give up on their own bounded waits)
      uint32_t any_bad;
      asm volatile(
          "{\n.reg .pred p, q;\nsetp.ne.b32 q, %1, 0;\nbar.red.or.pred p, 1, 256, q;\nselp.u32 %0, 1, 0, p;\n}\n"
          : "=r"(any_bad)
          : "r"(bad)
          : "memory");
      if (any_bad) {
        if (tid == 0) atomicExch(&g_decode_timeout, 1);
        return;
      }
    }
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const float4 x = *reinterpret_cast<const float4*>(&red[w][0][col]);
      r.x += x.x; r.y += x.y; r.z += x.z; r.w += x.w;
    }
    r.x = sc.y * (v.x - sc.x * r.x); r.y = sc.y * (v.y - sc.x * r.y);
    r.z = sc.y * (v.z - sc.x * r.z); r.w = sc.y * (v.w - sc.x * r.w);
    const uint64_t dec2 = pack2(sc.x, sc.x), rl = pack2(r.x, r.y), rh = pack2(r.z, r.w);
#pragma unroll
    for (int i = 0; i < RW; ++i) {
      const float2 lo = unpack2(fma2(k2[i], rl, mul2(st[i][0], dec2))), hi = unpack2(fma2(k2[i], rh, mul2(st[i][1], dec2)));
      *reinterpret_cast<float4*>(St + i * DV) = make_float4(lo.x, lo.y, hi.x, hi.y);
    }
    tc5::fence_async_smem();   // the new state is read by the mover's bulk copy
    __syncwarp();
    if (lane == 0) tc5::mbar_arrive(&freed[s]);
    if (warp == (j & 7) && lane < LPR) {   // the output row, by the warps in turn
      float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        const float4 x = *reinterpret_cast<const float4*>(&red[w][1][col]);
        o.x += x.x; o.y += x.y; o.z += x.z; o.w += x.w;
      }
      const int64_t at = (int64_t)item * DV + col;   // [sequence][head][V]
      Io<T>::st(a.o, at, sc.x * o.x + sc.z * r.x);
      Io<T>::st(a.o, at + 1, sc.x * o.y + sc.z * r.y);
      Io<T>::st(a.o, at + 2, sc.x * o.z + sc.z * r.z);
      Io<T>::st(a.o, at + 3, sc.x * o.w + sc.z * r.w);
    }
  }
}

// Elements of all states together (16 MiB) from which a single-token step streams them.  Measured, step kernel against stream:
// K = V = 128, 256 pairs 10.8 / 10.0 us, 512 pairs 18.0 / 15.8, 4096 pairs 106 / 91; K = V = 64, 512 pairs 7.2 / 8.2, 1024 pairs
// 12.0 / 11.7, 4096 pairs 37 / 32.
constexpr int64_t kStreamElements = 256 * 128 * 128;

template <int DK>
int launch(const b200gdn_recurrent_args& a, cudaStream_t st) {
  if constexpr (DK == 64 || DK == 128) {
    // one token per sequence at large batch: the streaming kernel (16-byte boundaries, [K,V] states, V = 64 or 128)
    if (!(a.flags & B200GDN_REC_STATE_V_FIRST) && (a.V == 64 || a.V == 128) && a.T == 1 && a.cu_seqlens == nullptr &&
        a.h0 != nullptr && a.ht != nullptr && (int64_t)a.n_seq * a.HV * DK * a.V >= kStreamElements &&
        (reinterpret_cast<uintptr_t>(a.h0) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.ht) & 15) == 0) {
      const int n_items = a.n_seq * a.HV, sms = sm_count();
      auto stream = [&](auto* kernel, size_t bytes) -> int {
        if (int e = ensure_smem(kernel, bytes)) return e;
        kernel<<<n_items < sms ? n_items : sms, kStreamThreads, bytes, st>>>(a, n_items);
        return 0;
      };
      int e;
#define STREAM(TY) e = a.V == 64 ? stream(decode_stream_kernel<DK, 64, TY>, DecodeSmem<DK, 64>::bytes) \
                                 : stream(decode_stream_kernel<DK, 128, TY>, DecodeSmem<DK, 128>::bytes)
      switch (a.qkv_dtype) {
        case 0: STREAM(__nv_bfloat16); break;
        case 1: STREAM(__half); break;
        default: STREAM(float); break;
      }
#undef STREAM
      if (e) return e;
      return check_launch("decode_stream");
    }
  }
  dim3 grid(a.V / VS, a.HV, a.n_seq);
  const bool vf = a.flags & B200GDN_REC_STATE_V_FIRST;
  const bool step = a.T == 1 && a.cu_seqlens == nullptr;   // one token per sequence: no block of tokens to stage
  // Tokens per sequence (on average) from which they are taken in pairs.  Measured, one by one / in pairs, K = V = 128 bf16: 1 x 16
  // heads, 8 tokens 6.2 / 6.3 us, 12 tokens 7.4 / 7.1, 24 tokens 12.1 / 10.6; 16 x 32 heads (2048 CTAs), 16 tokens 46.7 / 48.9, 24
  // tokens 66.9 / 64.8, 64 tokens 158 / 139 (fp32: 33 tokens 89.8 / 91.8, 64 tokens 156 / 147); K = V = 64: 8 tokens 5.7 / 5.0 and
  // 13.1 / 13.6, 12 tokens 6.7 / 5.6 and 16.4 / 15.7.  [V,K] states gain more, at every K (K = V = 256, 4 x 16 heads, 12 tokens: 29.0 /
  // 20.9; K = 32: a quarter).  K = 256 with [K,V] states starts late, its registers leave fewer CTAs per SM and a state comes in words
  // of 8 bytes: 4 x 16 heads, V = 256, 12 tokens 21.4 / 28.3 us in bf16 and 22.6 / 27.4 in fp32, 64 tokens 80.0 / 90.9 and 85.2 / 86.8;
  // V = 128 (256 CTAs) 64 tokens 47.2 / 48.9 and 51.6 / 46.4, 24 tokens in fp32 22.3 / 21.7; 1 x 16 heads (128 CTAs) 40 tokens in
  // bf16 24.4 / 24.7, 64 tokens 36.8 / 36.3, in fp32 16 tokens 12.3 / 12.2, 24 tokens 16.6 / 15.5.
  const int tokens = a.T / (a.cu_seqlens != nullptr && a.n_seq > 0 ? a.n_seq : 1);
  const int64_t ctas = (int64_t)grid.x * grid.y * grid.z, sms = sm_count();
  const bool fp32 = a.qkv_dtype != 0 && a.qkv_dtype != 1;
  const bool pairs = DK == 256 && !vf ? tokens >= (fp32 ? 24 : 64) && ctas <= (fp32 ? 2 : 1) * sms
                                      : tokens >= (DK >= 128 && ctas > 4 * sms ? 40 : 12);
  auto run = [&](auto* one, auto* few, auto* many) { (step ? one : pairs ? many : few)<<<grid, NTHREADS, 0, st>>>(a); };
#define RUN(VF, TY) run(recurrent_step_kernel<DK, VF, TY>, recurrent_few_kernel<DK, VF, TY>, recurrent_pairs_kernel<DK, VF, TY>)
  switch (a.qkv_dtype) {
    case 0: if (vf) RUN(true, __nv_bfloat16); else RUN(false, __nv_bfloat16); break;
    case 1: if (vf) RUN(true, __half); else RUN(false, __half); break;
    default: if (vf) RUN(true, float); else RUN(false, float); break;
  }
#undef RUN
  return check_launch("recurrent");
}

}  // namespace

int launch_recurrent(const b200gdn_recurrent_args& a, cudaStream_t st) {
  if (a.V % VS != 0) return set_error(B200GDN_ERR_UNSUPPORTED, "recurrent: V=%d must be a multiple of %d", a.V, VS);
  if ((a.flags & B200GDN_REC_GATE) && a.A_log == nullptr)
    return set_error(B200GDN_ERR_BAD_ARGUMENT, "recurrent: the in-kernel gate needs A_log");
  if (((reinterpret_cast<uintptr_t>(a.h0) | reinterpret_cast<uintptr_t>(a.ht)) & 15) != 0)
    return set_error(B200GDN_ERR_BAD_ARGUMENT, "recurrent: the states must start on a 16-byte boundary");
  switch (a.K) {
    case 32: return launch<32>(a, st);
    case 64: return launch<64>(a, st);
    case 128: return launch<128>(a, st);
    case 256: return launch<256>(a, st);
  }
  return set_error(B200GDN_ERR_UNSUPPORTED, "recurrent: K=%d not built (32, 64, 128, 256 are)", a.K);
}

// Reads and clears the flag a bounded device wait raises when it expires (synchronises with the device).
int decode_timeout_flag() {
  int v = 0, zero = 0;
  cudaMemcpyFromSymbol(&v, g_decode_timeout, sizeof(int));
  if (v) cudaMemcpyToSymbol(g_decode_timeout, &zero, sizeof(int));
  return v;
}

}  // namespace gdn
