// Token-by-token gated delta rule (decode and short prefill), forward only:
//     S *= exp(g);  r = beta (v - S^T k);  S += k r^T;  o = S^T (scale q)
// Replaces fused_recurrent_gated_delta_rule_fwd_kernel (fla/ops/gated_delta_rule/fused_recurrent.py:30-181),
// including its in-kernel options (q/k L2 norm, -exp(A_log) softplus(g + dt_bias) gate, sigmoid beta,
// V-first state layout).  fp32 arithmetic throughout.  Three kernels:
//   recurrent_step_kernel   one token per sequence, small and middling batches: latency of one pass over the state
//   decode_stream_kernel    one token per sequence, large batches: pure state traffic (read + write K*V fp32)
//   recurrent_kernel        several tokens per sequence: latency of the per-token chain
#include "gdn_common.cuh"
#include "rowio.cuh"
#include "tc5.cuh"
#include "tma.cuh"

namespace gdn {
namespace {

constexpr int NTHREADS = 128;
constexpr int VS = 32;  // value channels per CTA

__device__ __forceinline__ float ld_elem(const void* p, int64_t i, int dtype) {
  if (dtype == 0) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
  if (dtype == 1) return __half2float(reinterpret_cast<const __half*>(p)[i]);
  return reinterpret_cast<const float*>(p)[i];
}
__device__ __forceinline__ void st_elem(void* p, int64_t i, int dtype, float x) {
  if (dtype == 0) reinterpret_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16(x);
  else if (dtype == 1) reinterpret_cast<__half*>(p)[i] = __float2half(x);
  else reinterpret_cast<float*>(p)[i] = x;
}
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
__device__ __forceinline__ void gate_beta(const b200gdn_recurrent_args& a, int64_t row, int hv, float& dec, float& beta) {
  float gg = a.g ? ld_param(a.g, row * a.HV + hv, a.gb_dtype) : 0.f;
  float bb = ld_param(a.beta, row * a.HV + hv, a.gb_dtype);
  if (a.flags & B200GDN_REC_GATE) {
    if (a.dt_bias) gg += a.dt_bias[hv];
    gg = -expf(a.A_log[hv]) * softplus_f(gg);
  }
  if (a.flags & B200GDN_REC_BETA_SIGMOID) {
    bb = 1.f / (1.f + expf(-bb));
    if (a.flags & B200GDN_REC_NEG_EIGVAL) bb *= 2.f;
  }
  dec = expf(gg);
  beta = bb;
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

// Several tokens per sequence: a CTA of four warps owns 32 value channels of one (sequence, head).  q, k and v of TB tokens
// at a time reach shared memory as they are by asynchronous 16-byte copies, one block ahead (two buffers); the norms,
// <k,q>, e^g and beta of a block are formed once by the CTA; then every warp walks the block without a barrier.
// Bound by the latency of the per-token chain (K/32 multiply-adds, five shuffles in sequence, K/32 multiply-adds), about
// 0.26 us a token at K = 64 and 0.45 at K = 128.  4 sequences x 16 heads x 37 tokens, K = V = 128: 20.3 us (77.5 with the
// channels combined through shared memory, five barriers a token); 128 x 16 x 4: 75.8 (110.6).
template <int DK, bool VFIRST, typename T>
__global__ void __launch_bounds__(NTHREADS) recurrent_kernel(const b200gdn_recurrent_args a) {
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

// Single-token decode at large batch as a stream: the kernels above load a state, compute and store it, so the
// memory pipe of an SM idles while its CTAs compute.  Here one persistent CTA per SM walks its (sequence, head) items
// through a three-stage ring in shared memory: a producer warp brings each 64 KiB state (one contiguous bulk copy), the
// token's q, k, v rows and the activated gate scalars two items ahead and writes finished states back (one bulk copy);
// eight consumer warps only compute, shared memory to shared memory.  Every wait is bounded.
__device__ int g_decode_timeout = 0;

template <int DK>
struct DecodeSmem {
  static constexpr int NS = 3;
  static constexpr size_t state_bytes = (size_t)DK * 128 * 4;
  static constexpr size_t o_q = state_bytes, o_k = o_q + 512, o_v = o_k + 512, o_sc = o_v + 512;
  static constexpr size_t stage = o_sc + 128;
  static constexpr size_t o_red = NS * stage;
  static constexpr size_t o_bar = o_red + 8 * 128 * 4;
  static constexpr size_t bytes = o_bar + 128;
};

template <int DK>
__global__ void __launch_bounds__(288, 1) decode_stream_kernel(const b200gdn_recurrent_args a, const int n_items) {
  using S = DecodeSmem<DK>;
  constexpr int NS = S::NS, DV = 128, RW = DK / 8;
  extern __shared__ __align__(128) unsigned char dsm[];
  float (*red)[DV] = reinterpret_cast<float (*)[DV]>(dsm + S::o_red);
  uint64_t* full = reinterpret_cast<uint64_t*>(dsm + S::o_bar);
  uint64_t* done = full + NS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int esz = a.qkv_dtype == 2 ? 4 : 2;
  const int n_local = (n_items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int G = a.HV / a.H;

  if (tid == 0) {
    for (int s = 0; s < NS; ++s) {
      tc5::mbar_init(&full[s], 1);
      tc5::mbar_init(&done[s], 256);
    }
    tc5::fence_mbar_init();
  }
  __syncthreads();

  if (warp == 8) {
    // ---- producer: write-back of the item that used the stage last, then the load of the item NS further on
    if (lane == 0) {
      bool failed = false;
      for (int jj = 0; jj < n_local + NS && !failed; ++jj) {
        const int s = jj % NS;
        unsigned char* stg = dsm + (size_t)s * S::stage;
        if (jj >= NS) {
          const int item = (int)blockIdx.x + (jj - NS) * (int)gridDim.x;
          if (!tc5::mbar_wait(&done[s], ((jj - NS) / NS) & 1)) { failed = true; break; }
          bool writeback;
          const int64_t slot = state_slot(a, item / a.HV, &writeback);
          if (writeback) {
            float* ht = a.ht + (slot * a.HV + item % a.HV) * DK * DV;
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(ht), "r"(tc5::smem_addr(stg)),
                         "r"((uint32_t)S::state_bytes)
                         : "memory");
            tma::store_commit();
            tma::store_wait_read<0>();   // the stage may be refilled once the copy has read it
          }
        }
        if (jj < n_local) {
          const int item = (int)blockIdx.x + jj * (int)gridDim.x;
          const int n = item / a.HV, hv = item % a.HV, hq = hv / G;
          const int64_t row = n;   // one token per sequence
          float gg = a.g ? ld_param(a.g, row * a.HV + hv, a.gb_dtype) : 0.f;
          if (a.flags & B200GDN_REC_GATE) {
            if (a.dt_bias) gg += a.dt_bias[hv];
            gg = -expf(a.A_log[hv]) * softplus_f(gg);
          }
          float bb = ld_param(a.beta, row * a.HV + hv, a.gb_dtype);
          if (a.flags & B200GDN_REC_BETA_SIGMOID) {
            bb = 1.f / (1.f + expf(-bb));
            if (a.flags & B200GDN_REC_NEG_EIGVAL) bb *= 2.f;
          }
          float* sc = reinterpret_cast<float*>(stg + S::o_sc);
          sc[0] = expf(gg);
          sc[1] = bb;
          const uint32_t qk_bytes = (uint32_t)(DK * esz), v_bytes = (uint32_t)(DV * esz);
          tc5::mbar_expect_tx(&full[s], (uint32_t)S::state_bytes + 2 * qk_bytes + v_bytes);
          bool writeback_unused;
          const int64_t slot = state_slot(a, n, &writeback_unused);
          tma::load_1d(stg, a.h0 + (slot * a.HV + hv) * DK * DV, (uint32_t)S::state_bytes, &full[s]);
          tma::load_1d(stg + S::o_q, static_cast<const char*>(a.q) + (row * a.H + hq) * DK * esz, qk_bytes, &full[s]);
          tma::load_1d(stg + S::o_k, static_cast<const char*>(a.k) + (row * a.H + hq) * DK * esz, qk_bytes, &full[s]);
          tma::load_1d(stg + S::o_v, static_cast<const char*>(a.v) + (row * a.HV + hv) * DV * esz, v_bytes, &full[s]);
        }
      }
      tma::store_wait_all<0>();
      if (failed) atomicExch(&g_decode_timeout, 1);
    }
    return;
  }

  // ---- consumers (8 warps): warp w keeps rows [w RW, (w+1) RW), lane l the columns 4 l .. 4 l + 3
  const int col = 4 * lane, r0 = warp * RW;
  auto sync_consumers = [] { asm volatile("bar.sync 1, 256;\n" ::: "memory"); };
  for (int j = 0; j < n_local; ++j) {
    const int s = j % NS;
    unsigned char* stg = dsm + (size_t)s * S::stage;
    float* St = reinterpret_cast<float*>(stg);
    const int item = (int)blockIdx.x + j * (int)gridDim.x;
    const int hv = item % a.HV;
    {
      // the consumers agree on the outcome of the bounded wait (a barrier-wide OR), so that they leave together;
      // the producer then gives up on its own bounded wait
      const uint32_t bad = tc5::mbar_wait(&full[s], (j / NS) & 1) ? 0u : 1u;
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
    const float* sc = reinterpret_cast<const float*>(stg + S::o_sc);
    const float decay = sc[0], beta = sc[1];
    float qn = a.scale, kn = 1.f;
    if (a.flags & B200GDN_REC_L2NORM) {
      float sq = 0.f, sk = 0.f;
      for (int i = lane; i < DK; i += 32) {
        const float x = ld_elem(stg + S::o_q, i, a.qkv_dtype), y = ld_elem(stg + S::o_k, i, a.qkv_dtype);
        sq += x * x;
        sk += y * y;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        sq += __shfl_xor_sync(0xffffffffu, sq, o);
        sk += __shfl_xor_sync(0xffffffffu, sk, o);
      }
      qn = a.scale * rsqrtf(sq + 1e-6f);
      kn = rsqrtf(sk + 1e-6f);
    }
    float4 st[RW];
    float kr[RW];
    float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < RW; ++i) {
      st[i] = *reinterpret_cast<const float4*>(St + (r0 + i) * DV + col);
      kr[i] = ld_elem(stg + S::o_k, r0 + i, a.qkv_dtype) * kn;
      st[i].x *= decay; st[i].y *= decay; st[i].z *= decay; st[i].w *= decay;
      d.x += st[i].x * kr[i]; d.y += st[i].y * kr[i]; d.z += st[i].z * kr[i]; d.w += st[i].w * kr[i];
    }
    *reinterpret_cast<float4*>(&red[warp][col]) = d;
    sync_consumers();
    float4 r;
    {
      float4 sum = *reinterpret_cast<const float4*>(&red[0][col]);
#pragma unroll
      for (int w = 1; w < 8; ++w) {
        const float4 x = *reinterpret_cast<const float4*>(&red[w][col]);
        sum.x += x.x; sum.y += x.y; sum.z += x.z; sum.w += x.w;
      }
      const float v0 = ld_elem(stg + S::o_v, col, a.qkv_dtype), v1 = ld_elem(stg + S::o_v, col + 1, a.qkv_dtype);
      const float v2 = ld_elem(stg + S::o_v, col + 2, a.qkv_dtype), v3 = ld_elem(stg + S::o_v, col + 3, a.qkv_dtype);
      r.x = beta * (v0 - sum.x); r.y = beta * (v1 - sum.y); r.z = beta * (v2 - sum.z); r.w = beta * (v3 - sum.w);
    }
    sync_consumers();   // the partial sums have been read by everybody before they are overwritten
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < RW; ++i) {
      const float qq = ld_elem(stg + S::o_q, r0 + i, a.qkv_dtype) * qn;
      st[i].x += kr[i] * r.x; st[i].y += kr[i] * r.y; st[i].z += kr[i] * r.z; st[i].w += kr[i] * r.w;
      o.x += st[i].x * qq; o.y += st[i].y * qq; o.z += st[i].z * qq; o.w += st[i].w * qq;
      *reinterpret_cast<float4*>(St + (r0 + i) * DV + col) = st[i];
    }
    *reinterpret_cast<float4*>(&red[warp][col]) = o;
    tc5::fence_async_smem();       // the new state is read by the producer's bulk copy
    sync_consumers();
    if (tid < DV) {
      float sum = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) sum += red[w][tid];
      st_elem(a.o, ((int64_t)(item / a.HV) * a.HV + hv) * DV + tid, a.qkv_dtype, sum);
    }
    tc5::mbar_arrive(&done[s]);
    sync_consumers();   // red is free again for the next item
  }
}

// (sequence, head) pairs from which a single-token step streams its states: measured at K = V = 128, 512 pairs 12.4 us
// for the step kernel against 14.0, 1024 pairs 30.4 against 28.1, 4096 pairs 104 against 97.
constexpr int kStreamPairs = 768;

template <int DK>
int launch(const b200gdn_recurrent_args& a, cudaStream_t st) {
  if constexpr (DK == 64 || DK == 128) {
    // one token per sequence at large batch: the streaming kernel (state and token rows by bulk copies, ring of three;
    // it needs 16-byte boundaries, [K,V] states and V = 128)
    if (!(a.flags & B200GDN_REC_STATE_V_FIRST) && a.V == 128 && a.T == 1 && a.cu_seqlens == nullptr && a.h0 != nullptr &&
        a.ht != nullptr && (int64_t)a.n_seq * a.HV >= kStreamPairs && (reinterpret_cast<uintptr_t>(a.q) & 15) == 0 &&
        (reinterpret_cast<uintptr_t>(a.k) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.v) & 15) == 0 &&
        (reinterpret_cast<uintptr_t>(a.h0) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.ht) & 15) == 0) {
      using S = DecodeSmem<DK>;
      if (int e = ensure_smem(decode_stream_kernel<DK>, S::bytes)) return e;
      int dev = 0, sms = 148;
      cudaGetDevice(&dev);
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      const int n_items = a.n_seq * a.HV;
      decode_stream_kernel<DK><<<n_items < sms ? n_items : sms, 288, S::bytes, st>>>(a, n_items);
      return check_launch("decode_stream");
    }
  }
  dim3 grid(a.V / VS, a.HV, a.n_seq);
  const bool vf = a.flags & B200GDN_REC_STATE_V_FIRST;
  const bool step = a.T == 1 && a.cu_seqlens == nullptr;   // one token per sequence: no block of tokens to stage
  auto run = [&](auto* one, auto* many) { (step ? one : many)<<<grid, NTHREADS, 0, st>>>(a); };
#define RUN(VF, TY) run(recurrent_step_kernel<DK, VF, TY>, recurrent_kernel<DK, VF, TY>)
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
