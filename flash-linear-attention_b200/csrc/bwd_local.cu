// Everything of the backward pass that is local to a chunk, in one kernel per (chunk, value head): the gradients of q, k, v,
// the gate and beta from the tensors the two scans left.  Replaces chunk_bwd_kernel_dqkwg
// (fla/ops/common/chunk_o.py:172-342), prepare_wy_repr_bwd_kernel (fla/ops/gated_delta_rule/wy_fast.py:123-251) and the
// reverse chunk-local cumsum of dg (gated_delta_rule/chunk.py:244-246).
//
//     dP   = tril(do v_new^T 2^(gamma_i - gamma_j)) scale            do_s = do scale 2^gamma_i          dU = dv2
//     dq^T = h do_s^T + K^T dP^T                                     dW^T = -h dU^T
//     dA   = strict_tril((dW K^T) (beta 2^gamma)_j + (dU V^T) beta_j)
//     M2   = -strict_tril(A^T dA A^T) 2^(gamma_i - gamma_j) beta_i
//     dk^T = (dh v_new^T) 2^(gamma_last - gamma_j) + q^T dP + dW^T A_b + K^T M2^T + K^T M2,   A_b = A (beta 2^gamma)_col
//     dv^T = (dU^T A) beta_j
//     dbeta= c_kbg 2^gamma + c_vb + r_mk,   c_kbg = colsum(A . dW K^T), c_vb = colsum(A . dU V^T), r_mk = rowsum(M . K K^T)
//     dG_i = <dq_i,q_i> - <dk_loc_i,k_i> + c_kbg beta 2^gamma + beta r_mk - c_mk
//            (+ at the last valid row: 2^gamma_last <h,dh> + sum_j <dk_state_j, k_j>);     dg = reverse cumsum of dG
// with dk_loc the first two terms of dk, <dk_loc_j,k_j> = <dk_state_j,k_j> + colsum(dP . Q K^T)_j, c_mk = colsum(M2 . K K^T).
// (The WY terms of dk contribute c_kbg beta 2^gamma + beta r_mk + c_mk to <dk_i,k_i>, so dG could be had from the finished dk
// without Q K^T and c_mk; but then the bf16 operands of those terms do not cancel against the fp32 sums, and the sums of dg
// over a sequence, dA_log and ddt_bias, were twice as far from fp64 as with the terms kept apart: 0.016 against 0.008.)
//
// As two kernels (dq and the chunk-local part of dk; the WY backward) k, h and that part of dk went through HBM twice:
// 296 KiB per chunk and head at K = V = 128, 216 now, and nine dependent tensor-core phases are six.  Products with a
// K- or V-wide result are formed TRANSPOSED ([K x 64 tokens], M = 128): the same tcgen05 instruction then does twice the
// work of an M = 64 one, an accumulator takes 64 TMEM columns instead of 128, and every lane of a TMEM load carries data.
// Tiles leave token-major straight from registers (movmatrix, then 16-byte words).
// One CTA of eight warps; 256 TMEM columns (C0: dP, dq^T, dU V^T, K K^T, Q K^T; C1: the sum of dq over a group; C2: dW^T, dW K^T, Y, X,
// dv^T; C3: dk^T) and ~111 KiB of shared memory whose regions change hands, so two CTAs per SM overlap each other's phases:
//   R1: K      R2: do -> q      R3: v_new -> dU      R4: dh panel 0 -> h panel 0 -> dW^T
//   R5: dh panel 1 -> h panel 1 -> V -> dA | Y -> M2 | Y
// Grouped value heads, many chunks: a CTA takes the heads of a group in turn, K stays, the tiles of the next head are fetched
// under the last epilogue; the sum of dq waits in C1, that of dk in local memory (TMEM is full; 32 KiB per CTA that stay in L2).
// Few chunks: a CTA per head, the CTAs of a group form a cluster; each leaves its fp32 dq and dk in shared memory and adds up
// a share of the rows over distributed shared memory.  Both add in head order (no atomics, no fp32 tensors in HBM).
#include "tc5_tile.cuh"
#include "tma.cuh"

namespace gdn {
namespace {

constexpr int NTHREADS = 256;
__device__ int g_local_timeout = 0;

template <int DK>
struct LocalSmem {
  static constexpr size_t tile = BT * DK * 2;                       // [64][DK] bf16 = [DK][64] bf16
  static constexpr size_t o_k = 0, o_do = tile, o_vn = 2 * tile, o_h0 = 3 * tile, o_h1 = 4 * tile;
  static constexpr size_t h1_bytes = tile > 2 * BT * 128 ? tile : 2 * BT * 128;
  static constexpr size_t o_a = o_h1 + h1_bytes, o_ps = o_a + BT * 128, o_ab = o_ps + BT * 128;
  static constexpr size_t o_vec = o_ab + BT * 128;
  static constexpr int LDS = DK + 4;                                // fp32 row stride of the group-sum staging
  static constexpr size_t stage = (size_t)BT * LDS * 4;             // dq, then dk, from R2 on
  static constexpr size_t bytes = o_vec + 29 * BT * 4 + 160 + 1024; // + vectors, barriers, alignment slack
  static_assert(o_do + 2 * stage <= o_vec, "the group-sum staging fits over the dead tiles");
};

struct LocalMaps {
  CUtensorMap q, k, v, d_o, vn, du, a, h, dh;
};

// eight values per lane, each to be summed over the eight row-lanes of the warp (bits 2..4): recursive halving, 7 shuffles;
// the lane with row index g ends up with the sum of value g, i.e. of column 8 (g >> 1) + 2 t + (g & 1) of a 32-column block
__device__ __forceinline__ float sum8_over_g(const float (&v)[8], int g) {
  float w[4], x[2];
  const bool h4 = g & 4, h2 = g & 2, h1 = g & 1;
#pragma unroll
  for (int j = 0; j < 4; ++j) w[j] = (h4 ? v[4 + j] : v[j]) + __shfl_xor_sync(0xffffffffu, h4 ? v[j] : v[4 + j], 16);
#pragma unroll
  for (int j = 0; j < 2; ++j) x[j] = (h2 ? w[2 + j] : w[j]) + __shfl_xor_sync(0xffffffffu, h2 ? w[j] : w[2 + j], 8);
  return (h1 ? x[1] : x[0]) + __shfl_xor_sync(0xffffffffu, h1 ? x[0] : x[1], 4);
}
__device__ __forceinline__ float sum_over_t(float x) {
  x += __shfl_xor_sync(0xffffffffu, x, 1);
  x += __shfl_xor_sync(0xffffffffu, x, 2);
  return x;
}
__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// This warp's block of a transposed accumulator: rows (DK/4) q + 16 hf + {g, g + 8}, tokens cs + 8 i + 2 t + {0, 1}
template <int NH>
__device__ __forceinline__ void acc_ld_t(uint32_t tm, int q, int cs, float (&r)[NH][16]) {
#pragma unroll
  for (int hf = 0; hf < NH; ++hf) tc5::tmem_ld_16x256b_x4(tm + ((uint32_t)(32 * q + 16 * hf) << 16) + cs, r[hf]);
}
template <int NH>
__device__ __forceinline__ void add_t(float (&r)[NH][16], const float (&before)[NH][16]) {
#pragma unroll
  for (int hf = 0; hf < NH; ++hf)
#pragma unroll
    for (int e = 0; e < 16; ++e) r[hf][e] = before[hf][e] + r[hf][e];
}
// ... its dot products with the same block of a [token][column] tile, added over the rows: value 2 i + p of the result
// belongs to token 8 i + 2 t + p and still has to be summed over g
template <int NH>
__device__ __forceinline__ void dots_t(const float (&r)[NH][16], const unsigned char* tile, int row0, int cs, int lane, float (&pv)[8]) {
#pragma unroll
  for (int e = 0; e < 8; ++e) pv[e] = 0.f;
#pragma unroll
  for (int hf = 0; hf < NH; ++hf) {
    FragLoadT f;
    f.load(tile, BT, cs, row0 + 16 * hf, lane);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = f.lo2(i), y = f.hi2(i);
      pv[2 * i] += r[hf][4 * i] * x.x + r[hf][4 * i + 2] * y.x;
      pv[2 * i + 1] += r[hf][4 * i + 1] * x.y + r[hf][4 * i + 3] * y.y;
    }
  }
}
// ... and its way to token-major global memory (`base`: row 0 of the chunk, this warp's first column)
template <int NH>
__device__ __forceinline__ void store_t(const float (&r)[NH][16], __nv_bfloat16* base, int64_t stride, int cs, int len, int g, int t) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t w[4];
#pragma unroll
    for (int hf = 0; hf < NH; ++hf) {
      w[2 * hf] = transpose8(pack_bf16(r[hf][4 * i], r[hf][4 * i + 1]));
      w[2 * hf + 1] = transpose8(pack_bf16(r[hf][4 * i + 2], r[hf][4 * i + 3]));
    }
    const int tok = cs + 8 * i + g;
    if constexpr (NH == 2) {
      const uint4 v = quad_words(w, t);
      if (tok < len) *reinterpret_cast<uint4*>(base + tok * stride + 8 * t) = v;
    } else if (tok < len) {
      *reinterpret_cast<uint32_t*>(base + tok * stride + 2 * t) = w[0];
      *reinterpret_cast<uint32_t*>(base + tok * stride + 8 + 2 * t) = w[1];
    }
  }
}

// backward of the L2 norm on such a block: x = d w.r.t. the normalised row -> (x - y <x,y>) rstd, with y the tile, the dots in
// four partials per token and rstd per token
template <int NH>
__device__ __forceinline__ void l2_backward_t(float (&r)[NH][16], const unsigned char* tile, const float* dots, const float* rstd, int row0,
                                              int cs, int lane) {
  const int t = lane & 3;
  float2 d[4], rs[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int tok = cs + 8 * i + 2 * t;
    float2 p[4];
#pragma unroll
    for (int w = 0; w < 4; ++w) p[w] = *reinterpret_cast<const float2*>(&dots[w * BT + tok]);
    d[i] = make_float2((p[0].x + p[1].x) + (p[2].x + p[3].x), (p[0].y + p[1].y) + (p[2].y + p[3].y));
    rs[i] = *reinterpret_cast<const float2*>(&rstd[tok]);
  }
#pragma unroll
  for (int hf = 0; hf < NH; ++hf) {
    FragLoadT f;
    f.load(tile, BT, cs, row0 + 16 * hf, lane);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = f.lo2(i), y = f.hi2(i);
      r[hf][4 * i] = (r[hf][4 * i] - x.x * d[i].x) * rs[i].x;
      r[hf][4 * i + 1] = (r[hf][4 * i + 1] - x.y * d[i].y) * rs[i].y;
      r[hf][4 * i + 2] = (r[hf][4 * i + 2] - y.x * d[i].x) * rs[i].x;
      r[hf][4 * i + 3] = (r[hf][4 * i + 3] - y.y * d[i].y) * rs[i].y;
    }
  }
}

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// How the value heads of a q/k head meet: there is one; each has a CTA and the CTAs form a cluster; one CTA takes them in turn
enum Heads { kOne, kCluster, kTurns };

template <int DK, Heads MODE>
__global__ void __launch_bounds__(NTHREADS, 2) bwd_local_kernel(const b200gdn_chunk_args a, const __grid_constant__ LocalMaps maps) {
  constexpr bool GROUPED = MODE == kCluster;
  using S = LocalSmem<DK>;
  constexpr int NP = DK / 64;   // 64-column panels of a V-wide tile (V = K)
  constexpr int NH = DK / 64;   // 16-row halves of a transposed accumulator per warp
  extern __shared__ unsigned char smem_raw[];
  wait_for_predecessor();
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char *Ks = smem + S::o_k, *Do = smem + S::o_do, *Qs = Do, *Vn = smem + S::o_vn, *dUs = Vn, *H0 = smem + S::o_h0, *dWt = H0;
  unsigned char *H1 = smem + S::o_h1, *Vs = H1, *dAs = H1, *M2s = H1, *Ys = H1 + BT * 128;
  unsigned char *As = smem + S::o_a, *Ps = smem + S::o_ps, *Abs = smem + S::o_ab;
  float* const gs2 = reinterpret_cast<float*>(smem + S::o_vec);   // [2][64]: a head's and the next one's
  float *bet = gs2 + 2 * BT, *bge = bet + BT, *eg = bge + BT, *sgm = eg + BT, *gx = sgm + BT, *gv = gx + BT, *dGs = gv + BT, *rsq = dGs + BT, *rsk = rsq + BT;
  // sums over rows: each of the four row-quadrant warps leaves its partial in its own slot and the consumer adds the four in
  // a fixed order (no atomics: results are bit-reproducible)
  float* c_rq = rsk + BT;        // [4][64] <dq_i, q_i>
  float* c_rk = c_rq + 4 * BT;   // [4][64] <dk_loc_i, k_i> + c_mk
  float* c_kbg = c_rk + 4 * BT;  // [4][64] colsum(A . dW K^T)
  float* c_vb = c_kbg + 4 * BT;  // [4][64] colsum(A . dU V^T)
  float* r_mk = c_vb + 4 * BT;   // [2][64] rowsum(M . K K^T), two column halves
  float* red = r_mk + 2 * BT;    // [0..7] <h,dh> per warp, [8..15] sum of <dk_state, k> per warp, [16..19] gate sums
  uint64_t* bar = reinterpret_cast<uint64_t*>(red + 20);
  uint64_t *bar_a = bar + 1, *bar_k = bar + 2, *bar_b = bar + 3, *bar_c = bar + 4;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 5);

  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int q = warp & 3, hc = warp >> 2, g = lane >> 2, t = lane & 3;
  const int c = blockIdx.x, G = a.HV / a.H, hq = MODE == kTurns ? blockIdx.y : blockIdx.y / G;
  const int hv0 = MODE == kTurns ? hq * G : blockIdx.y, n_heads = MODE == kTurns ? G : 1;
  const ChunkMeta cm = load_chunk_meta(a.chunk_meta, c);
  const int64_t row0 = cm.row;
  const int r_lo = q * 16 + g, r_hi = r_lo + 8, cs = hc * 32;   // this warp's block of a [64][64] tile
  const int kr = (DK / 4) * q;                                  // ... and its first row of a transposed accumulator
  const int gcol = cs + 8 * (g >> 1) + 2 * t + (g & 1);         // the column whose sum sum8_over_g leaves in this lane

  // one thread: what a head's first phases need, and the rest into L2
  auto load_head = [&](int hv, bool first) {
    const int hrow = (c * a.HV + hv) * DK;   // the head's state snapshot in the [.., V] view
    tc5::mbar_expect_tx(bar_a, (uint32_t)(2 * S::tile + NP * DK * 128 + BT * 4));
    tma::load_3d(Do, &maps.d_o, cm.row, (hv * DK) / 64, bar_a);
    tma::load_3d(Vn, &maps.vn, cm.row, (hv * DK) / 64, bar_a);
    tma::load_1d(gs2 + ((hv - hv0) & 1) * BT, gamma_ptr(a.gamma, c, a.HV, hv), BT * 4, bar_a);
    for (int p = 0; p < NP; ++p) tma::load_2d(p ? H1 : H0, &maps.dh, p * 64, hrow, bar_a);
    tc5::mbar_expect_tx(bar_k, (uint32_t)((first ? S::tile : 0) + BT * 128));
    if (first) tma::load_3d(Ks, &maps.k, cm.row, (hq * DK) / 64, bar_k);
    tma::load_2d(As, &maps.a, hv * BT, cm.row, bar_k);
    for (int p = 0; p < NP; ++p) tma::prefetch_2d(&maps.h, p * 64, hrow);
    tma::prefetch_3d(&maps.du, cm.row, (hv * DK) / 64);
    if (first) tma::prefetch_3d(&maps.q, cm.row, (hq * DK) / 64);
    tma::prefetch_3d(&maps.v, cm.row, (hv * DK) / 64);
  };
  if (tid == 0) {
    for (int i = 0; i < 5; ++i) tc5::mbar_init(bar + i, 1);
    tc5::fence_mbar_init();
    load_head(hv0, true);
  }
  if (warp == 1) tc5::tmem_alloc(tmem_slot, 256);
  auto head_vectors = [&](int hv) {   // beta and, with the gate option, the gate's value and derivative
    if (tid < BT) {
      const bool ok = tid < cm.len;
      float b = ok ? ld_param(a.beta, (row0 + tid) * a.HV + hv, a.gb_dtype) : 0.f;
      if (a.options & B200GDN_PREP_BETA_SIGMOID) {   // raw beta: the kernels work with (1|2) sigmoid(beta)
        const float sg = 1.f / (1.f + expf(-b));
        sgm[tid] = sg;
        b = ok ? ((a.options & B200GDN_PREP_NEG_EIGVAL) ? 2.f : 1.f) * sg : 0.f;
      }
      bet[tid] = b;
    }
    if ((a.options & B200GDN_PREP_GATE) && tid >= 2 * BT && tid < 3 * BT) {
      // fused gate: g = -exp(A_log) softplus(x), x = g_raw + dt_bias; its value and derivative, while the tiles are on their way
      const int r = tid - 2 * BT;
      const float x = (r < cm.len ? ld_param(a.g, (row0 + r) * a.HV + hv, a.gb_dtype) : 0.f) + (a.dt_bias ? a.dt_bias[hv] : 0.f);
      const float negA = -expf(a.A_log[hv]);
      gx[r] = negA / (1.f + expf(-x));
      gv[r] = negA * (x > 20.f ? x : log1pf(expf(x)));
    }
  };
  head_vectors(hv0);
  if (!GROUPED && tid >= BT && tid < 2 * BT) {   // L2-norm option: reciprocal norms of the rows
    const int r = tid - BT;
    if (a.rstd_q != nullptr) rsq[r] = r < cm.len ? a.rstd_q[(row0 + r) * a.H + hq] : 0.f;
    if (a.rstd_k != nullptr) rsk[r] = r < cm.len ? a.rstd_k[(row0 + r) * a.H + hq] : 0.f;
  }
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tm = *tmem_slot;
  const uint32_t C0 = tm, C1 = tm + 64, C2 = tm + 128, C3 = tm + 192;
  PhaseBarrier ph{bar, 0u, &g_local_timeout};
  const uint32_t sK = tc5::smem_addr(Ks), sDo = tc5::smem_addr(Do), sVn = tc5::smem_addr(Vn), sH0 = tc5::smem_addr(H0), sH1 = tc5::smem_addr(H1);
  const uint32_t sA = tc5::smem_addr(As), sP = tc5::smem_addr(Ps), sAb = tc5::smem_addr(Abs);
  const Operand opK_k{sK, BT, 0}, opK_mn{sK, BT, 1};      // K as (rows = token, contraction = key dim), and the reverse
  const Operand opA_k{sA, BT, 0}, opA_mn{sA, BT, 1};
  bool failed = false;
  // turns: this thread's part of the sum of dk over the heads, in local memory between them
  __align__(16) float dk_local[MODE == kTurns ? 16 * NH : 4];
  const uint64_t dk_sum = __cvta_generic_to_local(dk_local);

  for (int hh = 0; hh < n_heads; ++hh) {
    const int hv = hv0 + hh, hrow = (c * a.HV + hv) * DK;
    const uint32_t par = hh & 1;
    const bool first = MODE != kTurns || hh == 0, last = MODE != kTurns || hh + 1 == n_heads;
    const float* gs = gs2 + par * BT;
    if (!tc5::mbar_wait(bar_a, par)) failed = true;
    if (cm.len < BT) {   // ragged chunk: the extra rows of the boxes belong to the next sequence
      zero_tail_rows<BT, DK>(Do, cm.len, tid, NTHREADS);
      zero_tail_rows<BT, DK>(Vn, cm.len, tid, NTHREADS);
      tc5::fence_async_smem();
    }
    if (__syncthreads_or(failed)) { failed = true; break; }

    // ---- phase 1: dP = do v_new^T | dk_state^T = dh v_new^T (column factor later)
    if (warp == 0) {
      tc5::fence_after_sync();
      issue_mma_t<DK / 16>(C0, Operand{sDo, BT, 0}, Operand{sVn, BT, 0}, 64, 64, 0);
#pragma unroll
      for (int p = 0; p < NP; ++p)
        issue_mma_t<4>(C3, Operand{p ? sH1 : sH0, DK, 0}, Operand{sVn + p * BT * 128, BT, 0}, DK, 64, p > 0);
      ph.commit();
    }
    const float g_lo = gs[r_lo], g_hi = gs[r_hi], glast = gs[BT - 1];
    if (tid < BT) {
      const float e = fast_exp2(gs[tid]);
      eg[tid] = e;
      bge[tid] = bet[tid] * e;
    }
    if (!tc5::mbar_wait(bar_k, par)) failed = true;
    if (cm.len < BT) {
      if (first) zero_tail_rows<BT, DK>(Ks, cm.len, tid, NTHREADS);
      zero_tail_rows<BT, BT>(As, cm.len, tid, NTHREADS);
      tc5::fence_async_smem();
    }
    if (__syncthreads_or(failed || !ph.wait())) { failed = true; break; }

    // ---- epilogue 1: dh into registers (for <h,dh>), then h takes its place and dU the place of v_new
    constexpr int ND = DK * 8 * NP / NTHREADS;
    uint4 dhr[ND];
#pragma unroll
    for (int n = 0; n < ND; ++n) {
      const int idx = tid + n * NTHREADS;   // 16-byte words of both panels; the same positions are read in h
      dhr[n] = *reinterpret_cast<const uint4*>((idx < DK * 8 ? H0 : H1 - DK * 128) + idx * 16);
    }
    // the reads above are only issued: without this fence the copy of h can overtake those still queued
    tc5::fence_async_smem();
    __syncthreads();
    if (tid == 0) {
      tc5::mbar_expect_tx(bar_b, (uint32_t)(NP * DK * 128 + S::tile));
      for (int p = 0; p < NP; ++p) tma::load_2d(p ? H1 : H0, &maps.h, p * 64, hrow, bar_b);
      tma::load_3d(dUs, &maps.du, cm.row, (hv * DK) / 64, bar_b);
    }
    {   // dP~ -> shared
      float r[16];
      acc_ld32q(C0, q, cs, r);
      tc5::tmem_ld_wait();
      FragStore fs;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int j0 = cs + i * 8 + 2 * t;
        const float2 gj = *reinterpret_cast<const float2*>(&gs[j0]);
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int ii = (e & 2) ? r_hi : r_lo, jj = j0 + (e & 1);
          v[e] = (ii >= jj) ? r[4 * i + e] * a.scale * fast_exp2(((e & 2) ? g_hi : g_lo) - ((e & 1) ? gj.y : gj.x)) : 0.f;
        }
        fs.set(i, v[0], v[1], v[2], v[3]);
      }
      fs.store(Ps, BT, q * 16, cs, lane);
    }
#pragma unroll
    for (int n = 0; n < BT * DK / 8 / NTHREADS; ++n) {   // do_s in place
      const int idx = tid + n * NTHREADS, row = (idx % (BT * 8)) / 8;
      const float fo = a.scale * eg[row];
      uint4* po = reinterpret_cast<uint4*>(Do + idx * 16);
      uint4 x = *po;
      uint32_t* xu = reinterpret_cast<uint32_t*>(&x);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 p = unpack_bf16(xu[e]);
        xu[e] = pack_bf16(p.x * fo, p.y * fo);
      }
      *po = x;
    }
    float dk_dot;   // this lane's part of c_rk
    {   // dk_state^T: column factors, the sum of its dots with k, back to TMEM where the other terms of dk accumulate
      float r[NH][16];
      acc_ld_t<NH>(C3, q, cs, r);
      tc5::tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 gj = *reinterpret_cast<const float2*>(&gs[cs + i * 8 + 2 * t]);
        const float e0 = fast_exp2(glast - gj.x), e1 = fast_exp2(glast - gj.y);
#pragma unroll
        for (int hf = 0; hf < NH; ++hf) {
          r[hf][4 * i] *= e0; r[hf][4 * i + 1] *= e1; r[hf][4 * i + 2] *= e0; r[hf][4 * i + 3] *= e1;
        }
      }
#pragma unroll
      for (int hf = 0; hf < NH; ++hf) tc5::tmem_st_16x256b_x4(C3 + ((uint32_t)(32 * q + 16 * hf) << 16) + cs, r[hf]);
      float pv[8];
      dots_t<NH>(r, Ks, kr, cs, lane, pv);
      dk_dot = sum8_over_g(pv, g);
      const float rs = warp_sum(dk_dot);
      if (lane == 0) red[8 + warp] = rs;
      tc5::tmem_st_wait();
    }
    if (!tc5::mbar_wait(bar_b, par)) failed = true;
    if (cm.len < BT) zero_tail_rows<BT, DK>(dUs, cm.len, tid, NTHREADS);
    {
      float hd = 0.f;
#pragma unroll
      for (int n = 0; n < ND; ++n) {
        const int idx = tid + n * NTHREADS;
        const uint4 x = *reinterpret_cast<const uint4*>((idx < DK * 8 ? H0 : H1 - DK * 128) + idx * 16);
        const uint32_t xu[4] = {x.x, x.y, x.z, x.w}, yu[4] = {dhr[n].x, dhr[n].y, dhr[n].z, dhr[n].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 p = unpack_bf16(xu[e]), y = unpack_bf16(yu[e]);
          hd += p.x * y.x + p.y * y.y;
        }
      }
      hd = warp_sum(hd);
      if (lane == 0) red[warp] = hd;
    }
    tc5::fence_async_smem();
    tc5::fence_before_sync();
    if (__syncthreads_or(failed)) { failed = true; break; }

    // ---- phase 2: dq^T = h do_s^T + K^T dP~^T | dW^T = -h dU^T
    if (warp == 0) {
      tc5::fence_after_sync();
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        issue_mma_t<4>(C2, Operand{p ? sH1 : sH0, DK, 0}, Operand{sVn + p * BT * 128, BT, 0}, DK, 64, p > 0, /*neg_a=*/1);
        issue_mma_t<4>(C0, Operand{p ? sH1 : sH0, DK, 0}, Operand{sDo + p * BT * 128, BT, 0}, DK, 64, p > 0);
      }
      issue_mma_t<4>(C0, opK_mn, Operand{sP, BT, 0}, DK, 64, 1);
      ph.commit();
    }
    {   // A with its columns scaled by beta 2^gamma, while phase 2 runs
      FragLoad fa;
      fa.load(As, BT, q * 16, cs, lane);
      FragStore fs;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 sc = *reinterpret_cast<const float2*>(&bge[cs + i * 8 + 2 * t]);
        const float2 al = fa.lo2(i), ah = fa.hi2(i);
        fs.set(i, al.x * sc.x, al.y * sc.y, ah.x * sc.x, ah.y * sc.y);
      }
      fs.store(Abs, BT, q * 16, cs, lane);
    }
    if (__syncthreads_or(!ph.wait())) { failed = true; break; }

    // ---- epilogue 2: q takes the place of do, V that of the second h panel; dW^T -> shared (over the first)
    if (tid == 0) {
      tc5::mbar_expect_tx(bar_c, (uint32_t)(2 * S::tile));
      tma::load_3d(Vs, &maps.v, cm.row, (hv * DK) / 64, bar_c);
      tma::load_3d(Qs, &maps.q, cm.row, (hq * DK) / 64, bar_c);
    }
    {
      float r[NH][16];
      acc_ld_t<NH>(C2, q, cs, r);
      tc5::tmem_ld_wait();
#pragma unroll
      for (int hf = 0; hf < NH; ++hf) {
        FragStore fs;
#pragma unroll
        for (int i = 0; i < 4; ++i) fs.set(i, r[hf][4 * i], r[hf][4 * i + 1], r[hf][4 * i + 2], r[hf][4 * i + 3]);
        fs.store(dWt, DK, kr + 16 * hf, cs, lane);
      }
    }
    float rq[NH][16];   // dq: C0 is phase 3's
    acc_ld_t<NH>(C0, q, cs, rq);
    if (!tc5::mbar_wait(bar_c, par)) failed = true;
    if (cm.len < BT) {
      zero_tail_rows<BT, DK>(Qs, cm.len, tid, NTHREADS);
      zero_tail_rows<BT, DK>(Vs, cm.len, tid, NTHREADS);
    }
    tc5::tmem_ld_wait();
    tc5::fence_async_smem();
    tc5::fence_before_sync();
    if (__syncthreads_or(failed)) { failed = true; break; }

    // ---- phase 3: dA1 = dW K^T | dA2 = dU V^T
    if (warp == 0) {
      tc5::fence_after_sync();
      issue_mma_t<DK / 16>(C2, Operand{sH0, DK, 1}, opK_k, 64, 64, 0);
      issue_mma_t<DK / 16>(C0, Operand{sVn, BT, 0}, Operand{sH1, BT, 0}, 64, 64, 0);
      ph.commit();
    }
    {   // dq: its dots with q, the sum over the heads (C1); ungrouped heads, and the last one in turn: it leaves
      float pv[8];
      dots_t<NH>(rq, Qs, kr, cs, lane, pv);
      c_rq[q * BT + gcol] = sum8_over_g(pv, g);
      if (!first) {
        float acc[NH][16];
        acc_ld_t<NH>(C1, q, cs, acc);
        tc5::tmem_ld_wait();
        add_t<NH>(rq, acc);
      }
      if (GROUPED || !last) {
#pragma unroll
        for (int hf = 0; hf < NH; ++hf) tc5::tmem_st_16x256b_x4(C1 + ((uint32_t)(32 * q + 16 * hf) << 16) + cs, rq[hf]);
        tc5::tmem_st_wait();
      } else {
        if (a.rstd_q != nullptr) {
          float* dots = c_rq;
          if (MODE == kTurns) {   // of the sum; c_kbg is free until epilogue 3
            dots = c_kbg;
            dots_t<NH>(rq, Qs, kr, cs, lane, pv);
            dots[q * BT + gcol] = sum8_over_g(pv, g);
          }
          __syncthreads();
          l2_backward_t<NH>(rq, Qs, dots, rsq, kr, cs, lane);
        }
        store_t<NH>(rq, reinterpret_cast<__nv_bfloat16*>(a.dq) + (row0 * a.H + hq) * DK + kr, (int64_t)a.H * DK, cs, cm.len, g, t);
      }
    }
    if (__syncthreads_or(!ph.wait())) { failed = true; break; }

    // ---- epilogue 3: dA -> shared (over V)
    {
      float r[16], dA2[16];
      acc_ld32q(C2, q, cs, r);
      acc_ld32q(C0, q, cs, dA2);
      tc5::tmem_ld_wait();
      FragStore fs;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int col = cs + i * 8 + 2 * t;
        const float2 bg = *reinterpret_cast<const float2*>(&bge[col]), bj = *reinterpret_cast<const float2*>(&bet[col]);
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int ii = (e & 2) ? r_hi : r_lo, jj = col + (e & 1);
          v[e] = (ii > jj) ? r[4 * i + e] * ((e & 1) ? bg.y : bg.x) + dA2[4 * i + e] * ((e & 1) ? bj.y : bj.x) : 0.f;
        }
        fs.set(i, v[0], v[1], v[2], v[3]);
      }
      fs.store(dAs, BT, q * 16, cs, lane);
      tc5::fence_async_smem();
      tc5::fence_before_sync();
      __syncthreads();
      // ---- phase 4: Y = dA A^T (all the chain waits for) | KK = K K^T
      if (warp == 0) {
        tc5::fence_after_sync();
        issue_mma_t<BT / 16>(C2, Operand{sH1, BT, 0}, opA_k, 64, 64, 0);
        ph.commit();
        issue_mma_t<DK / 16>(C0, opK_k, opK_k, 64, 64, 0);
      }
      FragLoad fa;
      fa.load(As, BT, q * 16, cs, lane);
      float pv[8], pw[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 al = fa.lo2(i), ah = fa.hi2(i);
        pv[2 * i] = al.x * r[4 * i] + ah.x * r[4 * i + 2];
        pv[2 * i + 1] = al.y * r[4 * i + 1] + ah.y * r[4 * i + 3];
        pw[2 * i] = al.x * dA2[4 * i] + ah.x * dA2[4 * i + 2];
        pw[2 * i + 1] = al.y * dA2[4 * i + 1] + ah.y * dA2[4 * i + 3];
      }
      c_kbg[q * BT + gcol] = sum8_over_g(pv, g);
      c_vb[q * BT + gcol] = sum8_over_g(pw, g);
    }
    if (__syncthreads_or(!ph.wait())) { failed = true; break; }

    // ---- epilogue 4: Y -> shared
    {
      float r[16];
      acc_ld32q(C2, q, cs, r);
      tc5::tmem_ld_wait();
      FragStore fs;
#pragma unroll
      for (int i = 0; i < 4; ++i) fs.set(i, r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
      fs.store(Ys, BT, q * 16, cs, lane);
    }
    tc5::fence_async_smem();
    tc5::fence_before_sync();
    __syncthreads();

    // ---- phase 5: X = A^T Y (all the chain waits for) | dk^T += q^T dP~ + dW^T A_b
    if (warp == 0) {
      tc5::fence_after_sync();
      issue_mma_t<BT / 16>(C2, opA_mn, Operand{sH1 + BT * 128, BT, 1}, 64, 64, 0);
      ph.commit();
      issue_mma_t<BT / 16>(C3, Operand{sDo, BT, 1}, Operand{sP, BT, 1}, DK, 64, 1);
      issue_mma_t<BT / 16>(C3, Operand{sH0, DK, 0}, Operand{sAb, BT, 1}, DK, 64, 1);
    }
    if (__syncthreads_or(!ph.wait())) { failed = true; break; }

    // ---- epilogue 5: M2 -> shared
    {
      const float b_lo = bet[r_lo], b_hi = bet[r_hi];
      float m[16], kk[16];
      acc_ld32q(C2, q, cs, m);
      acc_ld32q(C0, q, cs, kk);
      tc5::tmem_ld_wait();
      FragStore fs;
      float rmk_lo = 0.f, rmk_hi = 0.f, pv[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int col = cs + i * 8 + 2 * t;
        const float2 gj = *reinterpret_cast<const float2*>(&gs[col]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int ii = (e & 2) ? r_hi : r_lo, jj = col + (e & 1);
          m[4 * i + e] = (ii > jj) ? -m[4 * i + e] * fast_exp2(((e & 2) ? g_hi : g_lo) - ((e & 1) ? gj.y : gj.x)) : 0.f;
        }
        rmk_lo += m[4 * i] * kk[4 * i] + m[4 * i + 1] * kk[4 * i + 1];
        rmk_hi += m[4 * i + 2] * kk[4 * i + 2] + m[4 * i + 3] * kk[4 * i + 3];
        m[4 * i] *= b_lo; m[4 * i + 1] *= b_lo; m[4 * i + 2] *= b_hi; m[4 * i + 3] *= b_hi;
        pv[2 * i] = m[4 * i] * kk[4 * i] + m[4 * i + 2] * kk[4 * i + 2];
        pv[2 * i + 1] = m[4 * i + 1] * kk[4 * i + 1] + m[4 * i + 3] * kk[4 * i + 3];
        fs.set(i, m[4 * i], m[4 * i + 1], m[4 * i + 2], m[4 * i + 3]);
      }
      dk_dot += sum8_over_g(pv, g);
      fs.store(M2s, BT, q * 16, cs, lane);
      rmk_lo = sum_over_t(rmk_lo);
      rmk_hi = sum_over_t(rmk_hi);
      if (t == 0) {
        r_mk[hc * BT + r_lo] = rmk_lo;
        r_mk[hc * BT + r_hi] = rmk_hi;
      }
    }
    tc5::fence_async_smem();
    tc5::fence_before_sync();
    __syncthreads();

    // ---- phase 6: dv^T = dU^T A | dk^T += K^T M2^T + K^T M2 | QK = Q K^T
    if (warp == 0) {
      tc5::fence_after_sync();
      issue_mma_t<BT / 16>(C2, Operand{sVn, BT, 1}, opA_mn, DK, 64, 0);
      ph.commit();
      issue_mma_t<BT / 16>(C3, opK_mn, Operand{sH1, BT, 0}, DK, 64, 1);
      issue_mma_t<BT / 16>(C3, opK_mn, Operand{sH1, BT, 1}, DK, 64, 1);
      issue_mma_t<DK / 16>(C0, Operand{sDo, BT, 0}, opK_k, 64, 64, 0);
    }
    if (__syncthreads_or(!ph.wait())) { failed = true; break; }
    if (warp == 0) ph.commit();   // ... of the rest
    {
      float r[NH][16];
      acc_ld_t<NH>(C2, q, cs, r);
      tc5::tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 bj = *reinterpret_cast<const float2*>(&bet[cs + i * 8 + 2 * t]);
#pragma unroll
        for (int hf = 0; hf < NH; ++hf) {
          r[hf][4 * i] *= bj.x; r[hf][4 * i + 1] *= bj.y; r[hf][4 * i + 2] *= bj.x; r[hf][4 * i + 3] *= bj.y;
        }
      }
      store_t<NH>(r, reinterpret_cast<__nv_bfloat16*>(a.dv) + (row0 * a.HV + hv) * DK + kr, (int64_t)a.HV * DK, cs, cm.len, g, t);
    }
    if (__syncthreads_or(!ph.wait())) { failed = true; break; }
    if (!last && tid == 0) load_head(hv + 1, false);   // every tile but K is dead

    // ---- epilogue 6: dk and the gate and beta gradients
    float rk[NH][16];
    {
      float pv[8], qk[16];
      acc_ld32q(C0, q, cs, qk);
      acc_ld_t<NH>(C3, q, cs, rk);
      tc5::tmem_ld_wait();
      FragLoad fp;
      fp.load(Ps, BT, q * 16, cs, lane);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 pl = fp.lo2(i), phi = fp.hi2(i);
        pv[2 * i] = pl.x * qk[4 * i] + phi.x * qk[4 * i + 2];
        pv[2 * i + 1] = pl.y * qk[4 * i + 1] + phi.y * qk[4 * i + 3];
      }
      c_rk[q * BT + gcol] = dk_dot + sum8_over_g(pv, g);
      if (MODE == kTurns) {
        if (!first) {
          float acc[NH][16];
#pragma unroll
          for (int e = 0; e < NH * 4; ++e)
            asm volatile("ld.local.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                         : "=f"(acc[e / 4][4 * (e % 4)]), "=f"(acc[e / 4][4 * (e % 4) + 1]), "=f"(acc[e / 4][4 * (e % 4) + 2]),
                           "=f"(acc[e / 4][4 * (e % 4) + 3])
                         : "l"(dk_sum + 16 * e)
                         : "memory");
          add_t<NH>(rk, acc);
        }
        if (!last) {
#pragma unroll
          for (int e = 0; e < NH * 4; ++e)
            asm volatile("st.local.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(dk_sum + 16 * e), "f"(rk[e / 4][4 * (e % 4)]),
                         "f"(rk[e / 4][4 * (e % 4) + 1]), "f"(rk[e / 4][4 * (e % 4) + 2]), "f"(rk[e / 4][4 * (e % 4) + 3])
                         : "memory");
        }
      }
      if (!GROUPED && last && a.rstd_k != nullptr) {   // <dk, k> for the norm's backward, over a tile that is needed no more
        dots_t<NH>(rk, Ks, kr, cs, lane, pv);
        reinterpret_cast<float*>(Vn)[q * BT + gcol] = sum8_over_g(pv, g);
      }
    }
    __syncthreads();
    if (tid < BT) {
      const int i = tid;
      auto sum4 = [&](const float* v) { return (v[i] + v[BT + i]) + (v[2 * BT + i] + v[3 * BT + i]); };
      const float rmk = r_mk[i] + r_mk[BT + i], ckbg = sum4(c_kbg);
      float x = sum4(c_rq) - sum4(c_rk) + (ckbg * bge[i] + bet[i] * rmk);
      if (i == cm.len - 1) {
        float sh = 0.f, sr = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
          sh += red[w];
          sr += red[8 + w];
        }
        x += fast_exp2(glast) * sh + sr;
      }
      if (i < cm.len) {
        float db = ckbg * eg[i] + sum4(c_vb) + rmk;
        if (a.options & B200GDN_PREP_BETA_SIGMOID)   // chain rule through (1|2) sigmoid
          db *= ((a.options & B200GDN_PREP_NEG_EIGVAL) ? 2.f : 1.f) * sgm[i] * (1.f - sgm[i]);
        st_param(a.dbeta, (row0 + i) * a.HV + hv, a.gb_dtype, db);
      } else {
        x = 0.f;
      }
      // reverse cumsum as a two-warp suffix scan: the sum inside the warp here, the carry below
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float y = __shfl_down_sync(0xffffffffu, x, o);
        if (lane + o < 32) x += y;
      }
      dGs[i] = x;
    }
    if (!GROUPED && last) {
      if (a.rstd_k != nullptr) l2_backward_t<NH>(rk, Ks, reinterpret_cast<float*>(Vn), rsk, kr, cs, lane);
      store_t<NH>(rk, reinterpret_cast<__nv_bfloat16*>(a.dk) + (row0 * a.H + hq) * DK + kr, (int64_t)a.H * DK, cs, cm.len, g, t);
    } else if (GROUPED) {
      // this head's dq and dk in fp32, token-major, over the dead tiles
      float* sq = reinterpret_cast<float*>(smem + S::o_do);
      float* sk = reinterpret_cast<float*>(smem + S::o_do + S::stage);
      float r[NH][16];
      acc_ld_t<NH>(C1, q, cs, r);
      tc5::tmem_ld_wait();
#pragma unroll
      for (int hf = 0; hf < NH; ++hf)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int at = (cs + 8 * i + 2 * t + (e & 1)) * S::LDS + kr + 16 * hf + g + ((e & 2) ? 8 : 0);
            sq[at] = r[hf][4 * i + e];
            sk[at] = rk[hf][4 * i + e];
          }
    }
    __syncthreads();
    if (!(a.options & B200GDN_PREP_GATE)) {
      if (tid < cm.len) st_param(a.dg, (row0 + tid) * a.HV + hv, a.gb_dtype, dGs[tid] + (tid < 32 ? dGs[32] : 0.f));
    } else {
      // dg_raw = dg dg/dg_raw; dA_log += dg g and ddt_bias += dg_raw, summed over the chunk here and over the chunks by a second
      // kernel
      if (tid < BT) {
        float sA = 0.f, sB = 0.f;
        if (tid < cm.len) {
          const float dgi = dGs[tid] + (tid < 32 ? dGs[32] : 0.f);
          const float draw = dgi * gx[tid];
          st_param(a.dg, (row0 + tid) * a.HV + hv, a.gb_dtype, draw);
          sA = dgi * gv[tid];
          sB = draw;
        }
        sA = warp_sum(sA);
        sB = warp_sum(sB);
        if (lane == 0) {
          red[16 + 2 * warp] = sA;
          red[16 + 2 * warp + 1] = sB;
        }
      }
      __syncthreads();
      if (tid == 0) {
        a.gate_partials[((int64_t)c * a.HV + hv) * 2 + 0] = red[16] + red[18];
        a.gate_partials[((int64_t)c * a.HV + hv) * 2 + 1] = red[17] + red[19];
      }
    }
    if (!last) {
      __syncthreads();   // the vectors have been read
      head_vectors(hv + 1);
    }
  }

  if (GROUPED) {
    // every CTA of the group takes 64 / G of the rows; all of them come here, whatever happened above
    cluster_sync();
    if (!failed) {
      constexpr int LPT = DK / 4, TPR = NTHREADS / LPT;   // lanes per token (four columns each), tokens per round
      const int rank = hv0 % G, per = BT / G, col = (tid % LPT) * 4;
      for (int j = tid / LPT; j < per; j += TPR) {
        const int tok = rank * per + j;
#pragma unroll
        for (int w = 0; w < 2; ++w) {   // dq, then dk
          const uint32_t local = tc5::smem_addr(smem + S::o_do + w * S::stage) + (uint32_t)(tok * S::LDS + col) * 4u;
          float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
          for (int p = 0; p < G; ++p) {
            uint32_t peer;
            float4 x;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(peer) : "r"(local), "r"(p));
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "r"(peer) : "memory");
            s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w;
          }
          const int64_t at = (row0 + tok) * a.H + hq;
          const float* rstd = w ? a.rstd_k : a.rstd_q;
          if (rstd != nullptr) {
            float2 y0 = make_float2(0.f, 0.f), y1 = y0;
            if (tok < cm.len) {
              const uint2 u = *reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(w ? a.k : a.q) + at * DK + col);
              y0 = unpack_bf16(u.x);
              y1 = unpack_bf16(u.y);
            }
            float dot = s.x * y0.x + s.y * y0.y + s.z * y1.x + s.w * y1.y;
            // the lanes of a token are consecutive; `per` is a multiple of the tokens a warp holds, so none is missing
#pragma unroll
            for (int o = LPT / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
            const float rs = tok < cm.len ? rstd[at] : 0.f;
            s.x = (s.x - y0.x * dot) * rs; s.y = (s.y - y0.y * dot) * rs; s.z = (s.z - y1.x * dot) * rs; s.w = (s.w - y1.y * dot) * rs;
          }
          if (tok < cm.len)
            *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(w ? a.dk : a.dq) + at * DK + col) = make_uint2(pack_bf16(s.x, s.y), pack_bf16(s.z, s.w));
        }
      }
    }
    cluster_sync();   // shared memory must outlive the peers that read it
  }
  if (failed && tid == 0) atomicExch(&g_local_timeout, 1);
  tc5::fence_before_sync();
  __syncthreads();
  if (warp == 1) tc5::tmem_dealloc(tm, 256);
}

template <int DK, Heads MODE>
int launch(const b200gdn_chunk_args& a, cudaStream_t st) {
  using S = LocalSmem<DK>;
  static_assert(S::bytes <= 113 * 1024, "two CTAs per SM");
  if (int e = ensure_smem(bwd_local_kernel<DK, MODE>, S::bytes)) return e;
  LocalMaps m;
  const uint64_t pk = (uint64_t)a.H * DK, pv = (uint64_t)a.HV * DK, hrows = (uint64_t)a.n_chunks * a.HV * DK;
  int rc = 0;
  rc |= tma::encode_bf16_panels(&m.q, a.q, a.rows, pk, pk, BT, DK / 64);
  rc |= tma::encode_bf16_panels(&m.k, a.k, a.rows, pk, pk, BT, DK / 64);
  rc |= tma::encode_bf16_panels(&m.v, a.v, a.rows, pv, pv, BT, DK / 64);
  rc |= tma::encode_bf16_panels(&m.d_o, a.d_o, a.rows, pv, pv, BT, DK / 64);
  rc |= tma::encode_bf16_panels(&m.vn, a.v_new, a.rows, pv, pv, BT, DK / 64);
  rc |= tma::encode_bf16_panels(&m.du, a.dv2, a.rows, pv, pv, BT, DK / 64);
  rc |= tma::encode_bf16_2d(&m.a, a.A, a.rows, (uint64_t)a.HV * BT, (uint64_t)a.HV * BT, BT);
  rc |= tma::encode_bf16_2d(&m.h, a.h, hrows, DK, DK, DK);
  rc |= tma::encode_bf16_2d(&m.dh, a.dh, hrows, DK, DK, DK);
  if (rc != 0) return set_error(B200GDN_ERR_CUDA, "bwd_local: cuTensorMapEncodeTiled failed (%d)", rc);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a.n_chunks, MODE == kTurns ? a.H : a.HV);
  cfg.blockDim = dim3(NTHREADS);
  cfg.dynamicSmemBytes = S::bytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  cfg.numAttrs = 0;
  if (overlaps(a)) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (MODE == kCluster) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = 1;
    attr[cfg.numAttrs].val.clusterDim.y = a.HV / a.H;
    attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  cudaLaunchKernelEx(&cfg, bwd_local_kernel<DK, MODE>, a, m);
  if (int e = check_launch("bwd_local")) return e;
  return launch_gate_reduce(a, st);
}

// Several value heads per q/k head: in turn in one CTA, or a CTA each and the sums of dq and dk through a cluster.  A cluster
// costs about a quarter more per head (it holds its CTAs until the slowest has arrived and its sums have been read: 272 us
// against 242 at B4 T4096 8/16 heads of 128), but has G times as many CTAs, so it stays where turns would leave
// the device to a few: two fit on an SM, and the rounds of CTAs decide.  Group sizes other than two, four
// and eight are taken in turns always (the two kernels of the single stages, which such groups used where there are few chunks, also
// take heads in turn: 1 x 2048 tokens, 2/12 heads of 128: 122 us, 90 here; 1/3 heads of 64: 34, 32).  Both forms add the heads
// in the same order and precision.
bool in_turns(const b200gdn_chunk_args& a) {
  const int64_t slots = 2 * sm_count();
  const int64_t G = a.HV / a.H;
  if (G != 2 && G != 4 && G != 8) return true;
  const int64_t turns = G * ((a.n_chunks * (int64_t)a.H + slots - 1) / slots),
                cluster = (a.n_chunks * (int64_t)a.HV + slots - 1) / slots;
  return 4 * turns <= 5 * cluster;
}

template <int DK>
int launch_heads(const b200gdn_chunk_args& a, cudaStream_t st) {
  if (a.HV == a.H) return launch<DK, kOne>(a, st);
  return in_turns(a) ? launch<DK, kTurns>(a, st) : launch<DK, kCluster>(a, st);
}

}  // namespace

int launch_bwd_local(const b200gdn_chunk_args& a, cudaStream_t st) {
  if (int e = check_gate_args(a, "bwd_local")) return e;
  if (a.K == 128 && a.V == 128) return launch_heads<128>(a, st);
  if (a.K == 64 && a.V == 64) return launch_heads<64>(a, st);
  return set_error(B200GDN_ERR_UNSUPPORTED, "bwd_local: K=%d V=%d not built (64/64 and 128/128 are)", a.K, a.V);
}

// Reads and clears the flag a bounded device wait raises when it expires (synchronises with the device).
int bwd_local_timeout_flag() {
  int v = 0, zero = 0;
  cudaMemcpyFromSymbol(&v, g_local_timeout, sizeof(int));
  if (v) cudaMemcpyToSymbol(g_local_timeout, &zero, sizeof(int));
  return v;
}

}  // namespace gdn
