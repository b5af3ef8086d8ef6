// Intra-chunk forward: gamma = cumsum(g) log2(e);  A = (I + strict_tril(beta_i <k_i,k_j> 2^(gamma_i-gamma_j)))^-1;
// W = A (K beta 2^gamma);  U = A (V beta);  and (when q and a qk buffer are given)
// qk = tril(<q_i,k_j> 2^(gamma_i-gamma_j)), the chunk-local attention tile of chunk_fwd_kernel_o /
// chunk_bwd_kernel_dv_local (fla/ops/common/chunk_o.py:115-127, 505-520), which shares K, gamma and the gate factors
// with L.   One CTA of eight warps per (chunk, value head).
//
// Replaces chunk_local_cumsum (fla/ops/utils/cumsum.py:33-68), the fused K K^T + triangular solve
// (fla/ops/gated_delta_rule/chunk_fwd.py:40-328) and recompute_w_u_fwd (gated_delta_rule/wy_fast.py:43-106).
//   * K and V tiles arrive by TMA; K K^T, W and U run on tcgen05 with TMEM accumulators (128 columns, used
//     one product after the other); W, U leave through TMA stores (plain predicated stores for a ragged
//     chunk), A and qk from registers in 16-byte words; shared-memory regions are reused along the way so that four CTAs
//     share an SM and hide each other's latencies;
//   * the inverse is formed in exact fp32 on the CUDA cores: the four 16x16 diagonal blocks by forward substitution (one
//     thread per column), then two levels of block merges A21 = -A22 (L21 A11) (16 -> 32 -> 64); the reference uses tf32
//     tensor-core merges;
//   * the row scalings of the W/U right-hand sides are folded into the columns of A, so the K and V tiles are used exactly as
//     loaded (L2-norm option: as normalised in place).
// What bounds it is the shared-memory / L1 data pipe (counters: 76 % of its wavefronts with a lane-per-output mapping of the
// merges, 4-byte stores of qk and A and a zero fill of the inverse, 5.8 k wavefronts a CTA).  So every merge has one operand
// at an address that is uniform over the warp (one wavefront) and 16-byte reads along rows for the other, skips what is
// zero by triangularity, and nothing is filled with zeros first.
// Bounds of the chunk's state transition, where pre-scans will want them (TRANSITION_BOUNDS), cost 3 %: the squared norms of k are the
// diagonal of K K^T, and the largest of W and U is taken from the accumulators on their way out.  That is all they do where heads forget
// nothing: B1 T65536 H16 K=V=128 972 us for 957, with the backward pass 2687 for 2673 (gates of logsigmoid(N(0,1)): 617 and 1890).
// B4 T4096 H16 K=V=128: 87 us inside a step (105), 94 by itself between two events; with the L2 norm, gate and beta options
// 115 us (108 + 47 for a norm pass of its own; 120 with the norm's sums in scalars and normalised rows stored from registers), 109 with
// 8/16 heads.
#include "rowio.cuh"
#include "tc5_tile.cuh"
#include "tma.cuh"

namespace gdn {
namespace {

constexpr int NTHREADS = 256;
constexpr int LDF = 68;  // fp32 row stride of the 64x64 solve matrices
constexpr int LDT = 36;  // fp32 row stride of the (at most 32x32) merge temporary
__device__ int g_intra_timeout = 0;

template <int DK, int DV>
struct IntraSmem {
  // Regions are reused as the kernel advances (each hand-over is separated by a CTA barrier):
  //   K tile                      -> W staging
  //   fp32 L                      -> V tile (loaded once L is dead) -> U staging
  //   fp32 inverse                -> bf16 A (beta 2^gamma)_col | A beta_col
  //   fp32 merge temporary (32x32)
  // 56 896 bytes at K = V = 128: with the 1 KiB the system keeps per CTA, four CTAs fill the 228 KiB of an SM exactly,
  // which is why the dynamic window is used from its (1024-byte aligned, checked) start without an alignment slack.
  static constexpr size_t fmat = ((sizeof(float) * BT * LDF + 1023) / 1024) * 1024;
  static constexpr size_t o_k = 0;
  static constexpr size_t o_l = o_k + BT * DK * 2;
  static constexpr size_t o_a = o_l + (fmat > BT * DV * 2 ? fmat : BT * DV * 2);
  static constexpr size_t o_t = o_a + fmat;
  static constexpr size_t o_vec = o_t + sizeof(float) * 32 * LDT;
  static constexpr size_t bytes = o_vec + 4 * BT * 4 + 64;
  static_assert(fmat >= 2 * BT * 128, "two bf16 64x64 tiles fit in the fp32 inverse");
  static_assert((sizeof(float) * 32 * LDT) % 16 == 0, "vectors stay 16-byte aligned");
};

struct IntraMaps {
  CUtensorMap k, v, w, u, q, kn, qn;
};

// A21 = -A22 (L21 A11) for an N x N block below the diagonal whose corner is (r0, c0), T = L21 A11 going through a compact
// temporary (row stride LDT).  Both A11 and A22 are lower triangular.
// First product: a warp owns four columns of T (j0 ..), a lane a row: A11's row pieces are uniform over the warp, L21's rows
// are read in 16-byte words; rows m < j0 of A11 have only zeros in these columns.
// Second product: a warp owns four rows (i0 ..), a lane a column: A22's row pieces are uniform, T's rows are consecutive;
// columns m > i0 + 3 of A22 hold only zeros in these rows.
// N = 16: lanes 0-15 and 16-31 take halves of the contraction and add up at the end.
template <int N>
__device__ __forceinline__ void merge_step1(const float* Lf, const float* Af, float* T, int r0, int c0, int j0, int lane) {
  const int i = lane & (N - 1);
  const int m_beg = N == 32 ? j0 : (lane >> 4) * 8, m_end = N == 32 ? 32 : m_beg + 8;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
  for (int m = m_beg; m < m_end; m += 4) {
    const float4 l = *reinterpret_cast<const float4*>(&Lf[(r0 + i) * LDF + c0 + m]);
    const float ll[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float4 x = *reinterpret_cast<const float4*>(&Af[(c0 + m + e) * LDF + c0 + j0]);
      acc[0] += ll[e] * x.x; acc[1] += ll[e] * x.y; acc[2] += ll[e] * x.z; acc[3] += ll[e] * x.w;
    }
  }
  if (N == 16) {
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], 16);
    if (lane >= 16) return;
  }
  *reinterpret_cast<float4*>(&T[i * LDT + j0]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
}
template <int N>
__device__ __forceinline__ void merge_step2(const float* T, float* Af, int r0, int c0, int i0, int lane) {
  const int j = lane & (N - 1);
  const int m_beg = N == 32 ? 0 : (lane >> 4) * 8, m_end = N == 32 ? i0 + 4 : m_beg + 8;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
  for (int m = m_beg; m < m_end; m += 4) {
    float t[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) t[e] = T[(m + e) * LDT + j];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float4 x = *reinterpret_cast<const float4*>(&Af[(r0 + i0 + r) * LDF + r0 + m]);
      acc[r] += x.x * t[0] + x.y * t[1] + x.z * t[2] + x.w * t[3];
    }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    if (N == 16) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], 16);
    if (N == 32 || lane < 16) Af[(r0 + i0 + r) * LDF + c0 + j] = -acc[r];
  }
}

// L2-normalises the rows of a swizzled [64][DK] tile in place (four lanes per row), rounded to bf16; with `out` the rows also
// go to global memory and their reciprocal norms to `rstd`
template <int DK>
__device__ __forceinline__ void normalise_rows(unsigned char* tile, int tid, int len, float* rstd, int64_t rstride, __nv_bfloat16* out,
                                               int64_t ostride) {
  const int r = tid >> 2, seg = tid & 3;
  uint64_t x[DK / 32][4], s2[2] = {0ull, 0ull};   // pairs
  auto chunk = [&](int i) {   // the lane's i-th 16-byte word of the row
    const int c = seg + 4 * i;
    return reinterpret_cast<uint4*>(tile + (c >> 3) * (BT * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4));
  };
#pragma unroll
  for (int i = 0; i < DK / 32; ++i) {
    const uint4 w = *chunk(i);
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      x[i][e] = widen2<__nv_bfloat16>(u[e]);
      s2[e & 1] = fma2(x[i][e], x[i][e], s2[e & 1]);
    }
  }
  const float2 s = unpack2(add2(s2[0], s2[1]));
  float ss = s.x + s.y;
  ss += __shfl_xor_sync(0xffffffffu, ss, 1);
  ss += __shfl_xor_sync(0xffffffffu, ss, 2);
  const float y = 1.f / sqrtf(ss + 1e-6f);
  const uint64_t y2 = pack2(y, y);
  if (rstd != nullptr && seg == 0 && r < len) rstd[r * rstride] = y;
#pragma unroll
  for (int i = 0; i < DK / 32; ++i) {
    const uint4 w = make_uint4(narrow2<__nv_bfloat16>(mul2(x[i][0], y2)), narrow2<__nv_bfloat16>(mul2(x[i][1], y2)),
                               narrow2<__nv_bfloat16>(mul2(x[i][2], y2)), narrow2<__nv_bfloat16>(mul2(x[i][3], y2)));
    *chunk(i) = w;
    if (out != nullptr && r < len) *reinterpret_cast<uint4*>(out + r * ostride + (seg + 4 * i) * 8) = w;
  }
}

// the largest magnitude of three; NaN if one of them is
__device__ __forceinline__ float max_abs3(float a, float b, float c) {
  float d;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// a magnitude that is a finite bf16 when rounded (false for NaN)
__device__ __forceinline__ bool fits_bf16(float x) { return x <= 3.3895313892515355e38f; }

// BOUNDS: option TRANSITION_BOUNDS (an instantiation of its own: a small pass was 1 % slower with the branches alone)
template <int DK, int DV, bool BOUNDS>
__global__ void __launch_bounds__(NTHREADS, 4) intra_fwd_kernel(const b200gdn_chunk_args a, const __grid_constant__ IntraMaps maps,
                                                                const int pf_dist, const bool out_maps) {
  using S = IntraSmem<DK, DV>;
  constexpr int KB = DK / 64, VB = DV / 64;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  wait_for_predecessor();
  unsigned char* smem = smem_raw;
  if ((tc5::smem_addr(smem) & 1023u) != 0) {   // the swizzled tiles need it; never seen, but never silently wrong either
    if (threadIdx.x == 0) atomicExch(&g_intra_timeout, 2);
    return;
  }
  unsigned char* Ks = smem + S::o_k;      // later the W staging tile
  unsigned char* Vs = smem + S::o_l;      // after L; later the U staging tile
  float* Lf = reinterpret_cast<float*>(smem + S::o_l);
  float* Af = reinterpret_cast<float*>(smem + S::o_a);
  float* Tf = reinterpret_cast<float*>(smem + S::o_t);
  unsigned char* Aw = smem + S::o_a;      // after the fp32 inverse has been read into registers
  unsigned char* Au = Aw + BT * 128;
  float* gam = reinterpret_cast<float*>(smem + S::o_vec);
  float* bet = gam + BT;
  float* bge = bet + BT;
  float* graw = bge + BT;
  uint64_t* bar = reinterpret_cast<uint64_t*>(graw + BT);
  uint64_t* bar_k = bar + 1;
  uint64_t* bar_v = bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 3);

  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int q = warp & 3, hc = warp >> 2;
  const int g = lane >> 2, t = lane & 3;
  const int c = blockIdx.x, hv = blockIdx.y;
  const int G = a.HV / a.H, hq = hv / G;
  const ChunkMeta cm = load_chunk_meta(a.chunk_meta, c);
  const int64_t row0 = cm.row;
  const int r_lo = q * 16 + g, r_hi = r_lo + 8;
  const int cs = hc * 32;
  // with q and a qk buffer the kernel also emits the gated causal q k^T tile that the scans use for the chunk-local
  // parts of o and dv (so that they neither form nor mask it on their serial chain)
  const bool with_qk = a.qk != nullptr && a.q != nullptr;
  constexpr bool bounds = BOUNDS;
  unsigned char* Qs = smem + S::o_l;

  if (tid == 0) {
    tc5::mbar_init(bar, 1);
    tc5::mbar_init(bar_k, 1);
    tc5::mbar_init(bar_v, 1);
    tc5::fence_mbar_init();
    tc5::mbar_expect_tx(bar_k, (uint32_t)((with_qk ? 2 : 1) * BT * DK * 2));
    tma::load_3d(Ks, &maps.k, cm.row, (hq * DK) / 64, bar_k);
    if (with_qk) tma::load_3d(Qs, &maps.q, cm.row, (hq * DK) / 64, bar_k);   // lives where L will be written
    tma::prefetch_3d(&maps.v, cm.row, (hv * DV) / 64);   // V is loaded late (it reuses L's place): have it in L2 by then
  }
  if (warp == 1) tc5::tmem_alloc(tmem_slot, 128);
  // the gates of this thread's token: the loads are issued here and first used behind the barrier below
  float g_raw = 0.f, b_raw = 0.f;
  if (tid < cm.len) {
    g_raw = ld_param(a.g, (row0 + tid) * a.HV + hv, a.gb_dtype);
    b_raw = ld_param(a.beta, (row0 + tid) * a.HV + hv, a.gb_dtype);
  }
  tc5::fence_before_sync();
  __syncthreads();
  tc5::fence_after_sync();
  const uint32_t tm = *tmem_slot;
  PhaseBarrier ph{bar, 0u, &g_intra_timeout};
  bool failed = false;

  if (tid < BT) {
    // inclusive scan of g over the chunk: shuffle scan inside each of the two warps, carry added below
    if (a.options != 0 && tid < cm.len) {   // the layer's gate / beta activations, fused (rows past the end stay 0)
      if (a.options & B200GDN_PREP_GATE) {
        const float x = g_raw + (a.dt_bias ? a.dt_bias[hv] : 0.f);
        g_raw = -expf(a.A_log[hv]) * (x > 20.f ? x : log1pf(expf(x)));
      }
      if (a.options & B200GDN_PREP_BETA_SIGMOID)
        b_raw = ((a.options & B200GDN_PREP_NEG_EIGVAL) ? 2.f : 1.f) / (1.f + expf(-b_raw));
    }
    bet[tid] = b_raw;
    float s = g_raw;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    gam[tid] = s;
  }
  if (tid == 128) {   // while everybody waits for the K tile
    int c2, h2;
    if (successor_cta(pf_dist, c2, h2)) {   // L2 look-ahead for the CTA that will follow this one
      const int row2 = load_chunk_meta(a.chunk_meta, c2).row;
      tma::prefetch_3d(&maps.k, row2, ((h2 / G) * DK) / 64);
      // g and beta of a chunk are [64][HV] blocks: the HV CTAs of a chunk pull (up to) two lines each
      const int gb_bytes = a.gb_dtype == B200GDN_F32 ? 4 : 2, lines = BT * a.HV * gb_bytes / 128;
      for (int l = h2 * 2; l < h2 * 2 + 2 && l < lines; ++l) {
        tma::prefetch_line(static_cast<const char*>(a.g) + (int64_t)row2 * a.HV * gb_bytes + l * 128);
        tma::prefetch_line(static_cast<const char*>(a.beta) + (int64_t)row2 * a.HV * gb_bytes + l * 128);
      }
    }
  }
  if (!tc5::mbar_wait(bar_k, 0)) failed = true;
  if (cm.len < BT) {
    zero_tail_rows<BT, DK>(Ks, cm.len, tid, NTHREADS);
    tc5::fence_async_smem();
  }
  if ((a.options & B200GDN_PREP_L2NORM) && !failed) {   // q and k are the raw tensors; the scans read the normalised ones
    const bool lead = hv % G == 0;   // one of the value heads that share these q and k
    const bool rows_out = lead && !(out_maps && cm.len == BT);   // whole tiles leave by TMA below
    const int64_t at = row0 * a.H + hq, st = (int64_t)a.H * DK;
    if (cm.len < BT) __syncthreads();   // the zeroed tail of K
    normalise_rows<DK>(Ks, tid, cm.len, lead && a.rstd_k ? a.rstd_k + at : nullptr, a.H,
                       rows_out ? reinterpret_cast<__nv_bfloat16*>(a.kn) + at * DK : nullptr, st);
    if (with_qk) normalise_rows<DK>(Qs, tid, cm.len, lead && a.rstd_q ? a.rstd_q + at : nullptr, a.H,
                                    rows_out ? reinterpret_cast<__nv_bfloat16*>(a.qn) + at * DK : nullptr, st);
    tc5::fence_async_smem();
  }
  if (__syncthreads_or(failed)) {
    failed = true;
  } else {
    if (warp == 0) {
      tc5::fence_after_sync();
      issue_mma_t<DK / 16>(tm, Operand{tc5::smem_addr(Ks), BT, 0}, Operand{tc5::smem_addr(Ks), BT, 0}, 64, 64, 0);
      if (with_qk) issue_mma_t<DK / 16>(tm + 64, Operand{tc5::smem_addr(Qs), BT, 0}, Operand{tc5::smem_addr(Ks), BT, 0}, 64, 64, 0);
      ph.commit();
    }
    const bool tiles_out = out_maps && hv % G == 0 && cm.len == BT;
    if (tiles_out && tid == 32) {   // the normalised tiles leave while the products run
      if (with_qk) tma::store_3d(&maps.qn, (int)cm.row, (hq * DK) / 64, Qs);
      tma::store_3d(&maps.kn, (int)cm.row, (hq * DK) / 64, Ks);
      tma::store_commit();
    }
    if (tid < BT) graw[tid] = (gam[tid] + (tid >= 32 ? gam[31] : 0.f)) * 1.4426950216f;
    __syncthreads();
    if (tid < BT) {
      // entries past a ragged chunk's end repeat the last valid value exactly (the scan sums zeros there, but in an
      // order that depends on the lane, so its result may differ in the last bit)
      const float gm = graw[tid < cm.len ? tid : cm.len - 1];
      gam[tid] = gm;
      bge[tid] = bet[tid] * fast_exp2(gm);
      a.gamma[((int64_t)c * a.HV + hv) * BT + tid] = gm;   // padded rows carry the last valid value (their g is 0)
    }
    if (tiles_out && tid == 32) tma::store_wait_read<0>();   // L takes the place of q
    if (!ph.sync_wait()) failed = true;
  }

  if (!failed) {
    // ---- L = strict_tril(beta_i <k_i,k_j> 2^(gamma_i - gamma_j)) in fp32 (over the Q tile, which is dead by now), and
    //      qk = tril(<q_i,k_j> 2^(gamma_i - gamma_j)) with the same gate factors, as bf16 straight to global memory
    //      (rows past a ragged chunk's end are another sequence's rows and are not written)
    {
      __nv_bfloat16* Pg = reinterpret_cast<__nv_bfloat16*>(a.qk) + (row0 * a.HV + hv) * BT + cs + 8 * t;
      const int64_t pstride = (int64_t)a.HV * BT;
      if (q * 16 + 15 >= cs) {   // a block entirely above the diagonal is never read by the solve and is zero in qk
        float r[16], pq[16];
        acc_ld32q(tm, q, cs, r);
        if (with_qk) acc_ld32q(tm + 64, q, cs, pq);
        tc5::tmem_ld_wait();
        const float g_lo = gam[r_lo], g_hi = gam[r_hi];
        const float b_lo = bet[r_lo], b_hi = bet[r_hi];
        uint32_t p_lo[4], p_hi[4];
        float2 qk_lo[4], qk_hi[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int j0 = cs + i * 8 + 2 * t;
          const float2 gj = *reinterpret_cast<const float2*>(&gam[j0]);
          float v[4], w4[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int ii = (e & 2) ? r_hi : r_lo, jj = j0 + (e & 1);
            const float f = fast_exp2(((e & 2) ? g_hi : g_lo) - ((e & 1) ? gj.y : gj.x));
            v[e] = (ii > jj) ? r[4 * i + e] * ((e & 2) ? b_hi : b_lo) * f : 0.f;
            w4[e] = (with_qk && ii >= jj) ? pq[4 * i + e] * f : 0.f;
          }
          *reinterpret_cast<float2*>(&Lf[r_lo * LDF + j0]) = make_float2(v[0], v[1]);
          *reinterpret_cast<float2*>(&Lf[r_hi * LDF + j0]) = make_float2(v[2], v[3]);
          p_lo[i] = pack_bf16(w4[0], w4[1]);
          p_hi[i] = pack_bf16(w4[2], w4[3]);
          qk_lo[i] = make_float2(w4[0], w4[1]);
          qk_hi[i] = make_float2(w4[2], w4[3]);
        }
        if (bounds) {
          float kk_lo = 0.f, kk_hi = 0.f;   // |k|^2 of the two rows, where the diagonal is this thread's
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const int jj = cs + (e >> 2) * 8 + 2 * t + (e & 1);
            if ((e & 2) && jj == r_hi) kk_hi = r[e];
            if (!(e & 2) && jj == r_lo) kk_lo = r[e];
          }
          float x = log2f(fmaxf(1.f, fabsf(1.f - b_lo * kk_lo))) + log2f(fmaxf(1.f, fabsf(1.f - b_hi * kk_hi)));
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
          // a value of q that is not finite makes its row's product with k, at least the one on the diagonal, not finite either
          float s_lo = 0.f, s_hi = 0.f;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            s_lo = max_abs3(s_lo, qk_lo[i].x, qk_lo[i].y);
            s_hi = max_abs3(s_hi, qk_hi[i].x, qk_hi[i].y);
          }
          const bool odd = __any_sync(0xffffffffu, (r_lo < cm.len && !fits_bf16(s_lo)) || (r_hi < cm.len && !fits_bf16(s_hi)));
          if (lane == 0) {   // (the raw sums have been read)
            graw[warp] = x;
            graw[NTHREADS / 32 + warp] = odd;
          }
        }
        if (with_qk) {
          const uint4 lo = quad_words(p_lo, t), hi = quad_words(p_hi, t);
          if (r_lo < cm.len) *reinterpret_cast<uint4*>(Pg + r_lo * pstride) = lo;
          if (r_hi < cm.len) *reinterpret_cast<uint4*>(Pg + r_hi * pstride) = hi;
        }
      } else {
        if (bounds && lane == 0) graw[warp] = graw[NTHREADS / 32 + warp] = 0.f;
        if (with_qk && r_lo < cm.len) *reinterpret_cast<uint4*>(Pg + r_lo * pstride) = make_uint4(0, 0, 0, 0);
        if (with_qk && r_hi < cm.len) *reinterpret_cast<uint4*>(Pg + r_hi * pstride) = make_uint4(0, 0, 0, 0);
      }
    }
    tc5::fence_before_sync();
    __syncthreads();

    // ---- four 16x16 diagonal inverses, one per warp: lane cc (and its copy cc + 16) solves (I + L_bb) x = e_cc row by row;
    //      the rows of L_bb are uniform over the warp and do not depend on the chain, so their loads run ahead of it
    if (warp < 4) {
      const int b0 = warp * 16, cc = lane & 15;
      float s[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float x0 = (i == cc) ? 1.f : 0.f, x1 = 0.f;
#pragma unroll
        for (int j = 0; j < i; j += 4) {
          const float4 l = *reinterpret_cast<const float4*>(&Lf[(b0 + i) * LDF + b0 + j]);
          x1 -= l.x * s[j];
          if (j + 1 < i) x0 -= l.y * s[j + 1];
          if (j + 2 < i) x1 -= l.z * s[j + 2];
          if (j + 3 < i) x0 -= l.w * s[j + 3];
        }
        s[i] = x0 + x1;
        if (lane < 16) Af[(b0 + i) * LDF + b0 + cc] = s[i];
      }
    }
    __syncthreads();
    // ---- 16 -> 32: blocks (16,0) and (48,32), four warps each
    merge_step1<16>(Lf, Af, Tf + (warp >> 2) * 16, hc ? 48 : 16, hc ? 32 : 0, 4 * q, lane);
    __syncthreads();
    merge_step2<16>(Tf + (warp >> 2) * 16, Af, hc ? 48 : 16, hc ? 32 : 0, 4 * q, lane);
    __syncthreads();
    // ---- 32 -> 64: block (32,0), all warps
    merge_step1<32>(Lf, Af, Tf, 32, 0, 4 * warp, lane);
    __syncthreads();
    // L is dead: its place takes the V tile while the last merge step and the conversion run
    if (tid == 0) {
      tc5::fence_async_smem();
      tc5::mbar_expect_tx(bar_v, (uint32_t)(BT * DV * 2));
      tma::load_3d(Vs, &maps.v, cm.row, (hv * DV) / 64, bar_v);
    }
    merge_step2<32>(Tf, Af, 32, 0, 4 * warp, lane);
    __syncthreads();

    // ---- bf16 operand tiles (over the fp32 inverse and the merge temporary, hence through registers):
    //      A with its columns scaled for the W and U right-hand sides, and A itself
    {   // every warp converts its own 16 x 32 block (rows 16 q .., columns cs ..) in the accumulator-fragment layout
      float2 x_lo[4], x_hi[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int col = cs + i * 8 + 2 * t;
        x_lo[i] = *reinterpret_cast<const float2*>(&Af[r_lo * LDF + col]);
        x_hi[i] = *reinterpret_cast<const float2*>(&Af[r_hi * LDF + col]);
        // above the diagonal only the 16x16 diagonal blocks have been written
        if (col > r_lo) x_lo[i].x = 0.f;
        if (col + 1 > r_lo) x_lo[i].y = 0.f;
        if (col > r_hi) x_hi[i].x = 0.f;
        if (col + 1 > r_hi) x_hi[i].y = 0.f;
      }
      __syncthreads();
      FragStore fw, fu, fa;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int col = cs + i * 8 + 2 * t;
        const float2 sw = *reinterpret_cast<const float2*>(&bge[col]), su = *reinterpret_cast<const float2*>(&bet[col]);
        fw.set(i, x_lo[i].x * sw.x, x_lo[i].y * sw.y, x_hi[i].x * sw.x, x_hi[i].y * sw.y);
        fu.set(i, x_lo[i].x * su.x, x_lo[i].y * su.y, x_hi[i].x * su.x, x_hi[i].y * su.y);
        fa.set(i, x_lo[i].x, x_lo[i].y, x_hi[i].x, x_hi[i].y);
      }
      fw.store(Aw, BT, q * 16, cs, lane);
      fu.store(Au, BT, q * 16, cs, lane);
      // A itself goes straight to global memory, 64 contiguous bytes per row and quad
      __nv_bfloat16* Ag = reinterpret_cast<__nv_bfloat16*>(a.A) + (row0 * a.HV + hv) * BT + cs + 8 * t;
      const int64_t astride = (int64_t)a.HV * BT;
      if (!(a.options & B200GDN_FORWARD_ONLY)) {
        const uint4 lo = quad_words(fa.lo, t), hi = quad_words(fa.hi, t);
        if (r_lo < cm.len) *reinterpret_cast<uint4*>(Ag + r_lo * astride) = lo;
        if (r_hi < cm.len) *reinterpret_cast<uint4*>(Ag + r_hi * astride) = hi;
      }
    }
    tc5::fence_async_smem();
    tc5::fence_before_sync();
    __syncthreads();

    // ---- W = Aw K   (K as an MN-major B operand: contraction over the token rows)
    if (warp == 0) {
      tc5::fence_after_sync();
      issue_mma_t<BT / 16>(tm, Operand{tc5::smem_addr(Aw), BT, 0}, Operand{tc5::smem_addr(Ks), BT, 1}, 64, DK, 0);
      ph.commit();
    }
    if (!tc5::mbar_wait(bar_v, 0)) failed = true;
    if (cm.len < BT) {
      zero_tail_rows<BT, DV>(Vs, cm.len, tid, NTHREADS);
      tc5::fence_async_smem();
    }
    if (!ph.sync_wait(failed)) {
      failed = true;
    } else {
      const int ck = hc * (DK / 2), cv = hc * (DV / 2);
      float rw[KB][16];
#pragma unroll
      for (int b = 0; b < KB; ++b) acc_ld32q(tm, q, ck + b * 32, rw[b]);
      tc5::tmem_ld_wait();
      tc5::fence_before_sync();
      __syncthreads();   // W has left tensor memory, K is no longer an operand
      float size = 0.f;   // the largest of this thread's part of W and U; NaN if one of them is
      if (bounds) {
#pragma unroll
        for (int b = 0; b < KB; ++b)
#pragma unroll
          for (int e = 0; e < 16; e += 2) size = max_abs3(size, rw[b][e], rw[b][e + 1]);
      }
      // ---- U = Au V into the same columns, while W is converted and staged over the K tile
      if (warp == 0) {
        tc5::fence_after_sync();
        issue_mma_t<BT / 16>(tm, Operand{tc5::smem_addr(Au), BT, 0}, Operand{tc5::smem_addr(Vs), BT, 1}, 64, DV, 0);
        ph.commit();
      }
#pragma unroll
      for (int b = 0; b < KB; ++b) {
        FragStore fs;
#pragma unroll
        for (int i = 0; i < 4; ++i) fs.set(i, rw[b][4 * i], rw[b][4 * i + 1], rw[b][4 * i + 2], rw[b][4 * i + 3]);
        fs.store(Ks, BT, q * 16, ck + b * 32, lane);
      }
      tc5::fence_async_smem();
      if (!ph.sync_wait()) {
        failed = true;
      } else {
        if (cm.len == BT) {
          if (tid == 32) {
            tma::store_3d(&maps.w, (int)cm.row, (hv * DK) / 64, Ks);
            tma::store_commit();
          }
        } else {
          store_tile_swz<BT, DK, NTHREADS>(reinterpret_cast<__nv_bfloat16*>(a.w) + (row0 * a.HV + hv) * DK, (int64_t)a.HV * DK,
                                           Ks, cm.len, tid);
        }
        float ru[VB][16];
#pragma unroll
        for (int b = 0; b < VB; ++b) acc_ld32q(tm, q, cv + b * 32, ru[b]);
        tc5::tmem_ld_wait();
        if (bounds) {
#pragma unroll
          for (int b = 0; b < VB; ++b)
#pragma unroll
            for (int e = 0; e < 16; e += 2) size = max_abs3(size, ru[b][e], ru[b][e + 1]);
        }
#pragma unroll
        for (int b = 0; b < VB; ++b) {
          FragStore fs;
#pragma unroll
          for (int i = 0; i < 4; ++i) fs.set(i, ru[b][4 * i], ru[b][4 * i + 1], ru[b][4 * i + 2], ru[b][4 * i + 3]);
          fs.store(Vs, BT, q * 16, cv + b * 32, lane);
        }
        tc5::fence_async_smem();
        tc5::fence_before_sync();
        int odd = 0;
        if (bounds) odd = __syncthreads_or(!fits_bf16(size));
        else __syncthreads();
        if (bounds && tid == 0) {
          float x = gam[BT - 1], q_odd = 0.f;
#pragma unroll
          for (int w = 0; w < NTHREADS / 32; ++w) {
            x += graw[w];
            q_odd += graw[NTHREADS / 32 + w];
          }
          bounds_ptr(a.gamma, a.n_chunks, a.HV)[(int64_t)c * a.HV + hv] = odd ? INFINITY : tagged_bound(x, q_odd != 0.f);
        }
        if (cm.len == BT) {
          if (tid == 32) {
            tma::store_3d(&maps.u, (int)cm.row, (hv * DV) / 64, Vs);
            tma::store_commit();
          }
        } else {
          store_tile_swz<BT, DV, NTHREADS>(reinterpret_cast<__nv_bfloat16*>(a.u) + (row0 * a.HV + hv) * DV, (int64_t)a.HV * DV,
                                           Vs, cm.len, tid);
        }
      }
    }
  }
  if (tid == 32) tma::store_wait_all<0>();   // shared memory must outlive the bulk stores that read it
  if (failed && tid == 0) atomicExch(&g_intra_timeout, 1);
  tc5::fence_before_sync();
  __syncthreads();
  if (warp == 1) tc5::tmem_dealloc(tm, 128);
}

template <int DK, int DV, bool BOUNDS>
int launch(const b200gdn_chunk_args& a, cudaStream_t st) {
  using S = IntraSmem<DK, DV>;
  if (int e = ensure_smem(intra_fwd_kernel<DK, DV, BOUNDS>, S::bytes)) return e;
  IntraMaps m;
  const uint64_t pk = (uint64_t)a.H * DK, pw = (uint64_t)a.HV * DK, pv = (uint64_t)a.HV * DV;
  int rc = 0;
  rc |= tma::encode_bf16_panels(&m.k, a.k, a.rows, pk, pk, BT, DK / 64);
  rc |= tma::encode_bf16_panels(&m.v, a.v, a.rows, pv, pv, BT, DV / 64);
  rc |= tma::encode_bf16_panels(&m.w, a.w, a.rows, pw, pw, BT, DK / 64);
  rc |= tma::encode_bf16_panels(&m.u, a.u, a.rows, pv, pv, BT, DV / 64);
  if (a.q) rc |= tma::encode_bf16_panels(&m.q, a.q, a.rows, pk, pk, BT, DK / 64); else m.q = m.k;
  m.kn = m.qn = m.k;
  const bool out_maps = (a.options & B200GDN_PREP_L2NORM) && !overlaps(a);   // (small problems wait for the host, and a map costs it 0.6 us)
  if (out_maps) {
    rc |= tma::encode_bf16_panels(&m.kn, a.kn, a.rows, pk, pk, BT, DK / 64);
    rc |= tma::encode_bf16_panels(&m.qn, a.qn, a.rows, pk, pk, BT, DK / 64);
  }
  if (rc != 0) return set_error(B200GDN_ERR_CUDA, "intra_fwd: cuTensorMapEncodeTiled failed (%d)", rc);
  dim3 grid(a.n_chunks, a.HV);
  launch_overlapped(overlaps(a), intra_fwd_kernel<DK, DV, BOUNDS>, grid, NTHREADS, S::bytes, st, a, m, resident_ctas<intra_fwd_kernel<DK, DV, BOUNDS>>(NTHREADS, S::bytes), out_maps);
  return check_launch("intra_fwd");
}

}  // namespace

int launch_intra_fwd(const b200gdn_chunk_args& a, cudaStream_t st) {
  if ((a.options & B200GDN_PREP_GATE) && a.A_log == nullptr)
    return set_error(B200GDN_ERR_BAD_ARGUMENT, "intra_fwd: the fused gate needs A_log");
  if ((a.options & B200GDN_PREP_L2NORM) && (a.qn == nullptr || a.kn == nullptr))
    return set_error(B200GDN_ERR_BAD_ARGUMENT, "intra_fwd: the fused L2 norm needs qn and kn");
  const bool bounds = a.options & B200GDN_TRANSITION_BOUNDS;
  if (a.K == 128 && a.V == 128) return bounds ? launch<128, 128, true>(a, st) : launch<128, 128, false>(a, st);
  if (a.K == 64 && a.V == 64) return bounds ? launch<64, 64, true>(a, st) : launch<64, 64, false>(a, st);
  return set_error(B200GDN_ERR_UNSUPPORTED, "intra_fwd: K=%d V=%d not built (64/64 and 128/128 are)", a.K, a.V);
}

// Reads and clears the flag a bounded device wait raises when it expires (synchronises with the device).
int intra_fwd_timeout_flag() {
  int v = 0, zero = 0;
  cudaMemcpyFromSymbol(&v, g_intra_timeout, sizeof(int));
  if (v) cudaMemcpyToSymbol(g_intra_timeout, &zero, sizeof(int));
  return v;
}

}  // namespace gdn
