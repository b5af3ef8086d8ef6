// Everything of the backward pass that is local to a chunk, in one kernel per (chunk, value head): the gradients of q, k, v,
// the gate and beta from the tensors the two scans left.  Replaces chunk_bwd_kernel_dqkwg
// (fla/ops/common/chunk_o.py:172-342), prepare_wy_repr_bwd_kernel (fla/ops/gated_delta_rule/wy_fast.py:123-251) and the
// reverse chunk-local cumsum of dg (gated_delta_rule/chunk.py:244-246).
//
// With X the right-hand side of v_new = A X (X_i = beta_i (v_i - 2^gamma_i S^T k_i), A = (I + L)^-1), the adjoint of the triangular
// solve is Z = A^T dv_new, dX = Z, dL = -strict_tril(Z v_new^T): one product each, where dA = dv_new X^T and -A^T dA A^T through
// dW and dU took four in sequence (and rounded each of them to bf16).
//     Z    = A^T dU      dU = dv2                                   dP   = tril(do v_new^T 2^(gamma_i - gamma_j)) scale
//     dq^T = h do_s^T + K^T dP^T                                    do_s = do scale 2^gamma_i
//     M    = -strict_tril(Z v_new^T) 2^(gamma_i - gamma_j)          M2   = M beta_i
//     dk^T = (dh v_new^T) 2^(gamma_last - gamma_j) + q^T dP - (h Z^T) (beta 2^gamma)_j + K^T M2^T + K^T M2
//     dv   = beta Z
//     dbeta= c_kz 2^gamma + <Z_i,v_i> + r_mk,   c_kz_i = -<h Z_i, k_i>,  r_mk = rowsum(M . K K^T)
//     dG_i = <dq_i,q_i> - <dk_loc_i,k_i> + c_kz beta 2^gamma + beta r_mk - c_mk
//            (+ at the last valid row: 2^gamma_last <h,dh> + sum_j <dk_state_j, k_j>):     dg = reverse cumsum of dG
// with dk_loc the first two terms of dk, <dk_loc_j,k_j> = <dk_state_j,k_j> + colsum(dP . Q K^T)_j, c_mk = colsum(M2 . K K^T).
// (The other terms of dk contribute c_kz beta 2^gamma + beta r_mk + c_mk to <dk_i,k_i>, so dG could be had from the finished dk
// without Q K^T and c_mk; but then the bf16 operands of those terms do not cancel against the fp32 sums, and the sums of dg
// over a sequence, dA_log and ddt_bias, were twice as far from fp64 as with the terms kept apart: 0.016 against 0.008.
// Likewise dbeta = <Z_i, v_new_i> / beta_i, but v_new has been rounded as a difference: 0.0034 from fp64 against 0.0022.)
//
// Products with a K- or V-wide result are formed TRANSPOSED ([K x 64 tokens], M = 128): the same tcgen05 instruction then does
// twice the work of an M = 64 one, an accumulator takes 64 TMEM columns instead of 128, and every lane of a TMEM load carries
// data.  dq, dk and dv go through a shared tile (stmatrix with a transpose) and leave by TMA.  <h,dh> is the diagonal of h dh^T in
// 16 x 16 blocks by mma.sync, straight from the bf16 tiles: a tenth of the instructions of unpacking and multiplying.
// What bounds it is the latency of the phases at two CTAs per SM, i.e. the instructions of an epilogue (39 % of issue slots, DRAM
// 54 % of its peak rate), so epilogues work on fp32 pairs and skip blocks above the diagonal.
// The CTAs of a chunk are neighbours in launch order: a row of q, k, v or do is then read as a whole at about one time, which DRAM
// pages like better than 256 bytes of every row (chunks first: 187 us for 179, grouped heads in turn 226 for 217 at the time).  Pulling the
// next head's tiles into L2 while a head is worked on was slower (244 for 226).
// B4 T4096 H16 K=V=128: 179 us inside a step (228 with the solve's adjoint by way of dW, dU and dA, six dependent tensor-core phases
// where there are three now; 213 with three, but element-wise stores and scalar epilogues); 8/16 heads 201 (242; 217 with the load of dh waiting for the copy of dv to leave at once).
// One CTA of eight warps; 256 TMEM columns (C0: dP, dq^T, K K^T; C1: Z v_new^T, Q K^T; C2: Z^T; C3: dk_state^T, h Z^T, the rest of
// dk^T) and ~111 KiB of shared memory whose regions change hands, so two CTAs per SM overlap each other's phases:
//   R1: K   R2: do -> q   R3: v_new -> V   R4: dU -> Z^T -> dq   R5: dh -> h -> M2 | dv -> dk | dv   R6: A -> dP
// Grouped value heads, many chunks: a CTA takes the heads of a group in turn, K stays, the tiles of the next head are fetched
// under the last epilogue; the sum of dq waits in C1 (Z in registers and Z v_new^T in C2 instead), that of dk in local memory (TMEM
// is full; 32 KiB per CTA that stay in L2).
// Few chunks: a CTA per head, the CTAs of a group form a cluster; each leaves its fp32 dq and dk in shared memory and adds up
// a share of the rows over distributed shared memory.  Both add in head order (no atomics, no fp32 tensors in HBM).
#include "rowio.cuh"
#include "tc5_tile.cuh"
#include "tma.cuh"

namespace gdn {
namespace {

constexpr int NTHREADS = 256;
__device__ int g_local_timeout = 0;

template <int DK>
struct LocalSmem {
  static constexpr size_t tile = BT * DK * 2;                       // [64][DK] bf16 = [DK][64] bf16
  static constexpr size_t o_k = 0, o_do = tile, o_vn = 2 * tile, o_z = 3 * tile, o_h = 4 * tile;
  static constexpr size_t h_bytes = DK * 128 + (DK * 128 > tile ? DK * 128 : tile);   // h; later M2 (then dk) | dv
  static_assert(h_bytes >= DK * DK * 2, "every panel of h fits");
  static constexpr size_t o_a = o_h + h_bytes;
  static constexpr size_t o_vec = o_a + BT * 128;
  static constexpr int LDS = DK + 4;                                // fp32 row stride of the group-sum staging
  static constexpr size_t stage = (size_t)BT * LDS * 4;             // dq, then dk, from R2 on
  static constexpr size_t bytes = o_vec + 29 * BT * 4 + 160 + 1024; // + vectors, barriers, alignment slack
  static_assert(o_do + 2 * stage <= o_vec, "the group-sum staging fits over the dead tiles");
};

struct LocalMaps {
  CUtensorMap q, k, v, d_o, vn, du, a, h, dh, dq, dk, dv;
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
// ... tokens cs + 8 i + 2 t + {0, 1} of it times a factor per token; the same added to another block
template <int NH>
__device__ __forceinline__ void scale_t(float (&r)[NH][16], int i, float2 f) {
  const uint64_t f2 = pack2(f.x, f.y);
#pragma unroll
  for (int hf = 0; hf < NH; ++hf)
#pragma unroll
    for (int e = 4 * i; e < 4 * i + 4; e += 2) {
      const float2 x = unpack2(mul2(pack2(r[hf][e], r[hf][e + 1]), f2));
      r[hf][e] = x.x;
      r[hf][e + 1] = x.y;
    }
}
template <int NH>
__device__ __forceinline__ void scale_add_t(float (&to)[NH][16], const float (&r)[NH][16], int i, float2 f) {
  const uint64_t f2 = pack2(f.x, f.y);
#pragma unroll
  for (int hf = 0; hf < NH; ++hf)
#pragma unroll
    for (int e = 4 * i; e < 4 * i + 4; e += 2) {
      const float2 x = unpack2(fma2(pack2(r[hf][e], r[hf][e + 1]), f2, pack2(to[hf][e], to[hf][e + 1])));
      to[hf][e] = x.x;
      to[hf][e + 1] = x.y;
    }
}
// ... its dot products with the same block of a [token][column] tile, added over the rows: value 2 i + p of the result
// belongs to token 8 i + 2 t + p and still has to be summed over g
template <int NH>
__device__ __forceinline__ void dots_t(const float (&r)[NH][16], const unsigned char* tile, int row0, int cs, int lane, float (&pv)[8]) {
  uint64_t p2[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
  for (int hf = 0; hf < NH; ++hf) {
    FragLoadT f;
    f.load(tile, BT, cs, row0 + 16 * hf, lane);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      p2[i] = fma2(pack2(r[hf][4 * i], r[hf][4 * i + 1]), widen2<__nv_bfloat16>(f.lo[i]), p2[i]);
      p2[i] = fma2(pack2(r[hf][4 * i + 2], r[hf][4 * i + 3]), widen2<__nv_bfloat16>(f.hi[i]), p2[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 x = unpack2(p2[i]);
    pv[2 * i] = x.x;
    pv[2 * i + 1] = x.y;
  }
}
// ... and its way into a token-major bf16 tile
template <int NH>
__device__ __forceinline__ void stage_t(const float (&r)[NH][16], unsigned char* tile, int row0, int cs, int lane) {
#pragma unroll
  for (int hf = 0; hf < NH; ++hf) {
    FragStore fs;
#pragma unroll
    for (int i = 0; i < 4; ++i) fs.set(i, r[hf][4 * i], r[hf][4 * i + 1], r[hf][4 * i + 2], r[hf][4 * i + 3]);
    fs.store_trans(tile, BT, cs, row0 + 16 * hf, lane);
  }
}
// ... and to and from local memory (written out: as an array the compiler would hold it in registers)
template <int NH>
__device__ __forceinline__ void st_local(const float (&r)[NH][16], uint64_t at) {
#pragma unroll
  for (int e = 0; e < NH * 4; ++e)
    asm volatile("st.local.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(at + 16 * e), "f"(r[e / 4][4 * (e % 4)]), "f"(r[e / 4][4 * (e % 4) + 1]),
                 "f"(r[e / 4][4 * (e % 4) + 2]), "f"(r[e / 4][4 * (e % 4) + 3])
                 : "memory");
}
template <int NH>
__device__ __forceinline__ void add_local(float (&r)[NH][16], uint64_t at) {
  float x[NH][16];
#pragma unroll
  for (int e = 0; e < NH * 4; ++e)
    asm volatile("ld.local.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                 : "=f"(x[e / 4][4 * (e % 4)]), "=f"(x[e / 4][4 * (e % 4) + 1]), "=f"(x[e / 4][4 * (e % 4) + 2]), "=f"(x[e / 4][4 * (e % 4) + 3])
                 : "l"(at + 16 * e)
                 : "memory");
  add_t<NH>(r, x);
}

// 16 x 16 block `b` (row blocks first) of a swizzled [rows][rows] bf16 tile: words {rows 0-7, 8-15} x {columns 0-7, 8-15} in the order
// of the first operand of mma.m16n8k16; words {0, 2} and {1, 3} are the second operand for the block's rows 0-7 and 8-15
__device__ __forceinline__ void load_block16(uint32_t tile, int rows, int b, int lane, uint32_t (&x)[4]) {
  const int per_row = rows / 16;
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];\n"
               : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3])
               : "r"(tile + tc5::swz_offset((b / per_row) * 16 + (lane & 15), (b % per_row) * 16 + 8 * (lane >> 4), rows))
               : "memory");
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
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
__global__ void __launch_bounds__(NTHREADS, 2) bwd_local_kernel(const b200gdn_chunk_args a, const __grid_constant__ LocalMaps maps,
                                                                const bool out_maps) {
  constexpr bool GROUPED = MODE == kCluster, TURNS = MODE == kTurns;
  using S = LocalSmem<DK>;
  constexpr int NP = DK / 64;   // 64-column panels of a V-wide tile (V = K)
  constexpr int NH = DK / 64;   // 16-row halves of a transposed accumulator per warp
  extern __shared__ unsigned char smem_raw[];
  wait_for_predecessor();
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char *Ks = smem + S::o_k, *Do = smem + S::o_do, *Qs = Do, *Vn = smem + S::o_vn, *Vs = Vn, *dUs = smem + S::o_z, *Zt = dUs;
  unsigned char *Hs = smem + S::o_h, *M2s = Hs, *Dks = Hs, *Dvs = Hs + DK * 128, *Dqs = Zt, *As = smem + S::o_a, *Ps = As;
  float* const gs2 = reinterpret_cast<float*>(smem + S::o_vec);   // [2][64]: a head's and the next one's
  float *bet = gs2 + 2 * BT, *bge = bet + BT, *eg = bge + BT, *sgm = eg + BT, *gx = sgm + BT, *gv = gx + BT, *dGs = gv + BT, *rsq = dGs + BT, *rsk = rsq + BT;
  // sums over rows: each of the four row-quadrant warps leaves its partial in its own slot and the consumer adds the four in
  // a fixed order (no atomics: results are bit-reproducible)
  float* c_rq = rsk + BT;        // [4][64] <dq_i, q_i>
  float* c_rk = c_rq + 4 * BT;   // [4][64] <dk_loc_i, k_i> + c_mk
  float* c_kz = c_rk + 4 * BT;   // [4][64] -<h Z_i, k_i>
  float* c_vb = c_kz + 4 * BT;   // [4][64] <Z_i, v_i>
  float* r_mk = c_vb + 4 * BT;   // [2][64] rowsum(M . K K^T), two column halves
  float* red = r_mk + 2 * BT;    // [0..7] <h,dh> per warp, [8..15] sum of <dk_state, k> per warp, [16..19] gate sums
  uint64_t* bar = reinterpret_cast<uint64_t*>(red + 20);
  uint64_t *bar_a = bar + 1, *bar_b = bar + 2, *bar_c = bar + 3;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 4);

  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int q = warp & 3, hc = warp >> 2, g = lane >> 2, t = lane & 3;
  const int per_chunk = TURNS ? a.H : a.HV, c = blockIdx.x / per_chunk, head = blockIdx.x % per_chunk;
  const int G = a.HV / a.H, hq = TURNS ? head : head / G;
  const int hv0 = TURNS ? hq * G : head, n_heads = TURNS ? G : 1;
  const ChunkMeta cm = load_chunk_meta(a.chunk_meta, c);
  const int64_t row0 = cm.row;
  const bool by_tma = cm.len == BT && out_maps;   // how dq, dk and dv leave
  const int r_lo = q * 16 + g, r_hi = r_lo + 8, cs = hc * 32;   // this warp's block of a [64][64] tile
  const int kr = (DK / 4) * q;                                  // ... and its first row of a transposed accumulator
  const bool live = q * 16 + 15 >= cs;                          // some of that block is on or below the diagonal
  const int gcol = cs + 8 * (g >> 1) + 2 * t + (g & 1);         // the column whose sum sum8_over_g leaves in this lane

  auto load_dh = [&](int hv) {
    for (int p = 0; p < NP; ++p) tma::load_2d(Hs + p * DK * 128, &maps.dh, p * 64, (c * a.HV + hv) * DK, bar_a);
  };
  // one thread: what a head's first phase needs, and the rest into L2
  auto load_head = [&](int hv, bool first) {
    const int hrow = (c * a.HV + hv) * DK;   // the head's state snapshot in the [.., V] view
    tc5::mbar_expect_tx(bar_a, (uint32_t)((first ? 4 : 3) * S::tile + DK * DK * 2 + BT * 128 + BT * 4));
    tma::load_3d(Do, &maps.d_o, cm.row, (hv * DK) / 64, bar_a);
    tma::load_3d(Vn, &maps.vn, cm.row, (hv * DK) / 64, bar_a);
    tma::load_3d(dUs, &maps.du, cm.row, (hv * DK) / 64, bar_a);
    tma::load_2d(As, &maps.a, hv * BT, cm.row, bar_a);
    tma::load_1d(gs2 + ((hv - hv0) & 1) * BT, gamma_ptr(a.gamma, c, a.HV, hv), BT * 4, bar_a);
    if (first) tma::load_3d(Ks, &maps.k, cm.row, (hq * DK) / 64, bar_a);
    if (first) load_dh(hv);
    for (int p = 0; p < NP; ++p) {
      if (!first) tma::prefetch_2d(&maps.dh, p * 64, hrow);
      tma::prefetch_2d(&maps.h, p * 64, hrow);
    }
    if (first) tma::prefetch_3d(&maps.q, cm.row, (hq * DK) / 64);
    tma::prefetch_3d(&maps.v, cm.row, (hv * DK) / 64);
  };
  if (tid == 0) {
    for (int i = 0; i < 4; ++i) tc5::mbar_init(bar + i, 1);
    tc5::fence_mbar_init();
    load_head(hv0, true);
  }
  if (warp == 1) tc5::tmem_alloc(tmem_slot, 256);
  // beta and, with the gate option, the gate's value and derivative: the loads, and what becomes of them
  auto head_raw = [&](int hv) {
    const bool beta = tid < BT, gate = (a.options & B200GDN_PREP_GATE) && tid >= 2 * BT && tid < 3 * BT;
    const int r = beta ? tid : tid - 2 * BT;
    return (beta || gate) && r < cm.len ? ld_param(beta ? a.beta : a.g, (row0 + r) * a.HV + hv, a.gb_dtype) : 0.f;
  };
  auto head_vectors = [&](int hv, float raw) {
    if (tid < BT) {
      const bool ok = tid < cm.len;
      float b = raw;
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
      const float x = raw + (a.dt_bias ? a.dt_bias[hv] : 0.f);
      const float negA = -expf(a.A_log[hv]);
      gx[r] = negA / (1.f + expf(-x));
      gv[r] = negA * (x > 20.f ? x : log1pf(expf(x)));
    }
  };
  head_vectors(hv0, head_raw(hv0));
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
  const uint32_t sK = tc5::smem_addr(Ks), sDo = tc5::smem_addr(Do), sVn = tc5::smem_addr(Vn), sZ = tc5::smem_addr(Zt), sH = tc5::smem_addr(Hs);
  const uint32_t sA = tc5::smem_addr(As);
  const Operand opK_k{sK, BT, 0}, opK_mn{sK, BT, 1};      // K as (rows = token, contraction = key dim), and the reverse
  bool failed = false;
  // several heads: this thread's part of the sum of dk so far (turns) or of dq (cluster), in local memory between its uses
  __align__(16) float part_local[MODE != kOne ? 16 * NH : 4];
  const uint64_t part = __cvta_generic_to_local(part_local);
  // one head: Z waits in C2 for V, and Z v_new^T takes C1; turns: the sum of dq has C1, so Z waits in registers
  const uint32_t CZ = TURNS ? C2 : C1;

  for (int hh = 0; hh < n_heads; ++hh) {
    const int hv = hv0 + hh, hrow = (c * a.HV + hv) * DK;
    const uint32_t par = hh & 1;
    const bool first = !TURNS || hh == 0, last = !TURNS || hh + 1 == n_heads;
    const float* gs = gs2 + par * BT;
    if (!tc5::mbar_wait(bar_a, par)) failed = true;
    if (cm.len < BT) {   // ragged chunk: the extra rows of the boxes belong to the next sequence
      zero_tail_rows<BT, DK>(Do, cm.len, tid, NTHREADS);
      zero_tail_rows<BT, DK>(Vn, cm.len, tid, NTHREADS);
      zero_tail_rows<BT, DK>(dUs, cm.len, tid, NTHREADS);
      zero_tail_rows<BT, BT>(As, cm.len, tid, NTHREADS);
      if (first) zero_tail_rows<BT, DK>(Ks, cm.len, tid, NTHREADS);
      tc5::fence_async_smem();
    }
    if (__syncthreads_or(failed)) { failed = true; break; }

    // ---- phase 1: Z^T = dU^T A | dP = do v_new^T | dk_state^T = dh v_new^T (column factor later)
    if (warp == 0) {
      tc5::fence_after_sync();
      issue_mma_t<BT / 16>(C2, Operand{sZ, BT, 1}, Operand{sA, BT, 1}, DK, 64, 0);
      issue_mma_t<DK / 16>(C0, Operand{sDo, BT, 0}, Operand{sVn, BT, 0}, 64, 64, 0);
#pragma unroll
      for (int p = 0; p < NP; ++p)
        issue_mma_t<4>(C3, Operand{sH + p * DK * 128, DK, 0}, Operand{sVn + p * BT * 128, BT, 0}, DK, 64, p > 0);
      ph.commit();
    }
    // dh into registers (for <h,dh>) meanwhile
    constexpr int ND = DK * DK / 256 / 8;   // 16 x 16 blocks per warp
    uint32_t dhr[ND][4];
#pragma unroll
    for (int n = 0; n < ND; ++n) load_block16(sH, DK, warp * ND + n, lane, dhr[n]);
    const float g_lo = gs[r_lo], g_hi = gs[r_hi], glast = gs[BT - 1];
    if (tid < BT) {
      const float e = fast_exp2(gs[tid]);
      eg[tid] = e;
      bge[tid] = bet[tid] * e;
    }
    // the reads above are only issued: without this fence the copy of h can overtake those still queued
    tc5::fence_async_smem();
    if (__syncthreads_or(!ph.wait())) { failed = true; break; }

    // ---- epilogue 1: h takes the place of dh, Z^T that of dU, dP~ that of A
    if (tid == 0) {
      tc5::mbar_expect_tx(bar_b, (uint32_t)(DK * DK * 2));
      for (int p = 0; p < NP; ++p) tma::load_2d(Hs + p * DK * 128, &maps.h, p * 64, hrow, bar_b);
    }
    {   // Z -> shared; it stays in C2 as well
      float r[NH][16];
      acc_ld_t<NH>(C2, q, cs, r);
      tc5::tmem_ld_wait();
#pragma unroll
      for (int hf = 0; hf < NH; ++hf) {
        FragStore fs;
#pragma unroll
        for (int i = 0; i < 4; ++i) fs.set(i, r[hf][4 * i], r[hf][4 * i + 1], r[hf][4 * i + 2], r[hf][4 * i + 3]);
        fs.store(Zt, DK, kr + 16 * hf, cs, lane);
      }
    }
    {   // dP~ -> shared
      float r[16];
      FragStore fs = {};
      if (live) {
      acc_ld32q(C0, q, cs, r);
      tc5::tmem_ld_wait();
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
    float dk_dot;       // this lane's part of c_rk
    float rk[NH][16];   // dk as far as it is known
    {   // dk_state^T: column factors, the sum of its dots with k
      acc_ld_t<NH>(C3, q, cs, rk);
      tc5::tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 gj = *reinterpret_cast<const float2*>(&gs[cs + i * 8 + 2 * t]);
        scale_t<NH>(rk, i, make_float2(fast_exp2(glast - gj.x), fast_exp2(glast - gj.y)));
      }
      float pv[8];
      dots_t<NH>(rk, Ks, kr, cs, lane, pv);
      dk_dot = sum8_over_g(pv, g);
      const float rs = warp_sum(dk_dot);
      if (lane == 0) red[8 + warp] = rs;
    }
    if (!tc5::mbar_wait(bar_b, par)) failed = true;
    {
      float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int n = 0; n < ND; ++n) {
        uint32_t x[4];
        load_block16(sH, DK, warp * ND + n, lane, x);
        mma16816(d0, dhr[n], x[0], x[2]);
        mma16816(d1, dhr[n], x[1], x[3]);
      }
      const float hd = warp_sum((g == 2 * t ? d0[0] + d1[2] : 0.f) + (g == 2 * t + 1 ? d0[1] + d1[3] : 0.f));
      if (lane == 0) red[warp] = hd;
    }
    float z[NH][16];
    if (TURNS) {
      acc_ld_t<NH>(C2, q, cs, z);
      tc5::tmem_ld_wait();
    }
    tc5::fence_async_smem();
    tc5::fence_before_sync();
    if (__syncthreads_or(failed)) { failed = true; break; }

    // ---- phase 2: ZV = Z v_new^T | -h Z^T | dq^T = h do_s^T + K^T dP~^T
    if (warp == 0) {
      tc5::fence_after_sync();
      issue_mma_t<DK / 16>(CZ, Operand{sZ, DK, 1}, Operand{sVn, BT, 0}, 64, 64, 0);
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        issue_mma_t<4>(C3, Operand{sH + p * DK * 128, DK, 0}, Operand{sZ + p * BT * 128, DK, 1}, DK, 64, p > 0, /*neg_a=*/1);
        issue_mma_t<4>(C0, Operand{sH + p * DK * 128, DK, 0}, Operand{sDo + p * BT * 128, BT, 0}, DK, 64, p > 0);
      }
      issue_mma_t<4>(C0, opK_mn, Operand{sA, BT, 0}, DK, 64, 1);
      ph.commit();
    }
    if (__syncthreads_or(!ph.wait())) { failed = true; break; }

    // ---- epilogue 2: q takes the place of do, V that of v_new; M2 -> shared (over h)
    if (tid == 0) {
      tc5::mbar_expect_tx(bar_c, (uint32_t)(2 * S::tile));
      tma::load_3d(Qs, &maps.q, cm.row, (hq * DK) / 64, bar_c);
      tma::load_3d(Vs, &maps.v, cm.row, (hv * DK) / 64, bar_c);
    }
    float m[16];   // M, later its products with K K^T
    {
      FragStore fs = {};
      if (live) {
        const float b_lo = bet[r_lo], b_hi = bet[r_hi];
        acc_ld32q(CZ, q, cs, m);
        tc5::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int col = cs + i * 8 + 2 * t;
          const float2 gj = *reinterpret_cast<const float2*>(&gs[col]);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int ii = (e & 2) ? r_hi : r_lo, jj = col + (e & 1);
            m[4 * i + e] = (ii > jj) ? -m[4 * i + e] * fast_exp2(((e & 2) ? g_hi : g_lo) - ((e & 1) ? gj.y : gj.x)) : 0.f;
          }
          fs.set(i, m[4 * i] * b_lo, m[4 * i + 1] * b_lo, m[4 * i + 2] * b_hi, m[4 * i + 3] * b_hi);
        }
      }
      fs.store(M2s, BT, q * 16, cs, lane);
    }
    {   // -h Z^T: its dots with k; into dk with the factor beta 2^gamma
      float r[NH][16], pv[8];
      acc_ld_t<NH>(C3, q, cs, r);
      tc5::tmem_ld_wait();
      dots_t<NH>(r, Ks, kr, cs, lane, pv);
      c_kz[q * BT + gcol] = sum8_over_g(pv, g);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 bg = *reinterpret_cast<const float2*>(&bge[cs + i * 8 + 2 * t]);
        scale_add_t<NH>(rk, r, i, bg);
      }
    }
    auto finish_z = [&] {   // Z: its dots with v; dv = beta Z on its way out, over the second panel of h
      float pv[8];
      dots_t<NH>(z, Vs, kr, cs, lane, pv);   // (rows past a ragged chunk's end are not used)
      c_vb[q * BT + gcol] = sum8_over_g(pv, g);
#pragma unroll
      for (int i = 0; i < 4; ++i) scale_t<NH>(z, i, *reinterpret_cast<const float2*>(&bet[cs + i * 8 + 2 * t]));
      stage_t<NH>(z, Dvs, kr, cs, lane);
    };
    float rq[NH][16];   // dq: C0 is phase 3's
    if (!TURNS) acc_ld_t<NH>(C0, q, cs, rq);
    if (!tc5::mbar_wait(bar_c, par)) failed = true;
    if (TURNS) {
      finish_z();
      acc_ld_t<NH>(C0, q, cs, rq);
    }
    if (cm.len < BT) {
      zero_tail_rows<BT, DK>(Qs, cm.len, tid, NTHREADS);
      zero_tail_rows<BT, DK>(Vs, cm.len, tid, NTHREADS);
    }
    tc5::tmem_ld_wait();
    tc5::fence_async_smem();
    tc5::fence_before_sync();
    if (__syncthreads_or(failed)) { failed = true; break; }

    // ---- phase 3: the rest of dk^T = q^T dP~ + K^T M2^T + K^T M2 | KK = K K^T | QK = Q K^T
    if (warp == 0) {
      tc5::fence_after_sync();
      issue_mma_t<BT / 16>(C3, opK_mn, Operand{sH, BT, 0}, DK, 64, 0);
      issue_mma_t<BT / 16>(C3, opK_mn, Operand{sH, BT, 1}, DK, 64, 1);
      issue_mma_t<BT / 16>(C3, Operand{sDo, BT, 1}, Operand{sA, BT, 1}, DK, 64, 1);
      issue_mma_t<DK / 16>(C0, opK_k, opK_k, 64, 64, 0);
      issue_mma_t<DK / 16>(CZ, Operand{sDo, BT, 0}, opK_k, 64, 64, 0);
      ph.commit();
    }
    {   // dq: its dots with q, the sum over the heads; ungrouped heads, and the last one in turn: on its way out, over Z^T
      float pv[8];
      dots_t<NH>(rq, Qs, kr, cs, lane, pv);
      c_rq[q * BT + gcol] = sum8_over_g(pv, g);
      if (!first) {
        float acc[NH][16];
        acc_ld_t<NH>(C1, q, cs, acc);
        tc5::tmem_ld_wait();
        add_t<NH>(rq, acc);
      }
      if (GROUPED) {
        st_local<NH>(rq, part);
      } else if (!last) {
#pragma unroll
        for (int hf = 0; hf < NH; ++hf) tc5::tmem_st_16x256b_x4(C1 + ((uint32_t)(32 * q + 16 * hf) << 16) + cs, rq[hf]);
        tc5::tmem_st_wait();
      } else {
        if (a.rstd_q != nullptr) {
          float* dots = c_rq;
          if (TURNS) {   // of the sum; c_rk is free until epilogue 3
            dots = c_rk;
            dots_t<NH>(rq, Qs, kr, cs, lane, pv);
            dots[q * BT + gcol] = sum8_over_g(pv, g);
          }
          __syncthreads();
          l2_backward_t<NH>(rq, Qs, dots, rsq, kr, cs, lane);
        }
        stage_t<NH>(rq, Dqs, kr, cs, lane);
      }
    }
    if (!TURNS) {
      acc_ld_t<NH>(C2, q, cs, z);
      tc5::tmem_ld_wait();
      finish_z();
    }
    const float raw_next = last ? 0.f : head_raw(hv + 1);
    FragLoad fp;
    fp.load(Ps, BT, q * 16, cs, lane);
    tc5::fence_async_smem();   // the staged tiles are read, and what was read here is overwritten, by bulk copies
    tc5::fence_before_sync();
    if (__syncthreads_or(!ph.wait())) { failed = true; break; }
    if (by_tma) {
      if (tid == 0) {
        tma::store_3d(&maps.dv, cm.row, (hv * DK) / 64, Dvs);
        if (!GROUPED && last) tma::store_3d(&maps.dq, cm.row, (hq * DK) / 64, Dqs);
        tma::store_commit();
      }
    } else {
      store_tile_swz<BT, DK, NTHREADS>(reinterpret_cast<__nv_bfloat16*>(a.dv) + (row0 * a.HV + hv) * DK, (int64_t)a.HV * DK, Dvs, cm.len, tid);
      if (!GROUPED && last)
        store_tile_swz<BT, DK, NTHREADS>(reinterpret_cast<__nv_bfloat16*>(a.dq) + (row0 * a.H + hq) * DK, (int64_t)a.H * DK, Dqs, cm.len, tid);
      if (!last) {
        tc5::fence_async_smem();
        __syncthreads();
      }
    }
    if (!last && tid == 0) load_head(hv + 1, false);   // every tile but K is dead

    // ---- epilogue 3: dk and the gate and beta gradients
    {
      float kk[16], qk[16], pv[8], rmk_lo = 0.f, rmk_hi = 0.f;   // (blocks above the diagonal hold zeros)
      if (live) {
      acc_ld32q(C0, q, cs, kk);
      acc_ld32q(CZ, q, cs, qk);
      tc5::tmem_ld_wait();
      const float b_lo = bet[r_lo], b_hi = bet[r_hi];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int e = 0; e < 4; ++e) m[4 * i + e] *= kk[4 * i + e];
        rmk_lo += m[4 * i] + m[4 * i + 1];
        rmk_hi += m[4 * i + 2] + m[4 * i + 3];
        const float2 pl = fp.lo2(i), phi = fp.hi2(i);
        pv[2 * i] = (m[4 * i] * b_lo + m[4 * i + 2] * b_hi) + (pl.x * qk[4 * i] + phi.x * qk[4 * i + 2]);
        pv[2 * i + 1] = (m[4 * i + 1] * b_lo + m[4 * i + 3] * b_hi) + (pl.y * qk[4 * i + 1] + phi.y * qk[4 * i + 3]);
      }
      dk_dot += sum8_over_g(pv, g);
      rmk_lo = sum_over_t(rmk_lo);
      rmk_hi = sum_over_t(rmk_hi);
      }
      c_rk[q * BT + gcol] = dk_dot;
      if (t == 0) {
        r_mk[hc * BT + r_lo] = rmk_lo;
        r_mk[hc * BT + r_hi] = rmk_hi;
      }
      float r[NH][16];
      acc_ld_t<NH>(C3, q, cs, r);
      tc5::tmem_ld_wait();
      add_t<NH>(rk, r);
      if (TURNS) {
        if (!first) add_local<NH>(rk, part);
        if (!last) st_local<NH>(rk, part);
      }
      if (!GROUPED && last && a.rstd_k != nullptr) {   // <dk, k> for the norm's backward, over a tile that is needed no more
        dots_t<NH>(rk, Ks, kr, cs, lane, pv);
        reinterpret_cast<float*>(Ps)[q * BT + gcol] = sum8_over_g(pv, g);
      }
    }
    if (GROUPED && tid == 0) tma::store_wait_read<0>();   // the sums are staged over dv
    tc5::fence_before_sync();   // the next head's first phase writes what was read here
    __syncthreads();
    if (tid < BT) {
      const int i = tid;
      auto sum4 = [&](const float* v) { return (v[i] + v[BT + i]) + (v[2 * BT + i] + v[3 * BT + i]); };
      const float rmk = r_mk[i] + r_mk[BT + i], ckz = sum4(c_kz);
      float x = sum4(c_rq) - sum4(c_rk) + (ckz * bge[i] + bet[i] * rmk);
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
        float db = ckz * eg[i] + sum4(c_vb) + rmk;
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
      if (a.rstd_k != nullptr) l2_backward_t<NH>(rk, Ks, reinterpret_cast<float*>(Ps), rsk, kr, cs, lane);
      stage_t<NH>(rk, Dks, kr, cs, lane);   // over M2
      tc5::fence_async_smem();
    } else if (GROUPED) {
      // this head's dq and dk in fp32, token-major, over the dead tiles
      float* sq = reinterpret_cast<float*>(smem + S::o_do);
      float* sk = reinterpret_cast<float*>(smem + S::o_do + S::stage);
      float r[NH][16] = {};
      add_local<NH>(r, part);
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
    if (!GROUPED && last) {
      if (by_tma) {
        if (tid == 0) {
          tma::store_3d(&maps.dk, cm.row, (hq * DK) / 64, Dks);
          tma::store_commit();
        }
      } else {
        store_tile_swz<BT, DK, NTHREADS>(reinterpret_cast<__nv_bfloat16*>(a.dk) + (row0 * a.H + hq) * DK, (int64_t)a.H * DK, Dks, cm.len, tid);
      }
    }
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
      if (tid == 0) {   // dv of this head leaves from the place of dh; waited for here, where the copy has long been read
        tma::store_wait_read<0>();
        load_dh(hv + 1);
      }
      __syncthreads();   // the vectors have been read
      head_vectors(hv + 1, raw_next);
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
  if (tid == 0) tma::store_wait_read<0>();   // shared memory must outlive the bulk stores that read it
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
  // A tensor map costs the host 0.6 us: small problems, which wait for the host, store their results by rows
  const bool out_maps = !overlaps(a);
  m.dq = m.dk = m.dv = m.q;
  if (out_maps) {
    rc |= tma::encode_bf16_panels(&m.dq, a.dq, a.rows, pk, pk, BT, DK / 64);
    rc |= tma::encode_bf16_panels(&m.dk, a.dk, a.rows, pk, pk, BT, DK / 64);
    rc |= tma::encode_bf16_panels(&m.dv, a.dv, a.rows, pv, pv, BT, DK / 64);
  }
  rc |= tma::encode_bf16_2d(&m.a, a.A, a.rows, (uint64_t)a.HV * BT, (uint64_t)a.HV * BT, BT);
  rc |= tma::encode_bf16_2d(&m.h, a.h, hrows, DK, DK, DK);
  rc |= tma::encode_bf16_2d(&m.dh, a.dh, hrows, DK, DK, DK);
  if (rc != 0) return set_error(B200GDN_ERR_CUDA, "bwd_local: cuTensorMapEncodeTiled failed (%d)", rc);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)a.n_chunks * (MODE == kTurns ? a.H : a.HV));
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
    attr[cfg.numAttrs].val.clusterDim.x = a.HV / a.H;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  cudaLaunchKernelEx(&cfg, bwd_local_kernel<DK, MODE>, a, m, out_maps);
  if (int e = check_launch("bwd_local")) return e;
  return launch_gate_reduce(a, st);
}

// Several value heads per q/k head: in turn in one CTA, or a CTA each and the sums of dq and dk through a cluster.  A cluster
// costs more per head (it holds its CTAs until the slowest has arrived and its sums have been read: 260 us against 201 at B4 T4096
// 8/16 heads of 128, but 78 against 87 at B1 T3300 4/16 heads, whose turns are four rounds and whose clusters three), but has G times as many CTAs, so it stays where turns would leave
// the device to a few: two fit on an SM, and the rounds of CTAs decide.  Group sizes other than two, four
// and eight are taken in turns always.  Both forms add the heads
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
