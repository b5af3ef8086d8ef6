// out = M x + b (or M^T x + b) per head, fp32: folds a received state prefix through a shard's K x K
// transition matrix for context parallelism (merge step of fla/ops/cp/chunk_delta_h.py:332-460).
// Tiny (2 K^2 V flop per head), so a plain shared-memory tiled fp32 kernel: exact fp32 keeps the
// chained prefix as accurate as the reference's fp32 merge.
#include "gdn_common.cuh"
#include "rowio.cuh"

namespace gdn {
namespace {

constexpr int TM = 64, TN = 64, TK = 16;

__global__ void __launch_bounds__(256) affine_kernel(const b200gdn_affine_args a) {
  __shared__ float Ms[TK][TM + 1];
  __shared__ float Xs[TK][TN + 1];
  const int hv = blockIdx.z, i0 = blockIdx.y * TM, j0 = blockIdx.x * TN;
  const int K = a.K, V = a.V;
  const float* M = a.M + (int64_t)hv * K * K;
  const float* x = a.x + (int64_t)hv * K * V;
  const int tid = threadIdx.x, ty = tid / 16, tx = tid % 16;
  float acc[4][4] = {};
  for (int m0 = 0; m0 < K; m0 += TK) {
    for (int idx = tid; idx < TK * TM; idx += 256) {
      int mm = idx / TM, ii = idx % TM;
      int gi = i0 + ii, gm = m0 + mm;
      float val = 0.f;
      if (gi < K && gm < K) val = a.transpose_m ? M[(int64_t)gm * K + gi] : M[(int64_t)gi * K + gm];
      Ms[mm][ii] = val;
    }
    for (int idx = tid; idx < TK * TN; idx += 256) {
      int mm = idx / TN, jj = idx % TN;
      int gm = m0 + mm, gj = j0 + jj;
      Xs[mm][jj] = (gm < K && gj < V) ? x[(int64_t)gm * V + gj] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int mm = 0; mm < TK; ++mm) {
      float am[4], bx[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) am[r] = Ms[mm][ty * 4 + r];
#pragma unroll
      for (int c = 0; c < 4; ++c) bx[c] = Xs[mm][tx * 4 + c];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] += am[r] * bx[c];
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      int gi = i0 + ty * 4 + r, gj = j0 + tx * 4 + c;
      if (gi < K && gj < V) {
        int64_t o = (int64_t)hv * K * V + (int64_t)gi * V + gj;
        a.out[o] = acc[r][c] + (a.b ? a.b[o] : 0.f);
      }
    }
}

// The whole prefix fold of a rank in one launch: x = b_first; then x = M_j x + b_j for the following `count - 1`
// ranks j = first + step, first + 2 step, ... of the gathered pairs [world][HV][K][K + V] (M in columns [0, K), the
// state part in [K, K + V)), written to out [HV][K][V].  A CTA owns one head and CS value columns (the chain of a
// column slice is independent of the other columns) and keeps its x slice in shared memory; 2 threads per row.
constexpr int CS = 32;

__global__ void cp_fold_kernel(const b200gdn_fold_args a) {
  extern __shared__ float xs[];   // [2][K][CS]
  const int K = a.K, V = a.V, hv = blockIdx.y, c0 = blockIdx.x * CS;
  const int64_t stride = K + V;
  const int tid = threadIdx.x, r = tid >> 1, ch = (tid & 1) * (CS / 2);
  auto pair = [&](int j) { return a.gathered + ((int64_t)j * a.HV + hv) * K * stride; };
  const float* P = pair(a.first);
  float acc[CS / 2];
#pragma unroll
  for (int c = 0; c < CS / 2; ++c) {
    acc[c] = P[r * stride + K + c0 + ch + c];
    xs[r * CS + ch + c] = acc[c];
  }
  __syncthreads();
  int cur = 0;
  for (int i = 1; i < a.count; ++i) {
    P = pair(a.first + i * a.step);
    const float* x = xs + cur * K * CS;
#pragma unroll
    for (int c = 0; c < CS / 2; ++c) acc[c] = P[r * stride + K + c0 + ch + c];
    for (int m = 0; m < K; m += 4) {
      const float4 mv = *reinterpret_cast<const float4*>(&P[r * stride + m]);
      const float mm[4] = {mv.x, mv.y, mv.z, mv.w};
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int c = 0; c < CS / 2; ++c) acc[c] += mm[e] * x[(m + e) * CS + ch + c];
    }
    float* y = xs + (cur ^ 1) * K * CS;
#pragma unroll
    for (int c = 0; c < CS / 2; ++c) y[r * CS + ch + c] = acc[c];
    __syncthreads();
    cur ^= 1;
  }
#pragma unroll
  for (int c = 0; c < CS / 2; ++c) a.out[((int64_t)hv * K + r) * V + c0 + ch + c] = acc[c];
}

// Chains of affine maps inside one GPU (a long sequence cut into pieces that are scanned concurrently): for every
// chain c of the table, x = x0[c] (zeros, or the identity when x0 == NULL and identity != 0); out[first_out] = x; then
// for t = 0 .. count-2:  x = M[j_t] x + h[j_t],  out[o_t] = x, with
//   forward:  j_t = first_pre + t,              o_t = first_out + t + 1
//   reverse:  j_t = first_pre + count - 2 - t,  o_t = first_out + count - 2 - t   (out[first_out + count - 1] = x0 first)
// and, when `last` is given, last[c] = the chain's final x.
// A CTA owns one head and CP = 8 value columns of a chain (columns are independent).  The chain is serial, so its step is what
// counts.  A thread forms four rows x all eight columns over an eighth of the contraction: every element of M_j then belongs
// to one thread and comes straight from global memory into registers, a step ahead of its use (the maps do not depend on
// the chain), only x is shared, and the eight partial sums meet by recursive halving (28 shuffles).  Bound by the
// shared-memory reads of x and fp32 issue.  K = V = 128: 1.5 us a step with
// one CTA per SM (2.3 with M through shared memory, 13 with one row per thread and 32 columns per CTA); 64: 0.65.
constexpr int CP = 8;
template <int DK>
__global__ void __launch_bounds__(2 * DK, 256 / DK) cp_prefix_kernel(const b200gdn_prefix_args a) {
  constexpr int NB = DK / 32, RB = NB < 4 ? NB : 4;          // blocks of 32 columns of M; blocks held in registers
  constexpr int XS = DK * CP + (DK / 4) * 4;                 // x rows; four floats of padding after every four rows (banks)
  __shared__ __align__(16) float xs[2][XS];
  wait_for_predecessor();
  const int V = a.V, hv = blockIdx.y, c0 = blockIdx.x * CP, chain = blockIdx.z;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int mg = lane & 7, r0 = (warp * 4 + (lane >> 3)) * 4;                      // columns 32 b + 4 mg + e of rows r0 .. r0 + 3
  const int r = r0 + ((mg >> 1) & 2) + ((mg >> 1) & 1), ch = (mg & 1) * 4;          // the part of x that the halving leaves here
  const int first_out = a.table[3 * chain], count = a.table[3 * chain + 1], first_pre = a.table[3 * chain + 2];
  auto pair_of = [&](int t) { return a.reverse ? first_pre + count - 2 - t : first_pre + t; };
  float4 mreg[RB][4];
  auto fetch = [&](int t, int blk, float4 (&m)[4]) {
    if (t + 1 < count) {
      const float* M = a.M + (((int64_t)pair_of(t) * a.HV + hv) * DK + r0) * DK + 32 * blk + 4 * mg;
#pragma unroll
      for (int i = 0; i < 4; ++i) m[i] = *reinterpret_cast<const float4*>(M + i * DK);
    }
  };
  auto h_of = [&](int t) {
    return a.h != nullptr && t + 1 < count
               ? *reinterpret_cast<const float4*>(&a.h[(((int64_t)pair_of(t) * a.HV + hv) * DK + r) * V + c0 + ch])
               : make_float4(0.f, 0.f, 0.f, 0.f);
  };
#pragma unroll
  for (int i = 0; i < RB; ++i) fetch(0, i, mreg[i]);
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f), h = h_of(0);
  if (a.x0 != nullptr) {
    const float* x0 = &a.x0[(((int64_t)chain * a.HV + hv) * DK + r) * V + c0 + ch];   // a caller's tensor, on any boundary
    x = make_float4(x0[0], x0[1], x0[2], x0[3]);
  } else if (a.identity) {
    const int d = r - c0 - ch;
    x = make_float4(d == 0, d == 1, d == 2, d == 3);
  }
  auto keep = [&](int cur, int piece) {
    *reinterpret_cast<float4*>(&xs[cur][r * CP + (r >> 2) * 4 + ch]) = x;
    if (a.out != nullptr && piece >= 0) *reinterpret_cast<float4*>(&a.out[(((int64_t)piece * a.HV + hv) * DK + r) * V + c0 + ch]) = x;
  };
  keep(0, a.reverse ? first_out + count - 1 : first_out);
  int cur = 0;
  for (int t = 0; t + 1 < count; ++t) {
    __syncthreads();   // x of this step is complete (and that of the step before has been read)
    const float4 h_next = h_of(t + 1);
    uint64_t acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[i][c] = 0ull;
#pragma unroll
    for (int blk = 0; blk < NB; ++blk) {
      float4 (&m)[4] = mreg[blk % RB];
      const float* xr = &xs[cur][(32 * blk + 4 * mg) * CP + (8 * blk + mg) * 4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(xr + e * CP), hi = *reinterpret_cast<const ulonglong2*>(xr + e * CP + 4);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float f = e == 0 ? m[i].x : e == 1 ? m[i].y : e == 2 ? m[i].z : m[i].w;
          const uint64_t w = pack2(f, f);
          acc[i][0] = fma2(w, lo.x, acc[i][0]);
          acc[i][1] = fma2(w, lo.y, acc[i][1]);
          acc[i][2] = fma2(w, hi.x, acc[i][2]);
          acc[i][3] = fma2(w, hi.y, acc[i][3]);
        }
      }
      // the block RB further on takes this one's registers
      if (blk + RB < NB) fetch(t, blk + RB, m); else fetch(t + 1, blk + RB - NB, m);
    }
    // recursive halving over the eight lanes of a row group: rows, rows, columns; a lane hands over what its partner keeps
    uint64_t s2[2][4], s1[4], s0[2];
    const bool b2 = mg & 4, b1 = mg & 2, b0 = mg & 1;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) s2[i][c] = add2(b2 ? acc[2 + i][c] : acc[i][c], __shfl_xor_sync(0xffffffffu, (unsigned long long)(b2 ? acc[i][c] : acc[2 + i][c]), 4));
#pragma unroll
    for (int c = 0; c < 4; ++c) s1[c] = add2(b1 ? s2[1][c] : s2[0][c], __shfl_xor_sync(0xffffffffu, (unsigned long long)(b1 ? s2[0][c] : s2[1][c]), 2));
#pragma unroll
    for (int c = 0; c < 2; ++c) s0[c] = add2(b0 ? s1[2 + c] : s1[c], __shfl_xor_sync(0xffffffffu, (unsigned long long)(b0 ? s1[c] : s1[2 + c]), 1));
    const float2 lo = unpack2(s0[0]), hi = unpack2(s0[1]);
    x = make_float4(lo.x + h.x, lo.y + h.y, hi.x + h.z, hi.y + h.w);
    h = h_next;
    cur ^= 1;
    keep(cur, a.reverse ? first_out + count - 2 - t : first_out + t + 1);
  }
  if (a.last != nullptr) *reinterpret_cast<float4*>(&a.last[(((int64_t)chain * a.HV + hv) * DK + r) * V + c0 + ch]) = x;
}

template <int DK>
int launch_prefix(const b200gdn_prefix_args& a, cudaStream_t st) {
  launch_overlapped(true, cp_prefix_kernel<DK>, dim3(a.V / CP, a.HV, a.n_chains), 2 * DK, 0, st, a);
  return check_launch("cp_prefix");
}

}  // namespace

int launch_cp_prefix(const b200gdn_prefix_args& a, cudaStream_t st) {
  return a.K == 64 ? launch_prefix<64>(a, st) : a.K == 128 ? launch_prefix<128>(a, st) : launch_prefix<256>(a, st);
}

int launch_cp_fold(const b200gdn_fold_args& a, cudaStream_t st) {
  const size_t smem = (size_t)2 * a.K * CS * sizeof(float);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(cp_fold_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return set_error(B200GDN_ERR_CUDA, "cp_fold: %s", cudaGetErrorString(e));
  }
  dim3 grid(a.V / CS, a.HV);
  cp_fold_kernel<<<grid, 2 * a.K, smem, st>>>(a);
  return check_launch("cp_fold");
}

int launch_affine(const b200gdn_affine_args& a, cudaStream_t st) {
  dim3 grid((a.V + TN - 1) / TN, (a.K + TM - 1) / TM, a.HV);
  affine_kernel<<<grid, 256, 0, st>>>(a);
  return check_launch("affine_apply");
}

}  // namespace gdn
