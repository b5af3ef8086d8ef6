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
// A CTA owns one head and CP = 8 value columns of a chain (columns are independent), two threads per row.  The chain is
// serial, so its step is what counts: M_j streams through shared memory in chunks of MC columns, double-buffered by
// asynchronous 16-byte copies, while the row products are formed two columns at a time (f32x2).  Every thread reading its
// row of M from global memory, 32 columns per CTA, took 13 us a step at K = V = 128; 3.6 us now.
constexpr int CP = 8;
template <int DK>
struct PrefixTile {
  static constexpr int MC = DK == 256 ? 32 : DK / 2, NCH = DK / MC, LD = MC + 4;   // row stride: 16-byte reads of rows do not collide
  static constexpr size_t bytes = (size_t)(2 * DK * LD + 2 * DK * CP) * sizeof(float);
};

template <int DK>
__global__ void __launch_bounds__(2 * DK) cp_prefix_kernel(const b200gdn_prefix_args a) {
  using P = PrefixTile<DK>;
  extern __shared__ __align__(16) float sm[];   // M chunks [2][DK][LD], x [2][DK][CP]
  float* const xs = sm + 2 * DK * P::LD;
  const int V = a.V, hv = blockIdx.y, c0 = blockIdx.x * CP, chain = blockIdx.z;
  const int tid = threadIdx.x, r = tid >> 1, ch = (tid & 1) * (CP / 2);
  const int first_out = a.table[3 * chain], count = a.table[3 * chain + 1], first_pre = a.table[3 * chain + 2];
  const int n_chunks = (count - 1) * P::NCH;
  auto pair_of = [&](int t) { return a.reverse ? first_pre + count - 2 - t : first_pre + t; };
  auto fetch = [&](int i) {   // chunk i of the walk into buffer i & 1 (an empty group past the end)
    if (i < n_chunks) {
      const float* M = a.M + ((int64_t)pair_of(i / P::NCH) * a.HV + hv) * DK * DK + (i % P::NCH) * P::MC;
      float* dst = sm + (i & 1) * DK * P::LD;
      for (int e = tid; e < DK * P::MC / 4; e += 2 * DK) {
        const int row = e / (P::MC / 4), c = (e % (P::MC / 4)) * 4;
        cp_async16(dst + row * P::LD + c, M + (int64_t)row * DK + c);
      }
    }
    cp_async_commit();
  };
  fetch(0);
  fetch(1);
  float x[CP / 2];
#pragma unroll
  for (int c = 0; c < CP / 2; ++c) {
    const int col = c0 + ch + c;
    x[c] = a.x0 ? a.x0[(((int64_t)chain * a.HV + hv) * DK + r) * V + col] : ((a.identity && r == col) ? 1.f : 0.f);
  }
  auto keep = [&](int cur, int piece) {
    const float4 v = make_float4(x[0], x[1], x[2], x[3]);
    *reinterpret_cast<float4*>(&xs[(cur * DK + r) * CP + ch]) = v;
    if (a.out != nullptr && piece >= 0) *reinterpret_cast<float4*>(&a.out[(((int64_t)piece * a.HV + hv) * DK + r) * V + c0 + ch]) = v;
  };
  keep(0, a.reverse ? first_out + count - 1 : first_out);
  int cur = 0, i = 0;
  for (int t = 0; t + 1 < count; ++t) {
    uint64_t acc[2] = {0ull, 0ull};
    if (a.h) {
      const float4 h = *reinterpret_cast<const float4*>(&a.h[(((int64_t)pair_of(t) * a.HV + hv) * DK + r) * V + c0 + ch]);
      acc[0] = pack2(h.x, h.y);
      acc[1] = pack2(h.z, h.w);
    }
    for (int k = 0; k < P::NCH; ++k, ++i) {
      cp_async_wait<1>();
      __syncthreads();   // the chunk has landed for everybody (and x of this step is complete)
      const float* Mr = sm + (i & 1) * DK * P::LD + r * P::LD;
      const float* xr = xs + (cur * DK + k * P::MC) * CP + ch;
#pragma unroll 4
      for (int m = 0; m < P::MC; m += 4) {
        const float4 mv = *reinterpret_cast<const float4*>(Mr + m);
        const float mm[4] = {mv.x, mv.y, mv.z, mv.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint64_t* y = reinterpret_cast<const uint64_t*>(xr + (m + e) * CP);
          const uint64_t w = pack2(mm[e], mm[e]);
          acc[0] = fma2(w, y[0], acc[0]);
          acc[1] = fma2(w, y[1], acc[1]);
        }
      }
      __syncthreads();   // everybody has read the chunk before the next one takes its place
      fetch(i + 2);
    }
    const float2 p = unpack2(acc[0]), q = unpack2(acc[1]);
    x[0] = p.x; x[1] = p.y; x[2] = q.x; x[3] = q.y;
    cur ^= 1;
    keep(cur, a.reverse ? first_out + count - 2 - t : first_out + t + 1);
  }
  cp_async_wait<0>();
  if (a.last != nullptr)
    *reinterpret_cast<float4*>(&a.last[(((int64_t)chain * a.HV + hv) * DK + r) * V + c0 + ch]) = make_float4(x[0], x[1], x[2], x[3]);
}

template <int DK>
int launch_prefix(const b200gdn_prefix_args& a, cudaStream_t st) {
  if (int e = ensure_smem(cp_prefix_kernel<DK>, PrefixTile<DK>::bytes)) return e;
  cp_prefix_kernel<DK><<<dim3(a.V / CP, a.HV, a.n_chains), 2 * DK, PrefixTile<DK>::bytes, st>>>(a);
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
