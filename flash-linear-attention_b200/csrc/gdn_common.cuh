// Shared device helpers and host-side launch plumbing for the gated-delta-rule kernels (sm_100a): chunk tables,
// bf16 packing, small asynchronous copies, the per-chunk gate vector, the L2 look-ahead, launch prototypes.
// (The tensor-core / TMEM / TMA primitives live in tc5.cuh, tc5_tile.cuh and tma.cuh.)
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "../../include/b200gdn.h"

namespace gdn {

constexpr int BT = 64;   // tokens per chunk

struct ChunkMeta {
  int seq, row, len, local;
};

__device__ __forceinline__ ChunkMeta load_chunk_meta(const int32_t* chunk_meta, int c) {
  int4 m = reinterpret_cast<const int4*>(chunk_meta)[c];
  return ChunkMeta{m.x, m.y, m.z, m.w};
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---- asynchronous global -> shared copies ------------------------------------------------------------------
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// ---- bf16 pairs ------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack_bf16(uint32_t v) {
  __nv_bfloat162 b = *reinterpret_cast<__nv_bfloat162*>(&v);
  return __bfloat1622float2(b);
}

// ---- tensors read / written in the caller's precision (B200GDN_F32 / BF16 / F16) ----------------------------
__device__ __forceinline__ float ld_param(const void* p, int64_t i, int code) {
  if (code == B200GDN_F32) return static_cast<const float*>(p)[i];
  if (code == B200GDN_BF16) return __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]);
  return __half2float(static_cast<const __half*>(p)[i]);
}
__device__ __forceinline__ void st_param(void* p, int64_t i, int code, float x) {
  if (code == B200GDN_F32) static_cast<float*>(p)[i] = x;
  else if (code == B200GDN_BF16) static_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(x);
  else static_cast<__half*>(p)[i] = __float2half_rn(x);
}

// gamma is stored per chunk, [n_chunks][HV][64] fp32, entries past the chunk's valid length repeating the
// last valid value (so 2^(gamma_last - gamma_i) is 1 there): a chunk's 64 values are 256 contiguous,
// 256-byte aligned bytes that one bulk copy or one coalesced load brings in.
__device__ __forceinline__ const float* gamma_ptr(const float* gamma, int c, int HV, int hv) {
  return gamma + ((int64_t)c * HV + hv) * BT;
}

// bounds of the chunks' state transitions (option TRANSITION_BOUNDS), [n_chunks][HV] behind gamma; +infinity (or NaN) where w or u of the
// chunk is not finite.  The lowest bit says that the products of q and k are not: of no account for the state, but the gradient that
// leaves the chunk is not finite then, whatever the output's gradient is.
__device__ __forceinline__ float* bounds_ptr(float* gamma, int n_chunks, int HV) { return gamma + (int64_t)n_chunks * HV * BT; }

__device__ __forceinline__ float tagged_bound(float x, bool q_odd) { return __uint_as_float((__float_as_uint(x) & ~1u) | (q_odd ? 1u : 0u)); }

// Of the chunks of [c_first, c_first + nc), counted from the end (`step` -1: a forward scan's) or from the start (+1): `n`, as many as a
// scan has to walk.  For each of the others the transitions of ALL chunks nearer the end have a product of at most 2^-128, so of what
// it leaves in the state no more than that share arrives (gate factors below 2^-126 are flushed to zero within a chunk as well).  The
// sums are not monotonous where gates grow, so what counts is the last one that is not below the line, not the first one that is.
// `zero`: the product over all of them is at most 2^-128.  Where a chunk has values that are not finite (step +1: q among
// them) nothing is left out.
// Executed by a whole warp; a sum of infinities or NaN compares as "not below".
constexpr float kNothingReaches = -128.f;
struct Reach {
  int n;
  bool zero;
};
__device__ __forceinline__ Reach chunks_that_reach(const float* bounds, int HV, int hv, int c_first, int nc, int step, int lane) {
  int n = nc < 1 ? nc : 1;
  float sum = 0.f;
  bool finite = true;
  for (int j0 = 0; j0 < nc; j0 += 32) {
    const int j = j0 + lane;
    float b = j < nc ? bounds[(int64_t)(step > 0 ? c_first + j : c_first + nc - 1 - j) * HV + hv] : 0.f;
    finite = finite && __all_sync(0xffffffffu, b < INFINITY && !(step > 0 && (__float_as_uint(b) & 1u)));   // (false for NaN)
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float y = __shfl_up_sync(0xffffffffu, b, o);
      if (lane >= o) b += y;
    }
    // what lies beyond chunk j arrives: j + 2 chunks are walked at least
    const unsigned arrives = __ballot_sync(0xffffffffu, j + 1 < nc && !(sum + b < kNothingReaches));
    if (arrives != 0) n = j0 + 33 - __clz(arrives);
    sum += __shfl_sync(0xffffffffu, b, 31);
  }
  return finite ? Reach{n, sum < kNothingReaches} : Reach{nc, false};
}

// Look-ahead for the one-CTA-per-(chunk, head) kernels.  CTAs are dispatched in launch order (x fastest), so the
// CTA that will take this one's place on the device is `dist` CTAs further on (dist = CTAs resident at once).
// A CTA pulls that successor's tiles into L2 as it starts; the successor's own loads then see L2 latency
// instead of DRAM latency.  Returns false when there is no successor.
__device__ __forceinline__ bool successor_cta(int dist, int& c2, int& h2) {
  const int nxt = blockIdx.y * gridDim.x + blockIdx.x + dist;
  if (nxt >= (int)(gridDim.x * gridDim.y)) return false;
  c2 = nxt % gridDim.x;
  h2 = nxt / gridDim.x;
  return true;
}

// Kernels of a chain on one stream are launched while their predecessor finishes (its CTAs leave room SM by SM) and wait
// here, as the first thing they do, until it is complete and its writes are visible: no tensor memory is allocated and nothing
// global is touched before.  The successor's launch is released after that, so at most two kernels of a chain are resident.
__device__ __forceinline__ void wait_for_predecessor() {
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

}  // namespace gdn

// ---- host-side launch plumbing (one translation unit per kernel, collected by api.cu) ---------------
namespace gdn {
int launch_intra_fwd(const b200gdn_chunk_args& a, cudaStream_t st);
int launch_scan_fwd(const b200gdn_chunk_args& a, cudaStream_t st);
int launch_scan_out_fwd(const b200gdn_chunk_args& a, cudaStream_t st);
int launch_out_fwd(const b200gdn_chunk_args& a, cudaStream_t st);
int launch_dv_local(const b200gdn_chunk_args& a, cudaStream_t st);
int launch_scan_bwd(const b200gdn_chunk_args& a, cudaStream_t st);
int launch_scan_dvl_bwd(const b200gdn_chunk_args& a, cudaStream_t st);
int launch_bwd_dqk(const b200gdn_chunk_args& a, cudaStream_t st);
int launch_bwd_wy(const b200gdn_chunk_args& a, cudaStream_t st);
int launch_bwd_local(const b200gdn_chunk_args& a, cudaStream_t st);
int launch_gate_reduce(const b200gdn_chunk_args& a, cudaStream_t st);
int check_gate_args(const b200gdn_chunk_args& a, const char* who);
int launch_recurrent(const b200gdn_recurrent_args& a, cudaStream_t st);
int launch_affine(const b200gdn_affine_args& a, cudaStream_t st);
int launch_cp_fold(const b200gdn_fold_args& a, cudaStream_t st);
int launch_cp_prefix(const b200gdn_prefix_args& a, cudaStream_t st);
int launch_prep(const b200gdn_prep_args& a, cudaStream_t st, bool bwd);
int launch_conv(const b200gdn_conv_args& a, cudaStream_t st, bool bwd);
int launch_norm_gate(const b200gdn_norm_gate_args& a, cudaStream_t st, bool bwd);
int norm_gate_grid(int64_t rows);
int decode_timeout_flag();
int intra_fwd_timeout_flag();
int scan_fwd_timeout_flag();
int out_fwd_timeout_flag();
int dv_local_timeout_flag();
int scan_bwd_timeout_flag();
int bwd_dqk_timeout_flag();
int bwd_wy_timeout_flag();
int bwd_local_timeout_flag();
int set_error(int code, const char* fmt, ...);
int check_launch(const char* what);
void reset_launch_count();

// The dynamic shared memory limit of a kernel, set once per thread and device: the driver call costs about half a microsecond,
// which a decoding step would pay on every launch.
struct SmemLimits {
  struct Entry { const void* kern; int dev; };
  Entry set[64];
  int n = 0;
  bool has(const void* kern, int dev) const {
    for (int i = 0; i < n; ++i)
      if (set[i].kern == kern && set[i].dev == dev) return true;
    return false;
  }
  void add(const void* kern, int dev) {
    if (n < 64) set[n++] = Entry{kern, dev};
  }
};
inline SmemLimits& smem_limits() {
  static thread_local SmemLimits limits;
  return limits;
}

template <typename Kern>
int ensure_smem(Kern kern, size_t bytes) {   // `bytes` is a constant of the kernel's instantiation
  int dev = 0;
  cudaGetDevice(&dev);
  const void* key = reinterpret_cast<const void*>(kern);
  if (smem_limits().has(key, dev)) return 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess)
    return set_error(B200GDN_ERR_CUDA, "cudaFuncSetAttribute(%zu B): %s", bytes, cudaGetErrorString(cudaGetLastError()));
  smem_limits().add(key, dev);
  return 0;
}

// Launch that may begin while the kernel before it on the stream is finishing (`overlap`); the kernel calls
// wait_for_predecessor() before anything else.  Measured: 1 x 1024 tokens, 4 heads of 64, forward (two kernels) 29.5 -> 26.0 us;
// 16 x 86 tokens, 24 heads of 64, 39.8 -> 35.8.  With many waves of CTAs there is nothing to hide and the waiting CTAs are in the
// way: B4 T4096 16 heads forward and backward 513 -> 519 us, 65536 tokens, 32 heads 3890 -> 3960; so up to 2048 chunk-heads.
inline bool overlaps(const b200gdn_chunk_args& a) { return (int64_t)a.n_chunks * a.HV <= 2048; }
template <typename... P, typename... A>
void launch_overlapped(bool overlap, void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = overlap ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

// Streaming multiprocessors of the current device (148 where there is none to ask), looked up once per device.
inline int sm_count() {
  static std::atomic<int> known[64];
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = -1;
  if (dev >= 0 && (sms = known[dev].load(std::memory_order_relaxed)) > 0) return sms;
  if (dev < 0 || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) return 148;
  known[dev].store(sms, std::memory_order_relaxed);
  return sms;
}

// CTAs of a kernel resident on the whole device at once (SMs x CTAs per SM); looked up once per kernel and device.
template <auto KERN>
int resident_ctas(int threads, size_t smem) {
  static std::atomic<int> known[64];
  int dev = 0, per_sm = 1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = -1;
  const int hit = dev >= 0 ? known[dev].load(std::memory_order_relaxed) : 0;
  if (hit > 0) return hit;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, KERN, threads, smem) != cudaSuccess || per_sm < 1) per_sm = 1;
  const int ctas = per_sm * sm_count();
  if (dev >= 0) known[dev].store(ctas, std::memory_order_relaxed);
  return ctas;
}
}  // namespace gdn
