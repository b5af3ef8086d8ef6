// Element access for the HBM-streaming row kernels: one element, or eight consecutive elements (16 bytes of bf16 /
// fp16, 32 bytes of fp32) of a row, as floats.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include <type_traits>

namespace gdn {

template <typename T> struct Io;
template <> struct Io<__nv_bfloat16> {
  static __device__ __forceinline__ float ld(const void* p, int64_t i) { return __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]); }
  static __device__ __forceinline__ void st(void* p, int64_t i, float v) { static_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v); }
};
template <> struct Io<__half> {
  static __device__ __forceinline__ float ld(const void* p, int64_t i) { return __half2float(static_cast<const __half*>(p)[i]); }
  static __device__ __forceinline__ void st(void* p, int64_t i, float v) { static_cast<__half*>(p)[i] = __float2half_rn(v); }
};
template <> struct Io<float> {
  static __device__ __forceinline__ float ld(const void* p, int64_t i) { return static_cast<const float*>(p)[i]; }
  static __device__ __forceinline__ void st(void* p, int64_t i, float v) { static_cast<float*>(p)[i] = v; }
};

// eight packed elements (one 16-byte word of bf16 / fp16) to floats and back: two elements per 32-bit word, the
// conversions written out so that each pair costs two (bf16: a shift and a mask) resp. one instruction
template <typename T>
__device__ __forceinline__ void unpack8(const uint4& u, float (&x)[8]) {
  static_assert(sizeof(T) == 2, "16-bit element types");
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if constexpr (!std::is_same<T, __half>::value) {
      x[2 * i] = __uint_as_float(w[i] << 16);
      x[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    } else {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
      x[2 * i] = f.x;
      x[2 * i + 1] = f.y;
    }
  }
}
template <typename T>
__device__ __forceinline__ uint4 pack8(const float (&x)[8]) {
  static_assert(sizeof(T) == 2, "16-bit element types");
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if constexpr (!std::is_same<T, __half>::value) {
      const __nv_bfloat162 p = __floats2bfloat162_rn(x[2 * i], x[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&p);
    } else {
      const __half2 p = __floats2half2_rn(x[2 * i], x[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&p);
    }
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// 8 consecutive elements of a row as floats (16 bytes of bf16 / fp16, 32 bytes of fp32)
template <typename T>
__device__ __forceinline__ void load8(const void* base, int64_t idx, float (&x)[8]) {
  if constexpr (sizeof(T) == 2) {
    unpack8<T>(*reinterpret_cast<const uint4*>(static_cast<const T*>(base) + idx), x);
  } else {
    const float4 a = *reinterpret_cast<const float4*>(static_cast<const float*>(base) + idx);
    const float4 b = *reinterpret_cast<const float4*>(static_cast<const float*>(base) + idx + 4);
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
  }
}
template <typename T>
__device__ __forceinline__ void store8(void* base, int64_t idx, const float (&x)[8]) {
  if constexpr (sizeof(T) == 2) {
    *reinterpret_cast<uint4*>(static_cast<T*>(base) + idx) = pack8<T>(x);
  } else {
    *reinterpret_cast<float4*>(static_cast<float*>(base) + idx) = make_float4(x[0], x[1], x[2], x[3]);
    *reinterpret_cast<float4*>(static_cast<float*>(base) + idx + 4) = make_float4(x[4], x[5], x[6], x[7]);
  }
}

// ---- two fp32 operations in one instruction (channel or row pairs; each half rounds like the scalar instruction) ------
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;\n" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
// one 32-bit word of two 16-bit elements <-> an fp32 pair
template <typename T>
__device__ __forceinline__ uint64_t widen2(uint32_t w) {
  if constexpr (!std::is_same<T, __half>::value) {
    return pack2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  } else {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
    return pack2(f.x, f.y);
  }
}
template <typename T>
__device__ __forceinline__ uint32_t narrow2(uint64_t v) {
  const float2 f = unpack2(v);
  if constexpr (!std::is_same<T, __half>::value) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(f.x, f.y);
    return *reinterpret_cast<const uint32_t*>(&p);
  } else {
    const __half2 p = __floats2half2_rn(f.x, f.y);
    return *reinterpret_cast<const uint32_t*>(&p);
  }
}

// sigmoids of a pair with two MUFU instructions each (ex2.approx.ftz, rcp.approx.ftz: about 2 ulp each; the library forms of
// exp and division add range handling that costs more instructions than the rest of an element's work in these kernels)
__device__ __forceinline__ uint64_t fast_sigmoid2(uint64_t x) {
  const float2 z = unpack2(mul2(x, pack2(-1.4426950408889634f, -1.4426950408889634f)));
  float2 e, r;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(e.x) : "f"(z.x));
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(e.y) : "f"(z.y));
  const float2 d = unpack2(add2(pack2(e.x, e.y), pack2(1.f, 1.f)));
  asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(r.x) : "f"(d.x));
  asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(r.y) : "f"(d.y));
  return pack2(r.x, r.y);
}

}  // namespace gdn
