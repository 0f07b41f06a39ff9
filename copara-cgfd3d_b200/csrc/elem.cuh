// elem.cuh -- storage element types of the wavefield sets: FP32, or 16-bit
// (IEEE half, bfloat16) with one power-of-two scale per component.  All
// arithmetic is FP32: values are widened on load and rounded to nearest on
// store.  A stored 16-bit number s of component c stands for s * 2^k[c];
// because the scale is a power of two, scaling is exact and folds into the
// stencil's 1/h factor and the RK coefficients.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

namespace cgfd {

enum { ELEM_F32 = 0, ELEM_F16 = 1, ELEM_BF16 = 2 };

template <typename T> struct Elem;

template <> struct Elem<float> {
  static constexpr int kind = ELEM_F32;
  __device__ __forceinline__ static float ld(const float *p) { return *p; }
  __device__ __forceinline__ static void st(float *p, float v) { *p = v; }
  __device__ __forceinline__ static float2 ld2(const float *p) {
    return *reinterpret_cast<const float2 *>(p);
  }
  __device__ __forceinline__ static void st2(float *p, float2 v) {
    *reinterpret_cast<float2 *>(p) = v;
  }
};

template <> struct Elem<__half> {
  static constexpr int kind = ELEM_F16;
  __device__ __forceinline__ static float ld(const __half *p) { return __half2float(*p); }
  __device__ __forceinline__ static void st(__half *p, float v) { *p = __float2half_rn(v); }
  // a pair as its 32 bits
  __device__ __forceinline__ static float2 widen(unsigned u) {
    float2 r;
    asm("{\n .reg .b16 l, h;\n mov.b32 {l, h}, %2;\n cvt.f32.f16 %0, l;\n cvt.f32.f16 %1, h;\n}"
        : "=f"(r.x), "=f"(r.y) : "r"(u));
    return r;
  }
  __device__ __forceinline__ static unsigned narrow(float2 v) {
    unsigned u;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(u) : "f"(v.y), "f"(v.x));
    return u;
  }
  __device__ __forceinline__ static float2 ld2(const __half *p) {
    return widen(*reinterpret_cast<const unsigned *>(p));
  }
  __device__ __forceinline__ static void st2(__half *p, float2 v) {
    *reinterpret_cast<unsigned *>(p) = narrow(v);
  }
};

template <> struct Elem<__nv_bfloat16> {
  static constexpr int kind = ELEM_BF16;
  __device__ __forceinline__ static float ld(const __nv_bfloat16 *p) {
    return __bfloat162float(*p);
  }
  __device__ __forceinline__ static void st(__nv_bfloat16 *p, float v) {
    *p = __float2bfloat16_rn(v);
  }
  __device__ __forceinline__ static float2 widen(unsigned u) {  // BF16 is FP32's upper half
    return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
  }
  __device__ __forceinline__ static unsigned narrow(float2 v) {
    unsigned u;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(u) : "f"(v.y), "f"(v.x));
    return u;
  }
  __device__ __forceinline__ static float2 ld2(const __nv_bfloat16 *p) {
    return widen(*reinterpret_cast<const unsigned *>(p));
  }
  __device__ __forceinline__ static void st2(__nv_bfloat16 *p, float2 v) {
    *reinterpret_cast<unsigned *>(p) = narrow(v);
  }
};

inline size_t elem_size(int kind) { return kind == ELEM_F32 ? 4 : 2; }

}  // namespace cgfd
