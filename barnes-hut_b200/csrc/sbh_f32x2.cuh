// Packed FP32 arithmetic for the tree walks: two lanes' values per
// instruction on sm_100 (FFMA2 / FADD2 / FMUL2, through the float2
// intrinsics of the CUDA 12.8+ runtime headers). Each component rounds as the
// scalar round-to-nearest operation does. The scalar overloads let one
// template body serve a packed pair of target slots and a single leftover
// slot; every fused multiply-add is written out, so the two forms round the
// same way.
#pragma once

#include <cuda_runtime.h>

namespace sbh {

__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float vmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float2 vmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float vadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
// a b, at least 0 and at most 1 (0 for NaN); the packed form is two instructions.
__device__ __forceinline__ float vmul_sat(float a, float b) { return __saturatef(__fmul_rn(a, b)); }
__device__ __forceinline__ float2 vmul_sat(float2 a, float2 b) {
  return make_float2(vmul_sat(a.x, b.x), vmul_sat(a.y, b.y));
}

// 1 / sqrt(a) for a normal a (the walks' h = r^2 + eps^2 + 1e-12), with the maximum
// relative error that the PTX manual states for rsqrt.approx.ftz.f32, 2^-22.9.
__device__ __forceinline__ float vrsqrt(float a) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ float2 vrsqrt(float2 a) { return make_float2(vrsqrt(a.x), vrsqrt(a.y)); }

// 1 / a and 2^a by the special-function unit (a few ulps; normal arguments).
__device__ __forceinline__ float vrcp(float a) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ float2 vrcp(float2 a) { return make_float2(vrcp(a.x), vrcp(a.y)); }
__device__ __forceinline__ float vexp2(float a) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ float2 vexp2(float2 a) { return make_float2(vexp2(a.x), vexp2(a.y)); }
__device__ __forceinline__ float vneg(float a) { return -a; }
__device__ __forceinline__ float2 vneg(float2 a) { return make_float2(-a.x, -a.y); }

template <typename V>
__device__ __forceinline__ V vsplat(float s);
template <>
__device__ __forceinline__ float vsplat<float>(float s) {
  return s;
}
template <>
__device__ __forceinline__ float2 vsplat<float2>(float s) {
  return make_float2(s, s);
}

}  // namespace sbh
