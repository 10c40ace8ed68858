// Packed FP32 arithmetic of the time-stepping kernels.
#pragma once
#include <cuda_runtime.h>

#include "wave_common.cuh"

namespace wg {

// Packed FP32 arithmetic: a thread's column pair is one operand, each half rounded to nearest as the
// scalar operation is. ptxas contracts a packed product and sum into a packed fma even under
// -fmad=false and with explicit .rn, which would round once where the reference rounds twice. So a
// product that feeds a sum is formed as fma(a, b, -0) with the -0 taken from the kernel's arguments,
// where the compiler cannot see it: a b + (-0) is the rounded product bit for bit (signs of zeros
// included), and an fma is not contracted again.
struct Pk {
  float2 nz;  // (-0, -0), opaque
  __device__ __forceinline__ float2 mul(float2 a, float2 b) const { return __ffma2_rn(a, b, nz); }
  __device__ __forceinline__ float2 scale(float a, float2 b) const { return mul(make_float2(a, a), b); }
  // (((D2A u + D2B s1) - D2C s2) ka) kb; s1 / s2: sums of the neighbours at distance 1 / 2 (the
  // adjoint's (x + (-D2C) s2) is the same value)
  __device__ __forceinline__ float2 second(float2 u, float2 s1, float2 s2, float ka, float kb) const;
  // ((D1A d1) - D1B d2) rh; d1 / d2: differences of the neighbours at distance 1 / 2
  __device__ __forceinline__ float2 first(float2 d1, float2 d2, float rh) const;
};
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tsub.rn.f32x2 z, x, y;\n\t"
      "mov.b64 {%0, %1}, z;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
// a product that no sum reads (its reader is a store or another product)
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 dup2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 scale2(float a, float2 b) { return mul2(dup2(a), b); }
// Sums and differences at distance 1 along x of the own pair u between the pairs a (left) and b
// (right): they join an own column and a neighbour's, so they are formed per column.
__device__ __forceinline__ float2 side_sum(float2 a, float2 u, float2 b) { return make_float2(u.y + a.y, b.x + u.x); }
__device__ __forceinline__ float2 side_diff(float2 a, float2 u, float2 b) { return make_float2(u.y - a.y, b.x - u.x); }
__device__ __forceinline__ float2 Pk::second(float2 u, float2 s1, float2 s2, float ka, float kb) const {
  return scale(kb, scale2(ka, add2(add2(scale(F_D2A, u), scale(F_D2B, s1)), scale(-F_D2C, s2))));
}
__device__ __forceinline__ float2 Pk::first(float2 d1, float2 d2, float rh) const {
  return scale(rh, add2(scale(F_D1A, d1), scale(-F_D1B, d2)));
}

}  // namespace wg
