// closure_act.cuh -- the closure network's activation, shared by its kernels.
//
// GELU in its tanh form (Hendrycks & Gimpel, "Gaussian Error Linear Units",
// 2016): gelu(z) = z/2 (1 + tanh(sqrt(2/pi) (z + 0.044715 z^3))), with the
// hardware tanh approximation (PTX tanh.approx.f32).  The derivative is the
// exact derivative of that form.
#pragma once

__device__ __forceinline__ float tanh_hw(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

constexpr float kGeluA = 0.79788456080286536f;  // sqrt(2 / pi)
constexpr float kGeluB = 0.044715f;

// Two values at once in packed FP32 operations.
__device__ __forceinline__ float2 f2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 gelu2(float2 z) {
  const float2 u = __fmul2_rn(__fmul2_rn(f2(kGeluA), z), __ffma2_rn(__fmul2_rn(f2(kGeluB), z), z, f2(1.0f)));
  const float2 t = make_float2(tanh_hw(u.x), tanh_hw(u.y));
  return __fmul2_rn(__fmul2_rn(f2(0.5f), z), __fadd2_rn(f2(1.0f), t));
}
__device__ __forceinline__ float2 gelu_grad2(float2 z) {
  const float2 z2 = __fmul2_rn(z, z);
  const float2 u = __fmul2_rn(__fmul2_rn(f2(kGeluA), z), __ffma2_rn(f2(kGeluB), z2, f2(1.0f)));
  const float2 t = make_float2(tanh_hw(u.x), tanh_hw(u.y));
  const float2 h = __fmul2_rn(f2(0.5f), __fadd2_rn(f2(1.0f), t));
  const float2 d = __ffma2_rn(make_float2(-t.x, -t.y), t, f2(1.0f));  // 1 - t^2
  const float2 q = __fmul2_rn(__fmul2_rn(__fmul2_rn(f2(0.5f), z), d), f2(kGeluA));
  return __fadd2_rn(h, __fmul2_rn(q, __ffma2_rn(f2(3.0f * kGeluB), z2, f2(1.0f))));
}
