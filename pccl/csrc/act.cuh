// GELU (tanh form) and its derivative, shared by the elementwise kernels and the GEMM epilogue.
//
//   gelu(x)  = 0.5 x (1 + tanh(u)) = x * sigmoid(2u),   u = k (x + c x^3),  k = sqrt(2/pi), c = 0.044715
//   gelu'(x) = s + x s (1 - s) * 2 du/dx,               s = sigmoid(2u),    du/dx = k (1 + 3 c x^2)
//
// The forward form uses the hardware tanh (relative error about 2^-11, far inside one bf16
// rounding of the result).  The derivative multiplies (1 - s) by a factor that grows with x,
// so it takes the sigmoid from ex2 and rcp (a few ulp each) instead: about a dozen FMA-pipe
// instructions and two special-function ones per element.
#pragma once

namespace pccl {

__device__ __forceinline__ float tanh_hw(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float ex2_hw(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_hw(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float gelu_tanh(float x) {
  const float u = 0.7978845608028654f * x * (1.f + 0.044715f * x * x);
  return 0.5f * x * (1.f + tanh_hw(u));
}

__device__ __forceinline__ float gelu_tanh_grad(float x) {
  x = fminf(fmaxf(x, -20.f), 20.f);                          // beyond that the derivative is 0 or 1 to fp32 precision
  constexpr float k2 = 2.f * 0.7978845608028654f;            // 2k
  constexpr float log2e = 1.4426950408889634f;
  const float x2 = x * x;
  // exp(-2u) = 2^(x * (A + B x^2)); overflow gives s = 0, underflow s = 1
  const float e = ex2_hw(x * fmaf(x2, -k2 * 0.044715f * log2e, -k2 * log2e));
  const float s = rcp_hw(1.f + e);
  const float q = fmaf(x2, 3.f * 0.044715f * k2, k2);        // 2 du/dx
  return s * fmaf(x * (1.f - s), q, 1.f);
}

// ---- two elements at a time: fp32 multiplies and adds in pairs (one instruction for both halves), the
// special-function unit one by one.  Same formulas; halves the instructions the forms above spend beside it.
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ F2 f2(float a) { return f2(a, a); }
__device__ __forceinline__ void split(const F2& p, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p.v)); }
__device__ __forceinline__ F2 operator+(const F2& a, const F2& b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 operator*(const F2& a, const F2& b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 fma2(const F2& a, const F2& b, const F2& c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
// The two bf16 of a packed word as fp32.
__device__ __forceinline__ F2 unpack2(unsigned w) { return f2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }

__device__ __forceinline__ F2 gelu_tanh2(const F2& x) {
  constexpr float k = 0.7978845608028654f;
  const F2 u = x * fma2(x * x, f2(k * 0.044715f), f2(k));
  float a, b;
  split(u, a, b);
  const F2 h = x * f2(0.5f);
  return fma2(h, f2(tanh_hw(a), tanh_hw(b)), h);
}

// x within [-20, 20] (see gelu_tanh_grad).
__device__ __forceinline__ F2 gelu_tanh_grad2(const F2& x) {
  constexpr float k2 = 2.f * 0.7978845608028654f, log2e = 1.4426950408889634f;
  const F2 x2 = x * x;
  const F2 arg = x * fma2(x2, f2(-k2 * 0.044715f * log2e), f2(-k2 * log2e));
  float a, b;
  split(arg, a, b);
  const F2 den = f2(ex2_hw(a), ex2_hw(b)) + f2(1.f);
  split(den, a, b);
  const F2 s = f2(rcp_hw(a), rcp_hw(b));
  const F2 q = fma2(x2, f2(3.f * 0.044715f * k2), f2(k2));
  const F2 xr = x * fma2(s, f2(-1.f), f2(1.f));
  return s * fma2(xr, q, f2(1.f));
}

}  // namespace pccl
