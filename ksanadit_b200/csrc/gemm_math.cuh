// Arithmetic of the GEMM epilogues, two neighbouring columns at a time (packed fp32 instructions): shared by the kernels so
// that they give the same bits.
#pragma once
#include "common.cuh"

namespace ksb {
namespace gemm {

// acc * sa * sw + bias
__device__ __forceinline__ float2 scale_pair(float2 acc, float sa, float2 sw, float2 bias) {
  return __ffma2_rn(__fmul2_rn(acc, make_float2(sa, sa)), sw, bias);
}

// gelu_tanh of the value rounded to half:  0.5 x (1 + tanh(u)) = x / (1 + exp(-2u)),  u = sqrt(2/pi) (x + 0.044715 x^3).
// The two quotients share one reciprocal, 1 / (a b), which the exponents' cap keeps finite (at the cap x < -5.6 and the
// result is below 1e-17); ex2 and rcp are a fifth of this function's issue slots and all of its special-function time.
template <typename T> __device__ __forceinline__ float2 gelu_pair(float2 y) {
  const float2 x = HalfOps<T>::unpack2(HalfOps<T>::pack2(y));
  constexpr float C1 = -2.f * 0.7978845608028654f * 1.4426950408889634f, C2 = C1 * 0.044715f;
  const float2 w = __ffma2_rn(__fmul2_rn(x, x), make_float2(C2, C2), make_float2(C1, C1));
  const float2 e = __fmul2_rn(x, w);  // -2 u log2(e)
  const float2 d = __fadd2_rn(make_float2(fast_exp2(fminf(e.x, 60.f)), fast_exp2(fminf(e.y, 60.f))), make_float2(1.f, 1.f));
  const float r = __fdividef(1.f, d.x * d.y);
  return __fmul2_rn(x, __fmul2_rn(make_float2(d.y, d.x), make_float2(r, r)));
}

// resid + round(y) * gate
template <typename T> __device__ __forceinline__ float2 gate_pair(float2 y, float2 gate, float2 resid) {
  return __ffma2_rn(HalfOps<T>::unpack2(HalfOps<T>::pack2(y)), gate, resid);
}

// Sum of squares of one 16-byte unit (8 columns) of rounded outputs; the eight units of 64 columns are added as a binary tree.
template <typename T> __device__ __forceinline__ float unit_squares(const uint4& o) {
  const uint32_t w[4] = {o.x, o.y, o.z, o.w};
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 v = HalfOps<T>::unpack2(w[i]);
    s = __fmaf_rn(v.x, v.x, s);
    s = __fmaf_rn(v.y, v.y, s);
  }
  return s;
}

}  // namespace gemm
}  // namespace ksb
