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

// gelu_tanh of values rounded to half:  0.5 x (1 + tanh(u)) = x / (1 + exp(-2u)),  u = sqrt(2/pi) (x + 0.044715 x^3).
// SHARED: the two quotients of a pair share one reciprocal, 1 / (a b); ex2 and rcp are a fifth of this function's issue slots
// and all of its special-function time.  For x > GELU_SHARED_MIN the exponents stay below 60 and the product finite.
constexpr float GELU_SHARED_MIN = -7.25f;
template <typename T, bool SHARED> __device__ __forceinline__ float2 gelu_pair(float2 y) {
  const float2 x = HalfOps<T>::unpack2(HalfOps<T>::pack2(y));
  constexpr float C1 = -2.f * 0.7978845608028654f * 1.4426950408889634f, C2 = C1 * 0.044715f;
  const float2 w = __ffma2_rn(__fmul2_rn(x, x), make_float2(C2, C2), make_float2(C1, C1));
  const float2 e = __fmul2_rn(x, w);  // -2 u log2(e)
  const float2 d = __fadd2_rn(make_float2(fast_exp2(e.x), fast_exp2(e.y)), make_float2(1.f, 1.f));
  if (!SHARED) return make_float2(__fdividef(x.x, d.x), __fdividef(x.y, d.y));
  const float r = __fdividef(1.f, d.x * d.y);
  return __fmul2_rn(x, __fmul2_rn(make_float2(d.y, d.x), make_float2(r, r)));
}
// Eight values; where one is smaller or not a number, each takes a quotient of its own (x / inf is the -0 that large negative
// values tend to, and a NaN stays in its place).  The test costs 1.7 % where GELU bounds the launch (65 520 x 8960 x 1536:
// 805 -> 818 us); one per pair cost 4 %, one for 16 or 32 values, which runs out of registers, 3.7 %.
template <typename T> __device__ __forceinline__ void gelu8(float2 (&y)[4]) {
  const float m = fmin3_nan(fmin3_nan(y[0].x, y[0].y, y[1].x), fmin3_nan(y[1].y, y[2].x, y[2].y), fmin3_nan(y[3].x, y[3].y, y[3].y));
  if (m > GELU_SHARED_MIN) {
#pragma unroll
    for (int i = 0; i < 4; ++i) y[i] = gelu_pair<T, true>(y[i]);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) y[i] = gelu_pair<T, false>(y[i]);
  }
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
