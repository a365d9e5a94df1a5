// The activations of the gated non-linearity: 0 identity, 1 relu, 2 sigmoid.
#pragma once
#include <cstdint>

namespace ssc {

__device__ __forceinline__ float apply_act(float v, int kind) {
  if (kind == 1) return v > 0.f ? v : 0.f;
  if (kind == 2) return __frcp_rn(1.0f + expf(-v));   // the correctly rounded reciprocal: the bits of 1.0f / (...)
  return v;
}

// 1 / d for 1 <= d <= 2^125, correctly rounded as __frcp_rn(d) is: the approximate reciprocal and one step with the exact
// remainder (Markstein 1990).  A test compares all these denominators.
__device__ __forceinline__ float quick_reciprocal(float d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  return fmaf(fmaf(-d, r, 1.0f), r, r);
}

// N sigmoids side by side, with the bits of apply_act(v, 2).  __frcp_rn ends in a branch for unusual arguments, and N of
// them in a row are N dependent chains one after the other.  Denominators beyond the quick reciprocal's (results below 2^-125)
// take the function.
template <int N>
__device__ __forceinline__ void apply_sigmoids(float *v) {
  float d[N], top = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    d[i] = 1.0f + expf(-v[i]);
    top = fmaxf(top, d[i]);
    v[i] = quick_reciprocal(d[i]);
  }
  if (top > 0x1p125f) {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = __frcp_rn(d[i]);
  }
}

}  // namespace ssc
