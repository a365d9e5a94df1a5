// The activations of the gated non-linearity: 0 identity, 1 relu, 2 sigmoid.
#pragma once
#include <cstdint>

namespace ssc {

__device__ __forceinline__ float apply_act(float v, int kind) {
  if (kind == 1) return v > 0.f ? v : 0.f;
  if (kind == 2) return __frcp_rn(1.0f + expf(-v));   // the correctly rounded reciprocal: the bits of 1.0f / (...)
  return v;
}

// N sigmoids side by side, with the bits of apply_act(v, 2).  __frcp_rn ends in a branch for unusual arguments, and N of
// them in a row are N dependent chains one after the other.  Here the approximate reciprocal takes one step with the
// exact remainder, which rounds correctly (Markstein 1990) for every denominator from 1 to 2^125: all of them were compared.
// Larger ones (results below 2^-125) take the function.
template <int N>
__device__ __forceinline__ void apply_sigmoids(float *v) {
  float d[N], top = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    d[i] = 1.0f + expf(-v[i]);
    top = fmaxf(top, d[i]);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d[i]));
    v[i] = fmaf(fmaf(-d[i], r, 1.0f), r, r);
  }
  if (top > 0x1p125f) {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = __frcp_rn(d[i]);
  }
}

}  // namespace ssc
