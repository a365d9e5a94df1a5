// The activations of the gated non-linearity: 0 identity, 1 relu, 2 sigmoid.
#pragma once

namespace ssc {

__device__ __forceinline__ float apply_act(float v, int kind) {
  if (kind == 1) return v > 0.f ? v : 0.f;
  if (kind == 2) return __frcp_rn(1.0f + expf(-v));   // the correctly rounded reciprocal: the bits of 1.0f / (...)
  return v;
}

}  // namespace ssc
