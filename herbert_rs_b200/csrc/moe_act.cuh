// Activations of the routed feed-forward's experts.
#pragma once
#include "api.h"
#include "common.cuh"

// A gated expert's hidden value from its two products.  The clamped form (HB_ACT_SWISH_CLAMP, with a limit L):
// g' = min(g, L), v' = clamp(v, -L, L), g' sigmoid(1.702 g') (v' + 1); every other activation: act(g) v.
__device__ __forceinline__ float moe_act(float z, int act);
__device__ __forceinline__ float moe_glu(float g, float v, int act, float limit) {
  if (act == HB_ACT_SWISH_CLAMP) {
    g = fminf(g, limit);
    v = fminf(fmaxf(v, -limit), limit);
    return (g / (1.0f + expf(-HB_SWISH_CLAMP_SLOPE * g))) * (v + 1.0f);
  }
  return moe_act(g, act) * v;
}
__device__ __forceinline__ float moe_act(float z, int act) {
  if (act == HB_ACT_GELU) return 0.5f * z * (1.0f + erff(z * 0.70710678118654752440f));
  if (act == HB_ACT_GELU_TANH) return 0.5f * z * (1.0f + tanhf(0.79788456080286535588f * (z + 0.044715f * z * z * z)));
  return z / (1.0f + expf(-z));
}
