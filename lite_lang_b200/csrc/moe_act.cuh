// The activations of routed experts without a gate.
#pragma once

#include "common.cuh"

// act: 0 relu(z)^2, 1 silu(z), 2 gelu_tanh(z), 3 gelu(z) (the erf form).
__device__ __forceinline__ float moe_activation(float z, int act) {
  if (act == 0) {
    const float r = fmaxf(z, 0.f);
    return r * r;
  }
  if (act == 1) return z / (1.0f + expf(-z));
  if (act == 3) return 0.5f * z * (1.0f + erff(z * 0.7071067811865476f));
  return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}
// The expert's weight w for the token goes onto the activation's output, act(z) w, or (MOE_ACT_WEIGHT_IN set in
// `act`) onto its input, act(w z): the expert then works on w times the token's row, since U (w x) = w (U x).
#define MOE_ACT_WEIGHT_IN 16
__device__ __forceinline__ float moe_weighted_activation(float z, float w, int act) {
  return (act & MOE_ACT_WEIGHT_IN) ? moe_activation(z * w, act & 15) : moe_activation(z, act) * w;
}
