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
// N numbers and their weights, the choice outside: the same bits from a quarter of the code (an epilogue runs it once a unit of work,
// from memory that the instruction cache does not hold yet)
template <int ACT, int N> __device__ __forceinline__ void moe_weighted_act_all(float (&z)[N], const float (&w)[N], bool weight_in) {
#pragma unroll
  for (int i = 0; i < N; ++i) z[i] = weight_in ? z[i] * w[i] : z[i];
  if (ACT == 1) {
    ll_silu_all<N>(z);
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) z[i] = moe_activation(z[i], ACT);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) z[i] = weight_in ? z[i] : z[i] * w[i];
}
template <int N> __device__ __forceinline__ void moe_weighted_act_any(float (&z)[N], const float (&w)[N], int act) {
  const bool in = (act & MOE_ACT_WEIGHT_IN) != 0;
  act &= MOE_ACT_WEIGHT_IN - 1;
  if (act == 0) moe_weighted_act_all<0, N>(z, w, in);
  else if (act == 1) moe_weighted_act_all<1, N>(z, w, in);
  else if (act == 2) moe_weighted_act_all<2, N>(z, w, in);
  else moe_weighted_act_all<3, N>(z, w, in);
}
