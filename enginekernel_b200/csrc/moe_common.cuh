// What the experts' products share: the activations between their two products.
#pragma once
#include "common.cuh"

namespace ek {

constexpr int ACT_RELU2 = 1, ACT_SILU = 2, ACT_GELU_TANH = 3, ACT_CLAMPED = 4;      // 0: none

__device__ __forceinline__ float activate(float z, int act) {
  if (act == ACT_RELU2) { const float r = fmaxf(z, 0.f); return r * r; }
  if (act == ACT_SILU) return z / (1.f + expf(-z));
  if (act == ACT_GELU_TANH) return 0.5f * z * (1.f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
  return z;
}

// act(gate) * up; the clamped form is g sigmoid(1.702 g) (u + 1) with g = min(gate, limit), u = clamp(up, -limit, limit).
__device__ __forceinline__ float gated_value(float gate, float up, int act, float limit) {
  if (act == ACT_CLAMPED) {
    const float g = fminf(gate, limit), u = fminf(fmaxf(up, -limit), limit);
    return g / (1.f + expf(-1.702f * g)) * (u + 1.f);
  }
  return activate(gate, act) * up;
}

}  // namespace ek
