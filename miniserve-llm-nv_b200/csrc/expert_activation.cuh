// What an expert does between its two products, as an epilogue of the first.
#pragma once

#include "common.cuh"

namespace ms {

enum : int { kActNone = 0, kActReluSquare = 1, kActClampedGlu = 2, kActSiluGlu = 3 };

// silu(s gate) (s up): the expert computed on s times its input (s = 1 where the weight is applied to its output).
__device__ __forceinline__ float silu_glu(float gate, float up, float s) {
  const float g = s * gate;
  return g / (1.f + expf(-g)) * (s * up);
}

// g = min(gate, limit), u = clamp(up, -limit, limit); g sigmoid(1.702 g) (u + 1)
__device__ __forceinline__ float clamped_glu(float gate, float up, float limit) {
  const float g = fminf(gate, limit), u = fminf(fmaxf(up, -limit), limit);
  return g / (1.f + expf(-1.702f * g)) * (u + 1.f);
}

}  // namespace ms
