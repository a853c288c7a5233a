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

// The same for results that are rounded to bfloat16 behind them: the exponential and the quotient by the fast functions, good to a few
// 2^-22 (nothing overflows: the exponent is never positive) against the rounding's 2^-9.  The exact ones have branches, which keeps
// a thread's sixteen results of a tile from overlapping: the tile's read-out took longer than its multiplication.
__device__ __forceinline__ float fast_sigmoid(float z) {
  const float e = __expf(-fabsf(z)), r = __fdividef(1.f, 1.f + e);
  return z >= 0.f ? r : e * r;
}
__device__ __forceinline__ float silu_glu_bf16(float gate, float up, float s) {
  const float g = s * gate;
  return g * fast_sigmoid(g) * (s * up);
}
__device__ __forceinline__ float clamped_glu_bf16(float gate, float up, float limit) {
  const float g = fminf(gate, limit), u = fminf(fmaxf(up, -limit), limit);
  return g * fast_sigmoid(1.702f * g) * (u + 1.f);
}

}  // namespace ms
