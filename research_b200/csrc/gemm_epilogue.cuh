// Activations that the products' epilogues apply to fp32 sums. The quotients are __fdividef: an IEEE division is a branch to a
// slow path for every element, which keeps the compiler from overlapping them, and took a 256 x 256 tile's epilogue 30000 cycles
// beside 7000 of main loop (K = 896). 9820 x 9728 x 896 with silu: 317 -> 184 us.
// Rounded to bf16 the results' error against 64 bits is the same: 3.557e-3 silu, 1.658e-3 clamped, of the result's norm.
#pragma once
#include "common.cuh"

namespace rb {

__device__ __forceinline__ float clamped_glu_epi(float g, float u, float limit) {
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  return __fdividef(g, 1.f + __expf(-1.702f * g)) * (u + 1.f);
}

// silu(gate) * up with the rounding points of the unfused path: bf16(gate), bf16(silu), bf16(up); the caller rounds the product.
__device__ __forceinline__ float swiglu_epi(float gate, float up) {
  const float g = __bfloat162float(__float2bfloat16_rn(gate)), u = __bfloat162float(__float2bfloat16_rn(up));
  return __bfloat162float(__float2bfloat16_rn(silu_fast(g))) * u;
}

// Gradient to a logit x of a row with log-sum-exp l: of the target's log-probability (upstream gradient glp) and of the row's entropy H
// (gent).
__device__ __forceinline__ float dlogit_epi(float x, float l, float glp, float gent, float H, bool is_target) {
  const float lp = x - l;
  const float p = __expf(lp);
  return glp * ((is_target ? 1.f : 0.f) - p) - gent * p * (lp + H);
}

}  // namespace rb
