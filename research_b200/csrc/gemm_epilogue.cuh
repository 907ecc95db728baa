// Activations that the products' epilogues apply to fp32 sums.
#pragma once
#include "common.cuh"

namespace rb {

__device__ __forceinline__ float rcp_epi(float x) {      // x within 2^-126 .. 2^126 or infinite
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// n / (1 + 2^t) as the IEEE division gives it, without its branch to a slow path for every element, which keeps the compiler from
// overlapping them: it took a 256 x 256 tile's epilogue 30000 cycles beside 7000 of main loop (K = 896). 9820 x 9728 x 896 with silu:
// 238 -> 134 us, with a folded norm on the one-CTA kernel 272 -> 157 (__fdividef: 133 and 158, but 2 units in the last place, and 0 for a
// denominator above 2^126). An approximate quotient and one step of residual correction (P. W. Markstein, Computation of elementary
// functions on the IBM RISC System/6000 processor, IBM J. Res. Dev. 34, 1990), both sides scaled by a quarter to keep the reciprocal a normal
// number. 2^t below 2^-126 may be 0 beside 1. Equal to the division in every bit over 2^28 gates, but for the sign of a zero gate.
__device__ __forceinline__ float quotient_epi(float n, float t) {
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(t));
  const float d = fmaf(0.25f, e, 0.25f), r = rcp_epi(d);
  n *= 0.25f;
  const float q = n * r, rest = fmaf(-q, d, n);
  return fabsf(rest) < INFINITY ? fmaf(rest, r, q) : q;      // infinite sides have no remainder
}

__device__ __forceinline__ float clamped_glu_epi(float g, float u, float limit) {
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  return quotient_epi(g, (-1.702f * g) * 1.44269504f) * (u + 1.f);
}

// silu(gate) * up with the rounding points of the unfused path: bf16(gate), bf16(silu), bf16(up); the caller rounds the product.
__device__ __forceinline__ float swiglu_epi(float gate, float up) {
  const float g = __bfloat162float(__float2bfloat16_rn(gate)), u = __bfloat162float(__float2bfloat16_rn(up));
  return __bfloat162float(__float2bfloat16_rn(quotient_epi(g, g * -1.44269504f))) * u;
}

// Gradient to a logit x of a row with log-sum-exp l: of the target's log-probability (upstream gradient glp) and of the row's entropy H
// (gent).
__device__ __forceinline__ float dlogit_epi(float x, float l, float glp, float gent, float H, bool is_target) {
  const float lp = x - l;
  const float p = __expf(lp);
  return glp * ((is_target ? 1.f : 0.f) - p) - gent * p * (lp + H);
}

}  // namespace rb
