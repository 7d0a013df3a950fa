// The SiLU gate of many values at once (epilogues of the tcgen05 products).
#pragma once
#include "common.cuh"

namespace {

// g / (1 + exp(-alpha g)) of COUNT values. A division of its own for each, with its test for the rare operands, leaves a warp with
// one chain of some 80 cycles after the other (5.6 us for a 128 x 256 tile, staged 5.7); here the quotients of a thread go side by side:
// Newton's step for the reciprocal of a denominator between 1 and 2^116, then Markstein's correction of the quotient by its
// remainder (IBM J. Res. Dev. 34, 1990), which rounds as the division does. With alpha g beyond 80 the denominator is 1. Below -80 one
// plus it is it, and g exp(alpha g) stands for the quotient: within two roundings of the division's down to -88.7, where the
// division's denominator leaves the range and its quotient is -0; this one goes on down to 1e-45.
template <int COUNT>
__device__ __forceinline__ void silu_all(float (&g)[COUNT], float alpha = 1.f) {
  float v[COUNT];
  bool plain = true;
#pragma unroll
  for (int i = 0; i < COUNT; ++i) plain &= fabsf(alpha * g[i]) <= 80.f;  // not for NaN
#pragma unroll
  for (int i = 0; i < COUNT; ++i) {
    const float d = 1.0f + expf(-alpha * g[i]);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    r = fmaf(r, fmaf(-d, r, 1.0f), r);
    const float q = g[i] * r;
    v[i] = fmaf(fmaf(-d, q, g[i]), r, q);
  }
  if (!__all_sync(0xffffffffu, plain)) {
#pragma unroll
    for (int i = 0; i < COUNT; ++i) {
      const float z = alpha * g[i];
      v[i] = z > 80.f ? g[i] : z < -80.f ? g[i] * expf(z) : v[i];
    }
  }
#pragma unroll
  for (int i = 0; i < COUNT; ++i) g[i] = v[i];
}

}  // namespace
