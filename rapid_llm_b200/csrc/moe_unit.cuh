// The gated unit of the routed feed-forward, one for all of its product kernels.
#pragma once

namespace rl {

// The gated unit of an expert from its two float32 products: SiLU(g) * u, or with limit > 0 the clamped unit
// min(g, limit) * sigmoid(alpha * min(g, limit)) * (clamp(u, -limit, limit) + 1).
__device__ __forceinline__ float moe_unit(float g, float u, float limit, float alpha) {
  if (limit > 0.0f) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return g / (1.0f + expf(-alpha * g)) * (u + 1.0f);
  }
  return g / (1.0f + expf(-g)) * u;
}

// Sixteen of them, bit for bit, for a warp that has a multiprocessor's quarter to itself: a division's own test for odd
// operands keeps the next one from starting before it has ended.  The quotients come from an approximate reciprocal,
// refined once, and are corrected by their remainders, which leaves them rounded to nearest (Markstein, IBM Journal of
// Research and Development 34, 1990) while a remainder has room below its quotient; where one might not (also zeros,
// infinities, NaN) all sixteen are divided.
__device__ __forceinline__ void moe_units(float (&g)[16], float (&u)[16], float limit, float alpha, float (&out)[16]) {
  float by[16];
  bool plain = true;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    if (limit > 0.0f) {
      g[j] = fminf(g[j], limit);
      u[j] = fminf(fmaxf(u[j], -limit), limit) + 1.0f;
    }
    by[j] = 1.0f + expf(limit > 0.0f ? -alpha * g[j] : -g[j]);
    float inverse = __fdividef(1.0f, by[j]);
    inverse = fmaf(fmaf(-by[j], inverse, 1.0f), inverse, inverse);
    const float near = g[j] * inverse;
    plain = plain && by[j] < 0x1p126f && fabsf(near) > 0x1p-100f && fabsf(g[j]) < 0x1p100f;
    out[j] = fmaf(fmaf(-by[j], near, g[j]), inverse, near) * u[j];
  }
  if (plain) return;
#pragma unroll
  for (int j = 0; j < 16; ++j) out[j] = g[j] / by[j] * u[j];
}

}  // namespace rl
