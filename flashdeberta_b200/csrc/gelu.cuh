// GELU(v) = v * Phi(v) with Phi from the complementary error function in the rational form of Abramowitz & Stegun 7.1.26
// (absolute error 1.5e-7, far below half a bf16 ulp of the result): one reciprocal, one exponential and nine FMAs per
// element, about half of what erff costs — with erff the epilogue of the linear kernel would be longer than its main loop.
#pragma once

#include "sm100_ptx.cuh"

namespace fdb {

// v * Phi(v) with Phi(v) = 1/2 erfc(-v / sqrt 2):  v * Phi(v) = v / 2 + |v| * (1/2 - q),  q = 1/2 erfc(|v| / sqrt 2), for a pair.
// Two-wide forms where they exist: a third fewer instructions beside a main loop that is bound by power at large sizes
// (16384 x 768 -> 3072: 75.8 -> 74.7 us, against 63 us without the activation).
__device__ __forceinline__ uint64_t gelu_erf2(uint64_t v) {
  const uint64_t av = v & 0x7fffffff7fffffffull;
  const uint64_t z = ptx::mul_f32x2(av, ptx::pack_f32x2(0.70710678118654752f, 0.70710678118654752f));
  float d0, d1, e0, e1, t0, t1;
  ptx::unpack_f32x2(ptx::fma_f32x2(ptx::pack_f32x2(0.3275911f, 0.3275911f), z, ptx::pack_f32x2(1.f, 1.f)), d0, d1);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t0) : "f"(d0));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t1) : "f"(d1));
  ptx::unpack_f32x2(ptx::mul_f32x2(ptx::mul_f32x2(z, z), ptx::pack_f32x2(-1.4426950408889634f, -1.4426950408889634f)), e0, e1);
  const uint64_t e = ptx::pack_f32x2(ptx::ex2(e0), ptx::ex2(e1)), t = ptx::pack_f32x2(t0, t1);
  auto both = [](float c) { return ptx::pack_f32x2(c, c); };
  uint64_t p = ptx::fma_f32x2(both(-0.5f * 1.061405429f), t, both(-0.5f * -1.453152027f));  // negated: h = 1/2 - p t e below
  p = ptx::fma_f32x2(p, t, both(-0.5f * 1.421413741f));
  p = ptx::fma_f32x2(p, t, both(-0.5f * -0.284496736f));
  p = ptx::fma_f32x2(p, t, both(-0.5f * 0.254829592f));
  const uint64_t h = ptx::fma_f32x2(ptx::mul_f32x2(p, t), e, both(0.5f));
  return ptx::fma_f32x2(av, h, ptx::mul_f32x2(v, both(0.5f)));
}

}  // namespace fdb
