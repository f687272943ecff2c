// Quotients rounded to nearest without a branch between them.
#pragma once
#include "common.cuh"

namespace vb {

// a / d to the nearest, eight at a time and d >= 1: reciprocal, one Newton step, quotient, one correction by the exact remainder (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. R&D 34, 1990).  The corrected quotient is right
// where the reciprocal is.  From an estimate within two units of the last place one step leaves it wrong for a few dozen of the 2^23
// mantissas, and of those three of the largest have dividends that it spoils (tests/test_quotients.py walks them).  These mantissas, and
// dividends, divisors or quotients so large or small that a remainder would leave the normal range, send all eight to the division
// itself; there is no branch between the eight.  Zeros are right as they are, and a NaN stays one on either way.
__device__ __forceinline__ void div8(float (&a)[8], const float (&d)[8]) {
  float q[8], large = 0.f, small = 1.f;
  uint32_t mantissa = 0u;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d[i]));
    y = fmaf(fmaf(-d[i], y, 1.f), y, y);
    const float q0 = a[i] * y;
    const bool zero = a[i] == 0.f;
    q[i] = zero ? q0 : fmaf(fmaf(-q0, d[i], a[i]), y, q0);
    large = fmaxf(large, fmaxf(fabsf(a[i]), d[i]));
    small = fminf(small, zero ? 1.f : fabsf(q0));
    mantissa = max(mantissa, __float_as_uint(d[i]) | 0xff800000u);
  }
  if (!(large < 0x1p100f && small > 0x1p-100f) || mantissa >= 0xfffffffbu) {
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = a[i] / d[i];
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) a[i] = q[i];
}

}  // namespace vb
