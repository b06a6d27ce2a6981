// fh_quot.cuh -- a / b correctly rounded from a reciprocal of b made once, for
// divisions on the critical path of every step (an FP32 division takes ~300
// cycles there).
#pragma once
#include <math.h>

// a / b from r = RN(1 / b): the quotient corrected by two exact remainders
// (Markstein, IBM J. Res. Dev. 34, 1990).  A remainder is exact while it stays
// above the smallest subnormal, so a is taken times 2^64; where the quotient
// then leaves [2^-125, 2^60], or is not finite, the division itself runs.
__host__ __device__ __forceinline__ float fh_quot(float a, float b, float r) {
  const float s = a * 0x1p64f;
  float q = s * r;
  q = fmaf(fmaf(-q, b, s), r, q);  // faithful
  q = fmaf(fmaf(-q, b, s), r, q);  // correctly rounded
  q *= 0x1p-64f;
  const float m = fabsf(q);
  return m >= 0x1p-125f && m <= 0x1p60f ? q : a / b;
}
