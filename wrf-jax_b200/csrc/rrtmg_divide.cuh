// Correctly rounded reciprocal and quotient for operands known to be in range.
//
// The radiation kernels divide some thirty times per layer and g-point, and
// results must equal IEEE division bit for bit.  With operands that are known
// to be normal and away from the ends of the exponent range, Markstein's
// scheme ("Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34, 1990, theorems on division) needs no test
// of its operands, and quotients by the same divisor share the reciprocal:
//   * y = the reciprocal approximation improved by one Newton step with fused
//     multiply-adds; it is the correctly rounded reciprocal for every binary32
//     significand (checked exhaustively, tests/test_gpu_divide.py);
//   * q = a y, corrected by its exact remainder, is within one unit in the
//     last place, and corrected once more it is the correctly rounded a / b.
// Ranges: |b| and |a| in [2^-100, 2^100] (a positive zero a is fine), and the
// quotient's size in [2^-120, 2^117].  There no step leaves the normal numbers and
// the remainder a - b q, a multiple of 2^-148, is exact.
#pragma once

namespace rrtmg {

__device__ __forceinline__ float recip_in_range(float b) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
  return __fmaf_rn(__fmaf_rn(-b, y, 1.0f), y, y);
}

// a / b given y = recip_in_range(b)
__device__ __forceinline__ float quotient_by(float a, float b, float y) {
  float q = a * y;
  q = __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
  return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}

__device__ __forceinline__ float quotient_in_range(float a, float b) { return quotient_by(a, b, recip_in_range(b)); }

}  // namespace rrtmg
