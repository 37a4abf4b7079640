// icb_div.cuh — division by a number that stays the same for a whole launch.
// The double forms use IEEE operations only, so a host compiler evaluates
// them alike (the CPU test builds this header with one).
#pragma once

#include <cmath>
#include <cstdint>

namespace icb {

// a / b for a divisor that stays the same for a whole launch, y = RN(1 / b),
// b > 0 in [2^-300, 2^300] (checked where y is formed: y = 0 otherwise): the
// correctly rounded quotient by Markstein's correction (IBM J. Res. Dev. 34,
// 1990: with y the rounded reciprocal and q within an ulp of a / b,
// RN(q + RN(a - b q) y) is RN(a / b)); the first correction brings q = a y
// within an ulp.  Five dependent operations instead of the general
// division's reciprocal iteration and range handling.  Dividends outside
// [2^-623, 2^577] (and NaN) take the general division, zero keeps a y.
static __device__ __noinline__ double div_general(double a, double b) { return a / b; }
__device__ __forceinline__ double div_by(double a, double b, double y) {
    const double q = a * y;
    const uint32_t ea = (static_cast<uint32_t>(__double2hiint(a)) >> 20) & 0x7ffu;
    if (ea - 400u >= 1200u || y == 0.0) return (a == 0.0 && y != 0.0) ? q : div_general(a, b);
    const double q1 = fma(fma(-b, q, a), y, q);
    return fma(fma(-b, q1, a), y, q1);
}
__device__ __forceinline__ double div_reciprocal(double b) {
    const uint32_t eb = (static_cast<uint32_t>(__double2hiint(b)) >> 20);      // b > 0: sign bit clear
    return eb - 723u < 601u ? 1.0 / b : 0.0;
}
#ifdef __CUDACC__
// Float forms: one hardware reciprocal per launch instead of one per step
// (the values of -prec-div=false division, a times that reciprocal).
__device__ __forceinline__ float div_by(float a, float, float y) { return a * y; }
__device__ __forceinline__ float div_reciprocal(float b) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
    return y;
}
#endif

}  // namespace icb
