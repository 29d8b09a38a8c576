// a0 / b and a1 / b rounded to nearest, as the reference divides the projected
// coordinates by their depth, from one reciprocal instead of two divisions.
// With y = RN(1 / b), q = RN(a y) lies within two units of the last place of
// a / b; one residual correction brings it within one, and then
// RN(q + (a - q b) y) is the correctly rounded quotient (the residual is exact
// in one fused multiply-add; P. W. Markstein, IBM J. Res. Dev. 34(1), 1990).
//
// This holds while neither the residuals nor y leave the normal floats: for
// 2^-100 <= |b| <= 2^120 and quotients of at least 2^-26 in magnitude that do
// not overflow.  For b = 0, or a quotient that overflows, the results are
// infinite or NaN, though not always the same of the two; smaller quotients
// come out below 2^-25.  tests/test_quot_gpu.py compares it with the IEEE
// division over random operands and over quotients next to the middle of two
// floats.
#pragma once

namespace mvs {

__device__ __forceinline__ void quotients(float a0, float a1, float b, float &q0, float &q1)
{
    const float y = __frcp_rn(b);
    float p0 = __fmul_rn(a0, y), p1 = __fmul_rn(a1, y);
    p0 = __fmaf_rn(__fmaf_rn(-p0, b, a0), y, p0);
    p1 = __fmaf_rn(__fmaf_rn(-p1, b, a1), y, p1);
    q0 = __fmaf_rn(__fmaf_rn(-p0, b, a0), y, p0);
    q1 = __fmaf_rn(__fmaf_rn(-p1, b, a1), y, p1);
}

}  // namespace mvs
