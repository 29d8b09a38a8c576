// Division of a window sum by the window side, for the reference-arithmetic
// sweep (sweep.cu) and its exhaustive check (tests/cuda/div_win_check.cu).
#pragma once

#include <math.h>

namespace mvs {

// x / WIN rounded to nearest, as the reference divides its window sums by the
// window side, in three instructions instead of a division: with
// y = RN(1 / WIN), q = RN(x y) is within one ulp of x / WIN, the residual
// x - q WIN is exact in one fused multiply-add, and RN(q + residual * y) is
// the correctly rounded quotient (Markstein's correction: P. W. Markstein,
// IBM J. Res. Dev. 34(1), 1990).  Zero, infinite and NaN x keep q, which is
// then exact (the correction would turn -0 into +0 and inf into NaN).
// tests/test_div_win_gpu.py compares it with the IEEE division for every
// float bit pattern and every window side 3..15: no difference.
template <int WIN>
__device__ __forceinline__ float div_win(float x)
{
    constexpr float d = (float)WIN, y = 1.f / (float)WIN;
    const float q = __fmul_rn(x, y);
    const float r = __fmaf_rn(-q, d, x);
    return isfinite(x) && x != 0.f ? __fmaf_rn(r, y, q) : q;
}

// Two floats in a register pair, for the packed FP32 instructions (each half
// rounds as the scalar instruction does).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 p, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// div_win of both halves
template <int WIN>
__device__ __forceinline__ void div_win2(f32x2 x, float &oa, float &ob)
{
    constexpr float d = (float)WIN, y = 1.f / (float)WIN;
    const f32x2 yy = pack2(y, y), q = mul2(x, yy), z = fma2(fma2(q, pack2(-d, -d), x), yy, q);
    float xa, xb, qa, qb, za, zb;
    unpack2(x, xa, xb);
    unpack2(q, qa, qb);
    unpack2(z, za, zb);
    oa = isfinite(xa) && xa != 0.f ? za : qa;
    ob = isfinite(xb) && xb != 0.f ? zb : qb;
}

}  // namespace mvs
