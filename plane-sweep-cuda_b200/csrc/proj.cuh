// The reference's projections of dual variables, (float)(x / d) with
// d = (double)fmaxf(1, (float)sqrt(s)) where s > 1, in double
// (kernels.cu:296-303, TGV2_kernels.cu:72-83, 355-362), without the IEEE
// double square root and divisions, which took a third of an iteration of the
// TV-L1 denoise (640x480, one launch per iteration, 7.2 us).
//
// Only the float nearest to a correctly rounded double is wanted.  So the
// square root and the quotients are formed in double by Newton steps (the
// classical iterations for sqrt and 1 / d and the residual-corrected
// quotient) from the hardware's approximate reciprocal square root, to within
// one unit of the double's last place, and rounded to float.  That float is
// the reference's unless the double lies within that distance of the middle
// between two floats, where the reference's own rounding decides.  There (low
// 29 bits of the double within 4 of half a float unit: one value in 2^26),
// and for quotients below the normal floats or s above 2^100, the IEEE
// operations are used.
//
// Conversions between float and double run at a sixteenth of the FP32 rate, so
// sqrt(s) is rounded to float precision by Veltkamp's splitting (T. J. Dekker,
// Numer. Math. 18, 1971: the high part of x split by 2^29 + 1 is x rounded to
// the nearest 24-bit value) instead of a conversion to float and back.
#pragma once

#include <stdint.h>

namespace mvs {

// At most 64 if `q` lies within 4 units of its last place of the middle of two
// floats (its low 29 bits are then within 4 of 2^28).
__device__ __forceinline__ unsigned tie_distance(double q)
{
    return (unsigned)__double2loint(q) * 8u + (0x80000000u + 32u);
}
constexpr unsigned kNormalHi = 0x38100000u;   // high word of 2^-126, the smallest normal float
constexpr unsigned kLargeHi = 0x46300000u;    // high word of 2^100

// x / d rounded to float by the IEEE operations of the reference.
static __device__ __noinline__ float proj_div_ieee(double x, double s)
{
    if (!(s > 1.0)) return (float)x;
    const double d = (double)fmaxf(1.f, (float)sqrt(s));
    return (float)(x / d);
}

// A projection that project() could not decide; g: sqrt(s) to the last place,
// y: its approximate inverse.  Where one component is exactly zero (the last
// row and column of an image, whose forward difference is zero) s is a square
// and its root a short sum of floats, exactly the middle of two floats once in
// a few hundred pixels: a residual below half a unit of g's last place shows
// that g is the rounded root, which the conversion then rounds as the
// reference does.  Everything else takes the IEEE operations.
template <int N>
__device__ __forceinline__ void project_tie(double s, double g, double y, const double (&x)[N], float (&out)[N])
{
    const double e = fma(-g, g, s), d = (double)(float)g;
    bool sure = (tie_distance(g) == 32u || tie_distance(g) > 64u) && fabs(e) < g * g * 0x1p-54 && s < 0x1p100;
    const double r = fma(y, fma(-d, y, 1.0), y);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        double v = x[i] * r;
        v = fma(fma(v, d, -x[i]), -r, v);   // the sign of a zero stays, as below
        if (tie_distance(v) <= 64u || (unsigned)__double2hiint(v) * 2u - 1u < 2u * kNormalHi - 1u) sure = false;
        out[i] = (float)v;
    }
    if (!sure) {
#pragma unroll
        for (int i = 0; i < N; ++i) out[i] = proj_div_ieee(x[i], s);
    }
}

// M independent projections of N components each, side by side (their chains
// of dependent operations overlap): out[m][i] = (float)(x[m][i] / d[m]) where
// s[m] > 1, (float)x[m][i] elsewhere (a NaN s included, as in the reference).
// Where s <= 1 a neighbour's projection runs with s = 1, for which the steps
// below give d = 1 and the quotient x exactly.
template <int M, int N>
__device__ __forceinline__ void project(const double (&s)[M], const double (&x)[M][N], float (&out)[M][N])
{
    bool any = false;
#pragma unroll
    for (int m = 0; m < M; ++m) any = any || !(s[m] <= 1.0);   // a NaN goes the long way
    if (!any) {
#pragma unroll
        for (int m = 0; m < M; ++m)
#pragma unroll
            for (int i = 0; i < N; ++i) out[m][i] = (float)x[m][i];
        return;
    }
    double s1[M], g[M], y[M], r[M], d[M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        s1[m] = s[m] <= 1.0 ? 1.0 : s[m];
        asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y[m]) : "d"(s1[m]));   // 1 / sqrt(s)
    }
#pragma unroll
    for (int m = 0; m < M; ++m) g[m] = s1[m] * y[m];
#pragma unroll
    for (int k = 0; k < 2; ++k)   // sqrt(s): the relative error squares in each step, then the last place
#pragma unroll
        for (int m = 0; m < M; ++m) g[m] = fma(fma(-g[m], g[m], s1[m]), 0.5 * y[m], g[m]);
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const double c = 536870913.0 * g[m];           // 2^29 + 1
        d[m] = c - (c - g[m]);                         // g rounded to 24 bits
        r[m] = fma(y[m], fma(-d[m], y[m], 1.0), y[m]); // 1 / d
    }
    unsigned tie[M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        tie[m] = tie_distance(g[m]);
        unsigned small = 0xffffffffu;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            double v = x[m][i] * r[m];
            // the last place of a double; the negated residual of a zero x has the other
            // sign than x, so the sum keeps x's
            v = fma(fma(v, d[m], -x[m][i]), -r[m], v);
            tie[m] = min(tie[m], tie_distance(v));
            small = min(small, (unsigned)__double2hiint(v) * 2u - 1u);
            out[m][i] = (float)v;
        }
        // a quotient below the normal floats (zero wraps around), or s above 2^100 or NaN
        if (small < 2u * kNormalHi - 1u || (unsigned)__double2hiint(s1[m]) > kLargeHi) tie[m] = 0u;
        // (float)x itself has no doubt; x is often the middle of two floats, a
        // short sum of floats
        if (s[m] <= 1.0) tie[m] = 0xffffffffu;
    }
    unsigned t = tie[0];
#pragma unroll
    for (int m = 1; m < M; ++m) t = min(t, tie[m]);
    if (t <= 64u) {
#pragma unroll
        for (int m = 0; m < M; ++m)
            if (tie[m] <= 64u) project_tie(s[m], g[m], y[m], x[m], out[m]);
    }
}

}  // namespace mvs
