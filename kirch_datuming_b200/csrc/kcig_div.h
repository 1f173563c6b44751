// Divisions by a known divisor through its reciprocal, correctly rounded: the
// quotients of the traveltime sweeps (kcig_eikods.cu).  Also compiled for the
// host, where the tests compare them with the machine's division.
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define KCIG_DIV_FN __device__ __forceinline__
#define KCIG_DIV_MUL(a, b) __dmul_rn(a, b)
#define KCIG_DIV_FMA(a, b, c) __fma_rn(a, b, c)
#define KCIG_DIV_MULF(a, b) __fmul_rn(a, b)
#define KCIG_DIV_FMAF(a, b, c) __fmaf_rn(a, b, c)
#define KCIG_DIV_DIVF(a, b) __fdiv_rn(a, b)
#else
#define KCIG_DIV_FN static inline
#define KCIG_DIV_MUL(a, b) ((a) * (b))
#define KCIG_DIV_FMA(a, b, c) fma(a, b, c)
#define KCIG_DIV_MULF(a, b) ((a) * (b))
#define KCIG_DIV_FMAF(a, b, c) fmaf(a, b, c)
#define KCIG_DIV_DIVF(a, b) ((a) / (b))
#endif

namespace kcig {

// a / b correctly rounded, y = RN(1 / b): Markstein's theorem (IBM J. Res.
// Dev. 34, 1990) -- with q within an ulp of a / b and r = a - b q exact, q +
// r y rounds to RN(a / b); the first correction brings q within an ulp.
// The divisors of a point's update are few (sums of the axes' weights), so
// their reciprocals come from the host, and the serial chain that bounds a
// step shortens: five dependent operations for a general division's dozen.
// The operands are sums and products of a few FP32 values, whose quotients and
// remainders are far from the ends of the FP64 range.
KCIG_DIV_FN double div_by(double a, double b, double y)
{
    double q = KCIG_DIV_MUL(a, y);
    q = KCIG_DIV_FMA(KCIG_DIV_FMA(-b, q, a), y, q);
    return KCIG_DIV_FMA(KCIG_DIV_FMA(-b, q, a), y, q);
}

// The same in FP32 for a divisor in 2^-40 .. 2^40.  A dividend below 2^-80,
// whose remainder could underflow, or above 2^86 (a time that was never
// reached is FLT_MAX: its quotient by a squared spacing below 1 overflows),
// infinities and NaN go through the general division, as every dividend of
// another divisor does.
struct DivF {
    float b, y, hi;  // divisor, its reciprocal, largest quick dividend; other divisors: 0, 0, -1
    float div;       // the divisor, for the general division
};

inline DivF div_prepare(float b)
{
    if (b >= 9.09494702e-13f && b <= 1.09951163e12f) return {b, 1.0f / b, 7.73712525e25f, b};
    return {0.0f, b > 0.0f ? 0.0f : NAN, -1.0f, b};
}

KCIG_DIV_FN bool div_quick(float a, const DivF &d)
{
    return fabsf(a) >= 8.27180613e-25f && fabsf(a) <= d.hi;
}

// a / b for a quick dividend or 0
KCIG_DIV_FN float div_known(float a, const DivF &d)
{
    float q = KCIG_DIV_MULF(a, d.y);
    q = KCIG_DIV_FMAF(KCIG_DIV_FMAF(-d.b, q, a), d.y, q);
    return KCIG_DIV_FMAF(KCIG_DIV_FMAF(-d.b, q, a), d.y, q);
}

// a / b for any dividend
KCIG_DIV_FN float div_by(float a, const DivF &d)
{
    return div_quick(a, d) || a == 0.0f ? div_known(a, d) : KCIG_DIV_DIVF(a, d.div);
}

}  // namespace kcig
