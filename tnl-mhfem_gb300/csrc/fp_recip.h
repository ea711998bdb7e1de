// FP64 reciprocals and quotients with few operations on the FP64 pipe.
//
// GB300 issues FP64 at 1/57 of the FP32 rate and with 64 cycles of latency.
// An IEEE division takes 561 cycles, and where many are needed (the row scaling
// of the assembly, the LU pivots of the cell kernel) about as much of the FP64
// pipe as the rest of a face row.
//
// The header compiles as plain C++ too, so the host test suite compares both
// functions with the compiler's (IEEE) division.
#pragma once

#include <math.h>
#include <cstdint>
#include <cstring>

#include "fp_convert.h"

namespace mhfem {

#if defined(__CUDACC__)
static __host__ __device__ __noinline__ double div_ieee(double a, double b) { return a / b; }
#else
inline double div_ieee(double a, double b) { return a / b; }
#endif

MHFEM_HD int fp64_exponent(double v)
{
    uint64_t b;
    std::memcpy(&b, &v, sizeof b);
    return (int)((b >> 52) & 0x7ff);
}

// 1 / d.  One third-order step from an FP32 reciprocal estimate r0: with u = 1 -
// d r0, 1/d = r0 / (1 - u) = r0 (1 + u + u^2 + ...), truncated after u^2
// (Halley's iteration for f(r) = 1/r - d, cubic convergence): r = r0 + r0 (u +
// u^2).  The estimate's relative error is below 2^-22, so the truncation error
// is below 2^-66, under FP64 rounding: the result is within an ulp of the
// correctly rounded one.  The FP32 operand and the FP32 estimate move between
// the two IEEE formats by integer bit operations (sign, rebiased exponent,
// truncated mantissa), so the FP64 pipe only sees three fused multiply-adds.
// Magnitudes outside [2^-100, 2^100] (and 0, inf, NaN) take the IEEE division.
MHFEM_HD double recip_newton(double d)
{
    uint64_t b;
    std::memcpy(&b, &d, sizeof b);
    const int e = fp64_exponent(d);
    if (e < 1023 - 100 || e > 1023 + 100) return div_ieee(1.0, d);
    const uint32_t fb = ((uint32_t)(b >> 32) & 0x80000000u) | ((uint32_t)(e - 1023 + 127) << 23) |
                        (uint32_t)((b >> 29) & 0x7fffffu);
    float f, rf;
    std::memcpy(&f, &fb, sizeof f);
#if defined(__CUDA_ARCH__)
    rf = __frcp_rn(f);
#else
    rf = 1.0f / f;
#endif
    uint32_t rb;
    std::memcpy(&rb, &rf, sizeof rb);
    const uint64_t r64 = ((uint64_t)(rb & 0x80000000u) << 32) | ((uint64_t)(((rb >> 23) & 0xffu) - 127u + 1023u) << 52) |
                         ((uint64_t)(rb & 0x7fffffu) << 29);
    double r;
    std::memcpy(&r, &r64, sizeof r);
    const double u = fma(-d, r, 1.0);
    return fma(r, fma(u, u, u), r);
}

// a / b with r = recip_newton(b) at hand: q = a r and one correction by the
// remainder a - q b, which a fused multiply-add forms exactly (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// IBM J. Res. Develop. 34, 1990), so that the quotient is rounded once, like the
// division's: two operations more than the product.  Where the reciprocal was not
// formed that way, or the remainder could be lost below the normal numbers, the
// IEEE division: a quotient of two numbers near either end of the range is an
// ordinary number although the reciprocal is not.
MHFEM_HD bool quotient_in_range(double a, double b)
{
    const int ea = fp64_exponent(a), eb = fp64_exponent(b);
    return ea >= 1023 - 800 && ea <= 1023 + 800 && eb >= 1023 - 100 && eb <= 1023 + 100;
}
MHFEM_HD double quotient(double a, double b, double r)
{
    // the test beside the FP64 operations, not before them
    const double q = a * r, v = fma(fma(-q, b, a), r, q);
    return quotient_in_range(a, b) ? v : div_ieee(a, b);
}
MHFEM_HD double quotient(double a, double b) { return quotient(a, b, recip_newton(b)); }
// The same without the correction, within two units in the last place: for a
// factor whose own rounding does not reach the result.
MHFEM_HD double quotient_product(double a, double b, double r)
{
    return quotient_in_range(a, b) ? a * r : div_ieee(a, b);
}

}  // namespace mhfem
