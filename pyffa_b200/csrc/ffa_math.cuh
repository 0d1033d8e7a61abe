// ffa_math.cuh -- float64 reciprocals of the push kernels (device code).
#pragma once

namespace ffa {

// x^(-1/2) and 1 / x for normal positive x, without a branch: the hardware's
// approximation (relative error about 2^-20, PTX ISA rsqrt.approx / rcp.approx)
// refined by one third-order Householder step.  With e = 1 - x y^2 (or 1 - x y)
// the series of (1 - e)^(-1/2) (or 1 / (1 - e)) to e^2 leaves 5/16 e^3 (e^3),
// below 2^-58, so the result is right to about an ulp.  The library functions
// add range tests whose branches keep a step's chains from overlapping.  Zero,
// subnormal and infinite arguments give NaN (so callers keep them out), negative
// ones NaN (rsqrt64) or the reciprocal (rcp64).
__device__ __forceinline__ double rsqrt64(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x * y, y, 1.0);
    return fma(y * e, fma(e, 0.375, 0.5), y);
}

__device__ __forceinline__ double rcp64(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

}  // namespace ffa
