// 1/sqrt(x) and 1/x of normal positive numbers: the documented approximate instructions (rsqrt.approx.ftz.f64,
// rcp.approx.ftz.f64) and one step of a third-order iteration each.  In the pair and matrix kernels, whose
// arguments are squared distances and damping denominators, they leave out what the library functions
// add for special cases.  gfnff_reciprocal_ulps compares both with the library functions.
#pragma once

// y (1 + e/2 + 3/8 e^2), e = 1 - x y^2: Halley's third-order iteration for y^-2 - x in Householder's form
// (A. S. Householder, The Numerical Treatment of a Single Nonlinear Equation, 1970, chapter 4),
// the first terms of the binomial series of (1 - e)^(-1/2)
__device__ __forceinline__ double rsqrt_pos(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

// y (1 + e + e^2), e = 1 - x y: the third-order hyperpower iteration (M. Altman, Pacific J. Math. 10 (1960)
// 1107-1113)
__device__ __forceinline__ double rcp_pos(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
