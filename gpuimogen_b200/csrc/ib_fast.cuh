// ib_fast.cuh -- reciprocal and square root of the product build's flux arithmetic.
//
// The compiler's FP64 division and square root round correctly for every operand: a longer
// refinement and, at each call, a test and a branch to a slow path.  An HLLC sweep takes ten of them
// per cell and stage, on its critical path.  The forms here start from the hardware's documented
// seeds (rcp.approx.ftz.f64 and rsqrt.approx.ftz.f64, good to about 2^-20) and take one step of the
// third-order Householder iteration, whose error is of the order of the seed's cubed:
//     1/x:      e = 1 - x y,     y (1 + e + e^2)
//     sqrt(x):  s = x y, e = 1 - s y,  s (1 + e/2 + 3/8 e^2)
// Results are within one unit in the last place; sqrt_fast(0) = 0, square roots of negative numbers
// are NaN, and where IEEE gives an infinity (1/0, the root of infinity) the result is NaN: the sweeps
// turn either into a non-finite flux.  A branch to the IEEE operations for such operands was measured
// and not kept: its registers spill in every kernel (256^3 HLLC y sweep 0.604 ms with it out of
// line, 0.561 without).
#pragma once

#include <cuda_runtime.h>

namespace ib {

// 1/x; |x| a normal number below 2^1022
__device__ __forceinline__ double rcp_fast(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// 1/x for x >= 0 that may be subnormal or zero: finite there (the seed is that of the smallest normal
// number), for quotients whose numerator is then zero
__device__ __forceinline__ double rcp_fast_pos(double x)
{
    double y;
    const double z = __hiloint2double(max((unsigned)__double2hiint(x), 0x00100000u), 0);
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(z));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// a / x from ix, the rounded reciprocal: one correction by the remainder, whose error is that of the division
__device__ __forceinline__ double quotient_fast(double a, double x, double ix)
{
    const double q = a * ix;
    return fma(fma(-q, x, a), ix, q);
}

// sqrt(x); the seed's operand is at least the smallest normal number (unsigned: negative ones pass)
__device__ __forceinline__ double sqrt_fast(double x)
{
    double y;
    const double z = __hiloint2double(max((unsigned)__double2hiint(x), 0x00100000u), 0);
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(z));
    const double s = x * y;
    const double e = fma(-s, y, 1.0);
    return fma(s * e, fma(e, 0.375, 0.5), s);
}

// single precision: the hardware's own operations
__device__ __forceinline__ float rcp_fast(float x) { return 1.0f / x; }
__device__ __forceinline__ float rcp_fast_pos(float x) { return 1.0f / x; }
__device__ __forceinline__ float sqrt_fast(float x) { return sqrtf(x); }

}  // namespace ib
