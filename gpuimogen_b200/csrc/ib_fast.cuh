// ib_fast.cuh -- reciprocal and square root of the product build's flux arithmetic.
//
// The compiler's FP64 division and square root round correctly for every operand: a longer
// refinement and, at each call, a test and a branch to a slow path.  An HLLC sweep takes ten of them
// per cell and stage, on its critical path.  The forms here start from the hardware's documented
// seeds (rcp.approx.ftz.f64 and rsqrt.approx.ftz.f64, good to about 2^-20) and take one step of the
// third-order Householder iteration, whose error is of the order of the seed's cubed:
//     1/x:      e = 1 - x y,     y (1 + e + e^2)
//     sqrt(x):  s = x y, e = 1 - s y,  s (1 + e/2 + 3/8 e^2)
// In the operand ranges stated at each function the result is within one unit in the last place of the IEEE
// operation's.  Outside them the seeds flush, and the result is NaN (above 2^1022 the reciprocal is 0, and the
// root of a subnormal number infinite).  rcp_full and sqrt_full test their operand and take the IEEE operation
// there.  A test and a branch at each of the nine operations of a flux was measured and not kept: its registers
// spill in every kernel (256^3 HLLC y sweep 0.604 ms with the IEEE operation out of line, 0.561 without; one
// branch per flux, 0.586 against 0.535).  The sweeps let the NaN run instead: a NaN in one operation of a face
// reaches that face's mass flux and with it the densities beside it, so one test per cell and sweep finds every
// pencil with such an operand, and that pencil is computed again with IeeeOps (ieee_pencils in ib_sweep.cuh; in
// chunks, the same stages again).  Densities from 2^1000 on are sent there too, so that no flushed reciprocal
// passes.  (256^3 x/y/z, HLLC 0.469/0.535/0.553 ms without the test, which got such operands wrong, 0.465/0.541/
// 0.552 with it; HLL 0.512/0.551/0.559 and 0.532/0.564/0.572.)
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

namespace ib {

constexpr double kRcpTop = 4.4942328371557898e307;  // 2^1022: reciprocals from here on are subnormal

// 1/x; 2^-1022 <= |x| < 2^1022
__device__ __forceinline__ double rcp_fast(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// 1/x; x < 2^1022, normal or NaN; at zero and subnormal numbers finite and positive (the seed is that of the
// smallest normal number), for quotients whose numerator is then zero
__device__ __forceinline__ double rcp_fast_pos(double x)
{
    double y;
    const double z = __hiloint2double(max((unsigned)__double2hiint(x), 0x00100000u), 0);
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(z));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// sqrt(x); 2^-1022 <= x < infinity (negative x: NaN)
__device__ __forceinline__ double sqrt_fast(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double s = x * y;
    const double e = fma(-s, y, 1.0);
    return fma(s * e, fma(e, 0.375, 0.5), s);
}

// whether rcp_fast's range excludes x
__device__ __forceinline__ bool rcp_outside(double x)
{
    return 2u * (unsigned)__double2hiint(x) - 0x00200000u >= 0xff800000u;
}

// whether sqrt_fast's range excludes x (negative numbers, whose root is NaN, included)
__device__ __forceinline__ bool root_outside(double x) { return (unsigned)__double2hiint(x) - 0x00100000u >= 0x7fe00000u; }

// out of line, for places that seldom come to it
static __device__ __noinline__ double divide_ieee(double a, double b) { return a / b; }

// 1/x and sqrt(x) for every x: the IEEE operation's result where the short form does not reach
__device__ __forceinline__ double rcp_full(double x)
{
    double y = rcp_fast(x);
    if (rcp_outside(x)) y = 1.0 / x;
    return y;
}
__device__ __forceinline__ double sqrt_full(double x)
{
    double y = sqrt_fast(x);
    if (root_outside(x)) y = sqrt(x);
    return y;
}

// 1/x and sqrt(x) for every x without a call (in Xin-Jin the registers around one spill): the operand is scaled into
// the short form's range; zeros, infinities and NaN come out as the IEEE operation gives them
__device__ __forceinline__ double rcp_any(double x)
{
    const double s = (fabs(x) < 1.0) ? 0x1p300 : 0x1p-300, t = x * s;
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(t));
    const double e = fma(-t, y, 1.0);
    const double r = fma(y, fma(e, e, e), y);
    return ((fabs(x) > 0.0 && fabs(x) <= 1.7976931348623157e308) ? r : y) * s;
}
__device__ __forceinline__ double root_any(double x)
{
    const bool small = x < 1.0;
    const double r = sqrt_fast(x * (small ? 0x1p400 : 0x1p-400)) * (small ? 0x1p-200 : 0x1p200);
    return (x == 0.0 || x > 1.7976931348623157e308) ? x : r;
}

// a / x from ix = 1/x, both normal numbers: the quotient is corrected by its remainder (Markstein, IBM Journal
// of Research and Development 34, 1990), whose error is that of the division; an infinite quotient has no
// remainder
__device__ __forceinline__ double quotient_fast(double a, double x, double ix)
{
    const double q = a * ix;
    const double c = fma(fma(-q, x, a), ix, q);
    return (fabs(q) <= 1.7976931348623157e308) ? c : q;
}

// single precision: the hardware's own operations
__device__ __forceinline__ bool rcp_outside(float) { return false; }
__device__ __forceinline__ float rcp_fast(float x) { return 1.0f / x; }
__device__ __forceinline__ float rcp_fast_pos(float x) { return 1.0f / x; }
__device__ __forceinline__ float sqrt_fast(float x) { return sqrtf(x); }

// The arithmetic of a sweep.  FastOps: the short forms, NaN where they do not reach; GuardedOps: the same, each
// group of operations computed again with IeeeOps where the result is NaN; IeeeOps: the IEEE operations; WideOps: the
// scaled forms, for code in line that has no registers to spare for a call.
struct FastOps {
    template <typename FT> static __device__ __forceinline__ FT rcp(FT x) { return rcp_fast(x); }
    template <typename FT> static __device__ __forceinline__ FT root(FT x) { return sqrt_fast(x); }
};
struct GuardedOps {
    static __device__ __forceinline__ double rcp(double x) { return rcp_outside(x) ? divide_ieee(1.0, x) : rcp_fast(x); }
    static __device__ __forceinline__ float rcp(float x) { return 1.0f / x; }
};
struct IeeeOps {
    template <typename FT> static __device__ __forceinline__ FT rcp(FT x) { return (FT)1.0 / x; }
    static __device__ __forceinline__ double root(double x) { return sqrt(x); }
    static __device__ __forceinline__ float root(float x) { return sqrtf(x); }
};
struct WideOps {
    static __device__ __forceinline__ double rcp(double x) { return rcp_any(x); }
    static __device__ __forceinline__ float rcp(float x) { return 1.0f / x; }
    static __device__ __forceinline__ double root(double x) { return root_any(x); }
    static __device__ __forceinline__ float root(float x) { return sqrtf(x); }
};

#ifdef IB_STRICT_ARITH
template <typename OPS, typename FT> constexpr bool kPoison = false;
#else
// whether a NaN of the short forms has to be seen (FP32 arithmetic has no short forms)
template <typename OPS, typename FT>
constexpr bool kPoison = std::is_same<OPS, FastOps>::value && std::is_same<FT, double>::value;
#endif
// a density that sends its pencil to IeeeOps: NaN, infinite, or so large that a reciprocal may have been flushed
__device__ __forceinline__ bool density_suspect(double rho) { return !(fabs(rho) < 0x1p1000); }
// the same of a cell's primitives: a velocity v is NaN where 1 / rho is
__device__ __forceinline__ bool cell_suspect(double rho, double v) { return !(fma(v, 0.0, fabs(rho)) < 0x1p1000); }

}  // namespace ib
