// Quotients for the FP64 stencil kernels, in fewer instructions of the FP64 unit (which
// bounds them) than `/` takes, with its rounding.
//
// The reciprocal starts from the hardware's approximation (rcp.approx.ftz.f64) and is
// refined by one third-order step, y (1 + e + e^2) with e = 1 - b y, to within about an
// ulp; the quotient q = a y then takes Markstein's correction q + (a - q b) y, whose
// residual is exact by fused multiply-add (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990).  The value
// before the final rounding is within 2^-52 ulp of the quotient, so the result is the
// IEEE quotient unless that lies within 2^-52 ulp of a rounding boundary (4e9 random
// quotients and reciprocals: none).  For b, a / b and the residual normal and finite:
// callers keep their operands between 1e-200 and 1e200.
//
// The square root is refined from rsqrt.approx.ftz.f64 the same way, s (1 + e / 2 + 3 e^2 /
// 8) with e = 1 - s y, then corrected by its exact residual (Markstein again): eight FP64
// instructions, the rounding of sqrt() as above, for x normal, 1e-200 .. 1e200.
#pragma once
#include <cuda_runtime.h>

namespace vx {

__device__ __forceinline__ double rcp_approx(double b) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
    return r;
}

// 1 / b to within about an ulp.
__device__ __forceinline__ double rcp_ulp(double b) {
    const double y = rcp_approx(b);
    const double e = __fma_rn(-b, y, 1.0);
    return __fma_rn(y, __fma_rn(e, e, e), y);
}

// 1 / b, rounded as `1.0 / b`.
__device__ __forceinline__ double rcp_rn(double b) {
    const double y = rcp_ulp(b);
    return __fma_rn(y, __fma_rn(-b, y, 1.0), y);
}

// a / b, rounded as `a / b`, from y = rcp_ulp(b).
__device__ __forceinline__ double div_rn(double a, double b, double y) {
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-q, b, a), y, q);
}

// sqrt(x), rounded as sqrt().
__device__ __forceinline__ double sqrt_rn(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double s = __dmul_rn(x, y);
    const double e = __fma_rn(-s, y, 1.0);
    const double g = __dmul_rn(e, __fma_rn(e, 0.375, 0.5));
    const double r = __fma_rn(s, g, s);
    // half of the refined 1 / sqrt(x); halving y is an exponent decrement
    const double yh = __hiloint2double(__double2hiint(y) - 0x00100000, __double2loint(y));
    return __fma_rn(__fma_rn(-r, r, x), __fma_rn(yh, g, yh), r);
}

}  // namespace vx
