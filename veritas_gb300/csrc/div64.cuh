// Quotients for the FP64 stencil kernels, in fewer instructions of the FP64 unit (which
// bounds them) than `/` takes, with its rounding.
//
// The reciprocal starts from the hardware's approximation (rcp.approx.ftz.f64) and is
// refined by one third-order step, y (1 + e + e^2) with e = 1 - b y, to within an ulp; the
// quotient q = a y, within 2.5 ulp, then takes Markstein's correction q + (a - q b) y by
// fused multiply-add (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990).  The value before the final rounding
// is within 2^-48 ulp of the quotient (the correction's relative error is 2^-51: its
// reciprocal's, and that of a remainder of 54 or 55 bits), so the result is the IEEE
// quotient unless the quotient lies that close to a midpoint of two doubles.  Such quotients
// exist (a divisor of 53 ones with the right numerators): near_midpoint finds everything
// within 2^-20 of one, `hard` is set, and the caller takes `/`.  About one quotient in
// 10^5 does at most.  The test is made on the integer and FP32 units, which these kernels leave idle.
// For b, a / b and the remainder normal and finite: callers keep their operands between
// 1e-250 and 1e200.
//
// The square root is refined from rsqrt.approx.ftz.f64 the same way, s (1 + e / 2 + 3 e^2 /
// 8) with e = 1 - s y, then corrected by its remainder (Markstein again): eight FP64
// instructions, the rounding of sqrt() by the same argument.
#pragma once
#include <cuda_runtime.h>

namespace vx {

// The 24 leading bits of a normal double's significand, truncated, in [1, 2), and its exponent.
__device__ __forceinline__ float lead_bits(double x) {
    return __uint_as_float((__funnelshift_l((unsigned)__double2loint(x), (unsigned)__double2hiint(x), 3) & 0x7fffffu) |
                           0x3f800000u);
}
__device__ __forceinline__ int exp_bits(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// Whether q + c with c = r y, |c| <= 2.5 ulp(q), may lie next to a midpoint of two doubles.
// Midpoints are odd multiples of ulp(q) / 2 away from q, of ulp(q) / 4 below a power of two,
// and 2 ulp(q) away one past a power of two: any multiple of a quarter counts, but 0 and 1
// (q + ulp(q), or the power of two that ends q's binade: a weight of 1 has it every second
// time).  u = |c| / (ulp(q) / 4) from the truncated significands, low by at most 2^-21.6 of itself.
__device__ __forceinline__ bool near_midpoint(double q, double r, double y) {
    const int k = max(exp_bits(r) + exp_bits(y) - exp_bits(q) - (1023 - 52 - 2), -64);  // r = 0: u = 0
    const float m = __fmul_rn(lead_bits(r), lead_bits(y));
    const float u = __int_as_float(__float_as_int(m) + (k << 23));
    const float n = __fsub_rn(__fadd_rn(u, 12582912.0f), 12582912.0f);  // nearest whole number
    return fabsf(__fsub_rn(u, n)) <= __fmul_rn(u, 0x1p-20f) && n != 0.0f && n != 4.0f;
}

// `/` and sqrt() for what the short forms hand on, by a call: inlined behind a branch, the
// compiler moves their first FP64 instructions in front of it.
static __device__ __noinline__ double div_call(double a, double b) { return a / b; }
static __device__ __noinline__ double sqrt_call(double x) { return sqrt(x); }

__device__ __forceinline__ double rcp_approx(double b) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
    return r;
}

// 1 / b to within an ulp.
__device__ __forceinline__ double rcp_ulp(double b) {
    const double y = rcp_approx(b);
    const double e = __fma_rn(-b, y, 1.0);
    return __fma_rn(y, __fma_rn(e, e, e), y);
}

// 1 / b, rounded as `1.0 / b` (or hard is set).
__device__ __forceinline__ double rcp_rn(double b, bool &hard) {
    const double y = rcp_ulp(b);
    const double e = __fma_rn(-b, y, 1.0);
    hard = hard || near_midpoint(y, e, y);
    return __fma_rn(y, e, y);
}

// a / b but for the cases above, from y = rcp_ulp(b), for callers that check it themselves.
__device__ __forceinline__ double div_short(double a, double b, double y) {
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-q, b, a), y, q);
}

// a / b, rounded as `a / b` (or hard is set), from y = rcp_ulp(b).
__device__ __forceinline__ double div_rn(double a, double b, double y, bool &hard) {
    const double q = __dmul_rn(a, y);
    const double r = __fma_rn(-q, b, a);
    hard = hard || near_midpoint(q, r, y);
    return __fma_rn(r, y, q);
}

// sqrt(x), rounded as sqrt() (or hard is set: also for x outside 2^-660 .. 2^660).
__device__ __forceinline__ double sqrt_rn(double x, bool &hard) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double s = __dmul_rn(x, y);
    const double e = __fma_rn(-s, y, 1.0);
    const double g = __dmul_rn(e, __fma_rn(e, 0.375, 0.5));
    const double r = __fma_rn(s, g, s);
    // half of the refined 1 / sqrt(x); halving y is an exponent decrement
    const double yh = __hiloint2double(__double2hiint(y) - 0x00100000, __double2loint(y));
    const double h = __fma_rn(yh, g, yh), d = __fma_rn(-r, r, x);
    hard = hard || (unsigned)__double2hiint(x) - 0x16b00000u >= 0x52800000u || near_midpoint(r, d, h);
    return __fma_rn(d, h, r);
}

}  // namespace vx
