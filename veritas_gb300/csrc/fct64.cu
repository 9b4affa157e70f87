// FP64 "plain" Vlasov kernels: the per-patch FCT Runge-Kutta sub-steps of
// Rectangle::FCTTimeStep (Rectangle.cpp:1255-1623).
//
// This translation unit is compiled with --fmad=false: every double-precision
// expression below is evaluated with the same operations, operands and order as the
// reference C++ (separate IEEE multiply and add, IEEE division and square root), so the
// results are bit-identical to a non-FMA x86-64 / -ffp-contract=off build of the
// reference for the same inputs.
//
// Work decomposition: every kernel walks a list of 32(p) x 8(x) tiles that covers the
// padded block of every patch of every run in the launch, so one launch per sub-step
// serves a single patch, all patches of an AMR hierarchy, or a batch of independent runs.
//
// Compiled a second time with -DVX_FP64_FAST and contraction allowed: the FP64 form that
// trades the reference's rounding for fewer FP64 instructions (fused multiply-add, the
// WENO weights as one quotient, and the two quotients of a face value through a
// Newton-refined hardware reciprocal instead of five IEEE divisions).  Its kernels
// live in namespace vx::fast64 and its launcher is launch_fct64_substep_fast.
#include <cuda_runtime.h>
#include "amr.hpp"
#include "div64.cuh"
#include "vx_kernels.hpp"

#ifdef VX_FP64_FAST
#define VX_FCT64_NS fast64
#define VX_FCT64_LAUNCH launch_fct64_substep_fast
#else
#define VX_FCT64_NS exact64
#define VX_FCT64_LAUNCH launch_fct64_substep
#endif

namespace vx {
namespace VX_FCT64_NS {

using P64 = PatchT<double>;

// The bits of a double.  Through an instruction the compiler does not look into: it turns
// integer tests for a sign, zero or NaN on __double_as_longlong back into FP64 compares, of
// which each takes the FP64 unit's time like any other FP64 instruction (2.83 M cells:
// limiter R 75 -> 58 us, limiter C and update 65 -> 54 us).
__device__ __forceinline__ long long as_bits(double x) {
    long long b;
    asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
    return b;
}

// The four cells around a face where the reconstruction needs no weights.
// 2: all are +0.0, and so is the face value (every term of weno_face is +0.0).
// 1: every |f| < 1e-14.  The smoothness indicators are then below 27 max|f|^2 < 2.7e-27,
//    less than half an ulp of the regulariser 1e-10 they are added to, so both sums equal
//    it, wL = wR = 0.5, the mapped weights are 0.375 and the face weight is 0.375 / 0.75 =
//    0.5 exactly, whichever way the wind blows.
// 0: anything else (NaN and infinities included).
// f is a phase-space density in SI units, 1e46 or so where there is plasma: a thermal
// distribution falls below 1e-14 at 17 thermal widths, so most of the momentum range of a
// base patch is on one of the two short paths (4096 x 512, 1 keV: 60 % of it).  A warp is
// 32 neighbouring p of one row, so whole warps take it: decided with integer compares
// on the high words, off the FP64 unit that bounds these kernels.
__device__ __forceinline__ int weno_void(double f1, double f2, double f3, double f4) {
    const unsigned h1 = (unsigned)__double2hiint(f1), h2 = (unsigned)__double2hiint(f2);
    const unsigned h3 = (unsigned)__double2hiint(f3), h4 = (unsigned)__double2hiint(f4);
    constexpr unsigned kTiny = 0x3d06849bu;  // high word of 1e-14 (1e-14 = 0x3d06849b86a12b9b)
    const unsigned m = max(max(h1 & 0x7fffffffu, h2 & 0x7fffffffu), max(h3 & 0x7fffffffu, h4 & 0x7fffffffu));
    if (m >= kTiny) return 0;
    const unsigned any = h1 | h2 | h3 | h4 | (unsigned)__double2loint(f1) | (unsigned)__double2loint(f2) |
                         (unsigned)__double2loint(f3) | (unsigned)__double2loint(f4);
    return any == 0 ? 2 : 1;
}

// a > b and a < b for the mapped weights (positive, or NaN): on the bit patterns, where
// any NaN makes the face value NaN whichever weight is picked.
__device__ __forceinline__ bool wgt(double a, double b) {
    return as_bits(a) > as_bits(b);
}

// x / 2 and 2 x on the bits, rounded as the products (subnormal results to nearest even); no
// FP64 instruction even for the ends of the range, which would be issued switched off.  With
// the products these save, x faces of 2.83 M cells 275 -> 237 us.
__device__ __forceinline__ double half_of(double x) {
    const long long b = as_bits(x), m = b & 0x7FFFFFFFFFFFFFFFLL;
    const unsigned e = (unsigned)(m >> 52);
    if (e - 2u < 0x7fdu) return __longlong_as_double(b - (1LL << 52));
    const long long h = m >> 1, r = h + (m & h & 1);  // a subnormal or least normal: its bits are its multiple
    return e == 0x7ff ? x : __longlong_as_double((b ^ m) | r);
}
__device__ __forceinline__ double twice(double x) {
    const long long b = as_bits(x), m = b & 0x7FFFFFFFFFFFFFFFLL;
    const unsigned e = (unsigned)(m >> 52);
    if (e - 1u < 0x7fdu) return __longlong_as_double(b + (1LL << 52));
    const long long r = e == 0 ? m << 1 : 0x7FF0000000000000LL;
    return e == 0x7ff ? x : __longlong_as_double((b ^ m) | r);
}

// WENO-type upwind face value (Rectangle.cpp:980-1030; identical values to
// Rectangle.cpp:943-977).  f1..f4 are the four cells left-to-right around the face.  The
// smoothness weights do not depend on the velocity, so both upwind choices come out of one
// evaluation (BOTH: out_right with the larger mapped weight, out_left with the smaller);
// otherwise out_right is the choice for `right`.
// In the FP64 form its quotients go through div64.cuh (the two of a weight pair share a
// reciprocal): one FP64 instruction of this kernel costs 4.5 us per RK stage on the 4096 x
// 512 two-level workload, an IEEE division about sixteen of them, a reciprocal three and
// each quotient three more.
template <bool BOTH>
__device__ __forceinline__ void weno_values(double f1, double f2, double f3, double f4, bool right,
                                            double &out_right, double &out_left) {
    const int none = weno_void(f1, f2, f3, f4);
    if (none == 2) {
        out_right = 0.0;
        out_left = 0.0;
        return;
    }
    const double c6 = 1.0 / 6;
    const double c43 = 4.0 / 3;
#ifdef VX_FP64_FAST  // fused into the sums
    const double d2 = 2 * f2, d3 = 2 * f3;
#else
    const double d2 = twice(f2), d3 = twice(f3);
#endif
    double fL = c6 * (-f1 + 5 * f2 + d3);
    double fR = c6 * (d2 + 5 * f3 - f4);
    if (none == 1) {
        out_right = out_left = half_of(fL) + half_of(fR);
        return;
    }
    double AL = f1 - d2 + f3;
    double BL = f3 - f1;
    double AR = f2 - d3 + f4;
    double BR = f4 - f2;
    // with t = B / 2, exact as is every product with a power of two, B^2 / 4 is t^2 and A B / 2
    // is A t in the same rounding
    const double tL = half_of(BL), tR = half_of(BR);
#ifdef VX_FP64_FAST
    // the indicator is A (c43 A +- t) + t^2
    const double bL = __fma_rn(tL, tL, AL * __fma_rn(c43, AL, tL));
    const double bR = __fma_rn(tR, tR, AR * __fma_rn(c43, AR, -tR));
#else
    double bL = c43 * (AL * AL) + AL * tL + tL * tL;
    double bR = c43 * (AR * AR) - AR * tR + tR * tR;
#endif
    const double mm = 1.0e-10;
    const double dL = mm + bL, dR = mm + bR;
    double wL, wR;
#ifdef VX_FP64_FAST
    // oL / (oL + oR) with o = 0.5 / (mm + b)^2 is dR^2 / (dL^2 + dR^2)
    wL = (dR * dR) * rcp_ulp(dL * dL + dR * dR);
    wR = 1.0 - wL;
    constexpr bool plain = true;
#else
    // within 1e-10 .. 1e95 every intermediate of the short quotients is a normal number
    const bool plain = (unsigned)__double2hiint(dL) < 0x53a00000u && (unsigned)__double2hiint(dR) < 0x53a00000u;
    bool hard = !plain;
    if (plain) {
        // twice the reference's o = 0.5 / d^2, whose quotients are the same
        const double oL = rcp_rn(dL * dL, hard), oR = rcp_rn(dR * dR, hard);
        const double so = oL + oR, y = rcp_ulp(so);
        wL = div_rn(oL, so, y, hard);
        wR = div_rn(oR, so, y, hard);
    }
    if (hard) {
        const double oL = div_call(0.5, dL * dL), oR = div_call(0.5, dR * dR);
        wL = div_call(oL, oL + oR);
        wR = div_call(oR, oL + oR);
    }
#endif
    double wL0 = wL * (0.75 + wL * (wL - 0.5));
    double wR0 = wR * (0.75 + wR * (wR - 0.5));
    const double pr = wgt(wL0, wR0) ? wL0 : wR0, pl = wgt(wR0, wL0) ? wL0 : wR0;
    const double sw = wL0 + wR0;
#ifdef VX_FP64_FAST
    const double inv = rcp_ulp(sw);
    auto quot = [&](double a) { return a * inv; };
#else
    // the mapped weights sum to 0.75 .. 1.25, each 0 .. 1.25: below 1e-250 (a weight of a
    // face between regions 1e60 apart) the residual would leave the normal range
    const double inv = rcp_ulp(sw);
    auto quot = [&](double a) {
        bool gen = !(plain && (unsigned)__double2hiint(a) >= 0x0c000000u);
        const double q = div_rn(a, sw, inv, gen);
        return gen ? div_call(a, sw) : q;
    };
#endif
    const double w = quot(BOTH || right ? pr : pl);
    out_right = w * fL + (1 - w) * fR;
    if (BOTH) {
        const double v = quot(pl);
        out_left = v * fL + (1 - v) * fR;
    }
}

__device__ __forceinline__ double weno_face(double f1, double f2, double f3, double f4, bool right) {
    double v = 0.0, unused = 0.0;
    weno_values<false>(f1, f2, f3, f4, right, v, unused);
    return v;
}

__device__ __forceinline__ double vmax(double a, double b) { return (a > b) ? a : b; }
__device__ __forceinline__ double vmin(double a, double b) { return (a < b) ? a : b; }
// vmax(0.0, x) and vmin(0.0, x) decided on the bit pattern with integer instructions (the
// FP64 unit is the limiter's bottleneck): x < 0 exactly when the sign bit is set and x is
// neither -0 nor NaN; x > 0 when the sign bit is clear and x is neither +0 nor NaN.
__device__ __forceinline__ double vmax0(double x) {
    const long long b = as_bits(x);
    const long long m = b & 0x7FFFFFFFFFFFFFFFLL;
    return (b < 0 && m != 0 && m <= 0x7FF0000000000000LL) ? 0.0 : x;
}
__device__ __forceinline__ double vmin0(double x) {
    const long long b = as_bits(x);
    return (b > 0 && b <= 0x7FF0000000000000LL) ? 0.0 : x;
}
// x > 0.0 (false for zeros and NaN) on the bit pattern
__device__ __forceinline__ bool gt0(double x) {
    const long long b = as_bits(x);
    return b > 0 && b <= 0x7FF0000000000000LL;
}


// Both zeros (bits, of doubles or of several or-ed together), and finite.
__device__ __forceinline__ unsigned long long bits(double x) {
    return (unsigned long long)as_bits(x);
}
__device__ __forceinline__ bool zeros(unsigned long long b) { return (b << 1) == 0; }
__device__ __forceinline__ bool finite_hi(double x) {
    return ((unsigned)__double2hiint(x) & 0x7ff00000u) != 0x7ff00000u;
}

// Rectangle::GetEfield (Rectangle.cpp:1055-1067): mean of the finest-grid E_x over the
// rtb finest cells under coarse cell i; finest indices are periodic (EMSolver.cpp:137-154).
__device__ __forceinline__ double patch_efield(const P64 &P, const RunFields &F, int i) {
    int x = P.rtb * (i + P.x_pos);
    double t = 0.0;
    for (int k = 0; k < P.rtb; k++) {
        int y = x + k;
        y = (y > -1) ? y : (y + F.n);
        y = (y < F.n) ? y : (y - F.n);
        t += F.efin[y];
    }
    return t * P.rtb_inv;
}

__device__ __forceinline__ double a_sq_face(const P64 &P, const RunFields &F, int i) {
    int x = P.rtb * (i + P.x_pos);
    x = x < 0 ? 0 : (x > F.n ? F.n : x);
    return F.asq[x];
}

#define VX_TILE_PROLOGUE                                  \
    const TileRef t = tiles[blockIdx.x];                  \
    const P64 &P = patches[t.patch];                      \
    const int i = t.i0 + (int)threadIdx.y;                \
    const int j = t.j0 + (int)threadIdx.x;                \
    if (i > P.nx + 1 || j > P.np + 1) return;             \
    const int pit = P.pitch;                              \
    const int id = pidx(i, j, pit);

// Lorentz factor at every (x-face i, p-face j) node, i in [-1,nx+1], j in [-1,np+1]:
// Rectangle::Gamma (Rectangle.hpp:181) with A^2 at the finest face under x-face i
// (EMSolver::GetASquared, EMSolver.cpp:133) and p_j = Momentum(j) (Rectangle.hpp:86).
// A thread walks the rows of its p: what p alone needs (a conversion, a product, a sum and a
// square, of fifteen FP64 operations) is formed once per tile (2.83 M cells 78 -> 65 us; 58
// are the FP64 units' time).
__global__ void k64_gamma(const P64 *patches, const TileRef *tiles, const RunFields *fields, int rows) {
    VX_PDL_WAIT();
    const TileRef t = tiles[blockIdx.x];
    const P64 &P = patches[t.patch];
    const int j = t.j0 + (int)threadIdx.x, i1 = min(t.i0 + rows, P.nx + 2);
    if (j > P.np + 1 || j < -1) return;
    const RunFields &F = fields[P.run];
    double p = P.pmin + P.dp * (double)(j + P.p_pos);
    for (int i = max(t.i0, -1); i < i1; i++) {
        double as = P.qq * a_sq_face(P, F, i);
        const double x = 1.0 + ((p * p) + as) * P.g2;
        bool hard = false;
        double g = sqrt_rn(x, hard);
        if (hard) g = sqrt_call(x);
        P.gam[pidx(i, j, P.pitch)] = g;
    }
}

// The stage's antidiffusive flux of a face from its high-order flux `v` of stage s, those of
// the earlier stages and its low-order flux (Rectangle.cpp:1396-1517).  RK coefficients
// arrive pre-multiplied by dt.  Formed where the flux is: v need not be read again.  Zero
// where they all are (vacuum), without the operations: FP64 instructions bound the flux
// kernels, and warps of vacuum are a third of a laser run's base patch (the same in the
// passes below).
// The stage is a template argument: with it at run time the products of later stages are
// issued too, switched off lane by lane (2.83 M cells: x fluxes 90 to 102 us at every stage,
// with it 70 us on stage 0 to 90 us on stage 5).  The earlier stages' sum needs nothing of
// this stage: of the p faces it is formed before the solve's E_x is known (p fluxes after
// the solve 114 -> 87 us on the late stages).
// history64: the earlier stages' part of the sum, S > 0.
template <int S>
__device__ __forceinline__ double history64_s(double *const *H, int id, const double *a) {
    double x[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    unsigned long long any = 0;
#pragma unroll
    for (int k = 0; k < S; k++)
        if (!(S == 5 && k == 1)) {  // b_1 = 0 (Rectangle.cpp:1494)
            x[k] = H[k][id];
            any |= bits(x[k]);
        }
    if (zeros(any)) return 0.0;
    double h = a[0] * x[0];
#pragma unroll
    for (int k = 1; k < S; k++)
        if (!(S == 5 && k == 1)) h = h + a[k] * x[k];
    return h;
}
__device__ __forceinline__ double history64(double *const *H, int id, const double *a, int s) {
    switch (s) {  // uniform
        case 0: return 0.0;
        case 1: return history64_s<1>(H, id, a);
        case 2: return history64_s<2>(H, id, a);
        case 3: return history64_s<3>(H, id, a);
        case 4: return history64_s<4>(H, id, a);
        default: return history64_s<5>(H, id, a);
    }
}
// The rest, from that sum.
__device__ __forceinline__ double stage_flux64(double hist, const double *a, int s, double v, double low) {
    if (zeros(bits(hist) | bits(v) | bits(low))) return 0.0;
    return (s == 0 ? a[0] * v : hist + a[s] * v) - a[6] * low;
}

// Face velocities and reconstructed face values (Rectangle.cpp:1278-1312).
__global__ void k64_faces(const P64 *patches, const TileRef *tiles, const RunFields *fields, const double *params,
                          int step, int use_f0, int part) {
    VX_PDL_WAIT();
    VX_TILE_PROLOGUE
    const double *f = use_f0 ? P.f0 : P.f1;
    const double *g = P.gam;
    if ((part & 1) && i >= 0 && i <= P.nx && j >= -1 && j <= P.np) {
        double am = P.kx * (g[pidx(i, j + 1, pit)] - g[id]);
        P.ex[id] = am;
        P.fx[id] = weno_face(f[pidx(i - 2, j, pit)], f[pidx(i - 1, j, pit)], f[id], f[pidx(i + 1, j, pit)], gt0(am));
    }
    if ((part & 2) && i >= -1 && i <= P.nx && j >= 0 && j <= P.np) {
        const RunFields &F = fields[P.run];
        double Em = P.q * patch_efield(P, F, i);
        double am = Em - P.kp * (g[pidx(i + 1, j, pit)] - g[id]);
        P.ep[id] = am;
        P.fp[id] = weno_face(f[pidx(i, j - 2, pit)], f[pidx(i, j - 1, pit)], f[id], f[pidx(i, j + 1, pit)], gt0(am));
    }
    // The part of the p faces that does not need E_x, formed beside the Poisson solve: both
    // upwind candidates (fp and, as scratch, Rp), the velocity's second term (Rm; the limiter
    // rewrites both later in the stage) and, in FpDS, the earlier stages' part of the stage
    // flux.  k64_pflux_pick goes on from these.
    if ((part & 4) && i >= -1 && i <= P.nx && j >= 0 && j <= P.np) {
        double vr, vl;
        weno_values<true>(f[pidx(i, j - 2, pit)], f[pidx(i, j - 1, pit)], f[id], f[pidx(i, j + 1, pit)], true, vr, vl);
        P.fp[id] = vr;
        P.Rp[id] = vl;
        P.Rm[id] = P.kp * (g[pidx(i + 1, j, pit)] - g[id]);
        if (step > 0) P.FpDS[id] = history64(P.FpH, id, params + param_base(P.run, step), step);
    }
}

// High-order flux of a face from the velocities and values there and at its neighbours on
// either side.  Zero without the operations where the values are (and the velocities finite).
__device__ __forceinline__ double high_flux(double d_inv, double fm1, double fm, double fp1, double am1, double am,
                                            double ap1) {
    if (zeros(bits(fm1) | bits(fm) | bits(fp1)) && finite_hi(am1) && finite_hi(am) && finite_hi(ap1)) return 0.0;
    const double w3 = 1 / 48.0;
    return d_inv * (fm * am + w3 * (fp1 - fm1) * (ap1 - am1));
}
// Donor-cell flux; zero as above.
__device__ __forceinline__ double low_flux(double d_inv, double f, double am) {
    return zeros(bits(f)) && finite_hi(am) ? 0.0 : d_inv * (f * am);
}

// High-order fluxes for stage `step`, on stage 0 the donor-cell low-order fluxes
// (Rectangle.cpp:1313-1394), and the antidiffusive stage fluxes.  Coarse faces on a
// coarse/fine interface are skipped here and written by the interface kernel.
__global__ void k64_flux(const P64 *patches, const TileRef *tiles, const double *params, int step, int use_f0,
                         int part) {
    VX_PDL_WAIT();
    VX_TILE_PROLOGUE
    const double *f = use_f0 ? P.f0 : P.f1;
    const double *a = params + param_base(P.run, step);
    if ((part & 1) && i >= 0 && i <= P.nx && j >= -1 && j <= P.np && !(P.ifx && P.ifx[id])) {
        double am = P.ex[id], ap1 = P.ex[id + 1], am1 = P.ex[id - 1];
        double fm = P.fx[id], fp1 = P.fx[id + 1], fm1 = P.fx[id - 1];
        const double v = high_flux(P.dx_inv, fm1, fm, fp1, am1, am, ap1);
        P.FxH[step][id] = v;
        double low;
        if (step == 0) {
            low = low_flux(P.dx_inv, gt0(am) ? f[id - pit] : f[id], am);
            P.FxL[id] = low;
        } else {
            low = P.FxL[id];
        }
        P.FxDS[id] = stage_flux64(history64(P.FxH, id, a, step), a, step, v, low);
    }
    if ((part & 2) && i >= -1 && i <= P.nx && j >= 0 && j <= P.np && !(P.ifp && P.ifp[id])) {
        double am = P.ep[id], ap1 = P.ep[id + pit], am1 = P.ep[id - pit];
        double fm = P.fp[id], fp1 = P.fp[id + pit], fm1 = P.fp[id - pit];
        const double v = high_flux(P.dp_inv, fm1, fm, fp1, am1, am, ap1);
        P.FpH[step][id] = v;
        double low;
        if (step == 0) {
            low = low_flux(P.dp_inv, gt0(am) ? f[id - 1] : f[id], am);
            P.FpL[id] = low;
        } else {
            low = P.FpL[id];
        }
        P.FpDS[id] = stage_flux64(history64(P.FpH, id, a, step), a, step, v, low);
    }
}

// The p fluxes once E_x is known, from what k64_faces (part 4) left: velocity E - Rm, face
// value fp or Rp by its sign, for the face's row and the rows on either side.  q E_x is a
// row's value: formed once per block and row.  One pass in place of a face pass and a flux
// pass, and nothing of it waits for the solve but the velocity's difference: it is on the
// step's critical path (the solve is not).  The velocity itself is kept on stage 0, where
// the interface kernel reads it.
__global__ void k64_pflux_pick(const P64 *patches, const TileRef *tiles, const RunFields *fields, const double *params,
                               int step, int use_f0) {
    VX_PDL_WAIT();
    __shared__ double s_e[66];  // q E_x of the tile's rows i0 - 1 .. i0 + rows
    const TileRef t = tiles[blockIdx.x];
    const P64 &P = patches[t.patch];
    {
        const int r = (int)(threadIdx.y * blockDim.x + threadIdx.x), i = t.i0 - 1 + r;
        if (r < (int)blockDim.y + 2)
            s_e[r] = (i >= -1 && i <= P.nx) ? P.q * patch_efield(P, fields[P.run], i) : 0.0;
    }
    __syncthreads();
    const int i = t.i0 + (int)threadIdx.y, j = t.j0 + (int)threadIdx.x;
    if (i < -1 || i > P.nx || j < 0 || j > P.np) return;
    const int pit = P.pitch, id = pidx(i, j, pit);
    const double *f = use_f0 ? P.f0 : P.f1;
    const double *a = params + param_base(P.run, step);
    double am[3], fv[3];  // rows i-1, i, i+1; zero past the face range, as the planes are there
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const int k = i - 1 + d, kd = id + (d - 1) * pit;
        am[d] = fv[d] = 0.0;
        if (k >= -1 && k <= P.nx) {
            am[d] = s_e[(int)threadIdx.y + d] - P.Rm[kd];
            fv[d] = gt0(am[d]) ? P.fp[kd] : P.Rp[kd];
        }
    }
    if (step == 0) P.ep[id] = am[1];
    if (P.ifp && P.ifp[id]) return;
    const double v = high_flux(P.dp_inv, fv[0], fv[1], fv[2], am[0], am[1], am[2]);
    P.FpH[step][id] = v;
    double low;
    if (step == 0) {
        low = low_flux(P.dp_inv, gt0(am[1]) ? f[id - 1] : f[id], am[1]);
        P.FpL[id] = low;
    } else {
        low = P.FpL[id];
    }
    P.FpDS[id] = stage_flux64(step > 0 ? P.FpDS[id] : 0.0, a, step, v, low);
}

__device__ __forceinline__ bool active_face(const P64 &P, int i, int j) {
    return i >= P.xm && i < P.xp && j >= P.pm && j < P.pp;
}

// The low-order solution f2 = f0 + div(LS) on the interior in the reference's accumulation
// order (Rectangle.cpp:1518-1534).  It needs only the step's stage-0 fluxes, so after
// stage 0 it is formed beside the stage's field work.
__global__ void k64_f2(const P64 *patches, const TileRef *tiles, const double *params, int s) {
    VX_PDL_WAIT();
    VX_TILE_PROLOGUE
    if (i < 0 || i >= P.nx || j < 0 || j >= P.np) return;
    const double asum = params[param_base(P.run, s) + 6];
    const double lx = P.FxL[id], lp = P.FpL[id], lpn = P.FpL[id + 1], lxn = P.FxL[id + pit];
    double v = P.f0[id];
    if (!zeros(bits(lx) | bits(lp) | bits(lpn) | bits(lxn))) {
        double lsx = asum * lx;
        double lsp = asum * lp;
        if (active_face(P, i, j)) v += lsx;
        if (active_face(P, i, j)) v += lsp;
        if (active_face(P, i, j + 1)) v -= asum * lpn;
        if (active_face(P, i + 1, j)) v -= asum * lxn;
    }
    P.f2[id] = v;
}

// vmin for limiter values on the bit patterns: b where either is NaN, else the lesser (-0
// before +0; the limiter's values are not negative).
__device__ __forceinline__ double vmin_r(double a, double b) {
    constexpr long long kAbs = 0x7FFFFFFFFFFFFFFFLL, kInf = 0x7FF0000000000000LL;
    const long long p = as_bits(a), q = as_bits(b);
    const bool nan = (p & kAbs) > kInf || (q & kAbs) > kInf;
    return !nan && (p ^ ((p >> 63) & kAbs)) < (q ^ ((q >> 63) & kAbs)) ? a : b;
}

// Zalesak R+/R- on i in [-1,nx], j in [-1,np] (Rectangle.cpp:1536-1579).
__global__ void k64_limR(const P64 *patches, const TileRef *tiles) {
    VX_PDL_WAIT();
    VX_TILE_PROLOGUE
    if (i < -1 || i > P.nx || j < -1 || j > P.np) return;
    const double *DX = P.FxDS, *DP = P.FpDS, *f0 = P.f0, *f2 = P.f2;
    double dxi = DX[id], dxn = DX[id + pit], dpi = DP[id], dpn = DP[id + 1];
    double Pp = 0.0, Pm = 0.0;
    if (!zeros(bits(dxi) | bits(dxn) | bits(dpi) | bits(dpn))) {
        Pp = vmax0(dxi) - vmin0(dxn) + vmax0(dpi) - vmin0(dpn);
        Pm = vmax0(dxn) - vmin0(dxi) + vmax0(dpn) - vmin0(dpi);
    }
    const bool up = gt0(Pp), um = gt0(Pm);
    double rp = 0.0, rm = 0.0;
    if (up || um) {  // no antidiffusive flux touches the cell otherwise: both are 0
        const double v[10] = {f0[id],       f2[id],       f0[id + pit], f2[id + pit], f0[id - pit],
                              f2[id - pit], f0[id + 1],   f2[id + 1],   f0[id - 1],   f2[id - 1]};
        const double c2 = v[1];
        // f is not negative (the limiter's purpose), and non-negative doubles order as
        // their bit patterns: the eighteen compares of the extrema leave the FP64 unit
        // (one FP64 instruction of this kernel is 4.5 us per stage on the 4096 x 512
        // workload).  A negative value, -0 or NaN among the ten takes the general path.
        long long hi = 0, lo = 0x7FF0000000000000LL;
        int sign = 0;
#pragma unroll
        for (int k = 0; k < 10; k++) {
            const long long b = as_bits(v[k]);
            sign |= __double2hiint(v[k]);
            hi = b > hi ? b : hi;
            lo = b < lo ? b : lo;
        }
        double wMax, wMin;
        if (sign >= 0 && hi <= 0x7FF0000000000000LL) {
            wMax = __longlong_as_double(hi);
            wMin = __longlong_as_double(lo);
        } else {
            wMax = vmax(vmax(v[0], v[1]), vmax(vmax(v[2], v[3]), vmax(vmax(v[4], v[5]), vmax(vmax(v[6], v[7]), vmax(v[8], v[9])))));
            wMin = vmin(vmin(v[0], v[1]), vmin(vmin(v[2], v[3]), vmin(vmin(v[4], v[5]), vmin(vmin(v[6], v[7]), vmin(v[8], v[9])))));
        }
        const double Qm = -wMin + c2;
        const double Qp = wMax - c2;
        // min(1, Q/P) is 1 whenever Q >= P and P is finite: the quotient (Q infinite
        // included) is then >= 1 however it rounds; P > 0, so Q >= P is a compare of the
        // bit patterns once Q's sign is known.  Every other case, NaN and infinite P
        // among them, takes the division as written.  Most cells of a smooth solution
        // skip the division; within 2^-600 .. 2^600 it takes the short form.
        auto ratio = [](double Q, double P) {
            const long long q = as_bits(Q), p = as_bits(P);
            if (q >= p && p < 0x7FF0000000000000LL && q <= 0x7FF0000000000000LL) return 1.0;
            const unsigned hq = (unsigned)(q >> 32) - 0x1a700000u, hp = (unsigned)(p >> 32) - 0x1a700000u;
            bool gen = !(hq < 0x4b000000u && hp < 0x4b000000u);
            double v = 0.0;
            if (!gen) v = div_rn(Q, P, rcp_ulp(P), gen);
            if (gen) v = div_call(Q, P);
            return vmin_r(1.0, v);
        };
        if (up) rp = ratio(Qp, Pp);
        if (um) rm = ratio(Qm, Pm);
    }
    P.Rp[id] = rp;
    P.Rm[id] = rm;
}

// Limiter coefficients on interior faces, 1 elsewhere (Rectangle.cpp:1581-1594).
__global__ void k64_limC(const P64 *patches, const TileRef *tiles) {
    VX_PDL_WAIT();
    VX_TILE_PROLOGUE
    if (i < -2 || j < -2) return;
    double cx = 1.0, cp = 1.0;
    if (i >= 1 && i < P.nx && j >= 0 && j < P.np) {
        const double *Rp = P.Rp, *Rm = P.Rm;
        const bool ux = gt0(P.FxDS[id]), up = gt0(P.FpDS[id]);
        cx = vmin_r(Rp[ux ? id : id - pit], Rm[ux ? id - pit : id]);
        cp = vmin_r(Rp[up ? id : id - 1], Rm[up ? id - 1 : id]);
    }
    P.Cx[id] = cx;
    P.Cp[id] = cp;
}

// Antidiffusive update f1 = f2 + div(C * DS) (Rectangle.cpp:1595-1612).
__global__ void k64_update(const P64 *patches, const TileRef *tiles) {
    VX_PDL_WAIT();
    VX_TILE_PROLOGUE
    if (i < 0 || i >= P.nx || j < 0 || j >= P.np) return;
    double v = P.f2[id];
    if (active_face(P, i, j)) v += P.Cx[id] * P.FxDS[id];
    if (active_face(P, i, j)) v += P.Cp[id] * P.FpDS[id];
    if (active_face(P, i, j + 1)) v -= P.Cp[id + 1] * P.FpDS[id + 1];
    if (active_face(P, i + 1, j)) v -= P.Cx[id + pit] * P.FxDS[id + pit];
    P.f1[id] = v;
}

// The two above in one pass, for the cells beside which no limiter exchange takes place: C
// of a cell's four faces is formed from R where it is used, so neither C plane is written
// or read.  Cells of the exchange (cmask) keep their C values for it and are updated
// after it (late_update).
__global__ void k64_cupdate(const P64 *patches, const TileRef *tiles) {
    VX_PDL_WAIT();
    VX_TILE_PROLOGUE
    if (i < -2 || j < -2) return;
    const uint8_t mask = P.cmask ? P.cmask[id] : 0;
    const bool cell = i >= 0 && i < P.nx && j >= 0 && j < P.np;
    if (!cell && !(mask & kCStore)) return;
    const double *Rp = P.Rp, *Rm = P.Rm, *DX = P.FxDS, *DP = P.FpDS;
    auto face_x = [&](int a, int k, double d) {  // C of x face (a, j), k its index
        if (!(a >= 1 && a < P.nx)) return 1.0;
        const bool up = gt0(d);
        return vmin_r(Rp[up ? k : k - pit], Rm[up ? k - pit : k]);
    };
    auto face_p = [&](int b, int k, double d) {  // C of p face (i, b)
        if (!(i >= 1 && i < P.nx && b < P.np)) return 1.0;
        const bool up = gt0(d);
        return vmin_r(Rp[up ? k : k - 1], Rm[up ? k - 1 : k]);
    };
    double cx = 1.0, cp = 1.0;
    if (cell) {
        const double dx = DX[id], dp = DP[id], dpn = DP[id + 1], dxn = DX[id + pit];
        double v = P.f2[id];
        // nothing to limit (vacuum): R is not read either
        if (mask || !zeros(bits(dx) | bits(dp) | bits(dpn) | bits(dxn))) {
            cx = face_x(i, id, dx);
            cp = face_p(j, id, dp);
            if (active_face(P, i, j)) v += cx * dx;
            if (active_face(P, i, j)) v += cp * dp;
            if (active_face(P, i, j + 1)) v -= face_p(j + 1, id + 1, dpn) * dpn;
            if (active_face(P, i + 1, j)) v -= face_x(i + 1, id + pit, dxn) * dxn;
        }
        P.f1[id] = v;
    }
    if (mask & kCStore) {
        P.Cx[id] = cx;
        P.Cp[id] = cp;
    }
}

// The update of the cells beside an exchanged face, from the C planes.
__global__ void k64_late(const P64 *patches, const CellOp *ops, int n) {
    VX_PDL_WAIT();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const CellOp op = ops[k];
    const P64 &P = patches[op.patch];
    const int i = op.i, j = op.j, pit = P.pitch, id = pidx(i, j, pit);
    double v = P.f2[id];
    if (active_face(P, i, j)) v += P.Cx[id] * P.FxDS[id];
    if (active_face(P, i, j)) v += P.Cp[id] * P.FpDS[id];
    if (active_face(P, i, j + 1)) v -= P.Cp[id + 1] * P.FpDS[id + 1];
    if (active_face(P, i + 1, j)) v -= P.Cx[id + pit] * P.FxDS[id + pit];
    P.f1[id] = v;
}

// Last stage: f0 = f1 over the padded block (Rectangle.cpp:1614-1621).
__global__ void k64_copy10(const P64 *patches, const TileRef *tiles) {
    VX_PDL_WAIT();
    VX_TILE_PROLOGUE
    if (i < -2 || j < -2) return;
    P.f0[id] = P.f1[id];
}

}  // namespace VX_FCT64_NS

// --------------------------------------------------------------------------------
void VX_FCT64_LAUNCH(const FctLaunch &L, int sub) {
    using namespace VX_FCT64_NS;
    dim3 blk(L.tile_j ? L.tile_j : 32, L.tile_i ? L.tile_i : 8);
    const P64 *pp = (const P64 *)L.patches;
    if (L.ntiles == 0) return;
    switch (sub) {
        case kSubGamma:
            vx_launch(k64_gamma, L.ntiles, blk.x, 0, L.stream, pp, L.tiles, L.fields, (int)blk.y);
            break;
        case kSubFaces:
            vx_launch(k64_faces, L.ntiles, blk, 0, L.stream, pp, L.tiles, L.fields, L.params, L.step, L.use_f0,
                      L.part ? L.part : 3);
            break;
        case kSubFlux:
            if (L.part == 8)
                vx_launch(k64_pflux_pick, L.ntiles, blk, 0, L.stream, pp, L.tiles, L.fields, L.params, L.step, L.use_f0);
            else
                vx_launch(k64_flux, L.ntiles, blk, 0, L.stream, pp, L.tiles, L.params, L.step, L.use_f0,
                          L.part ? L.part : 3);
            break;
        case kSubF2:
            vx_launch(k64_f2, L.ntiles, blk, 0, L.stream, pp, L.tiles, L.params, L.step);
            break;
        case kSubLimR:
            vx_launch(k64_limR, L.ntiles, blk, 0, L.stream, pp, L.tiles);
            break;
        case kSubLimC:
            vx_launch(k64_limC, L.ntiles, blk, 0, L.stream, pp, L.tiles);
            break;
        case kSubUpdate:
            vx_launch(k64_update, L.ntiles, blk, 0, L.stream, pp, L.tiles);
            break;
        case kSubCUpdate:
            vx_launch(k64_cupdate, L.ntiles, blk, 0, L.stream, pp, L.tiles);
            break;
        case kSubLate:
            if (L.nlate) vx_launch(k64_late, (L.nlate + 127) / 128, 128, 0, L.stream, pp, L.late, L.nlate);
            break;
        case kSubCopy10:
            vx_launch(k64_copy10, L.ntiles, blk, 0, L.stream, pp, L.tiles);
            break;
    }
}

}  // namespace vx
