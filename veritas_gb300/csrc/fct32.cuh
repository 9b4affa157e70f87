// FP32 precision form of the per-patch FCT Runge-Kutta sub-steps
// (Rectangle::FCTTimeStep, Rectangle.cpp:1255-1623): the device bodies, one tile or strip
// per call, shared by the per-sub-step kernels (fct32.cu) and the persistent stage kernel
// (stage32.cu).  Both translation units are compiled with fused multiply-add allowed, and
// the bodies are the same source, so the two launch forms give the same bits.
//
// Same sub-steps and face windows as the FP64 kernels (gamma, faces and fluxes fused per
// direction; the cell-wise sub-steps with 128-bit accesses); the arithmetic differs where
// FP32 needs it:
//   * f is stored scaled by the run's fnorm (1 / the peak of the initial distribution),
//     so every plane stays far inside FP32 range; the FCT update is linear in f and its
//     limiter is scale free, so nothing else changes;
//   * momenta are carried as p / (m c) and A^2 as q^2 A^2 / (m c)^2, so the Lorentz
//     factor is sqrt(1 + p^2 + a^2) in dimensionless FP32;
//   * the velocity differences of the reference, c^2 m (gamma(p_{j+1}) - gamma(p_j)) / dp
//     and c^2 m (gamma(A_{i+1}) - gamma(A_i)) / dx, are evaluated in the rationalised
//     form (p_{j+1}^2 - p_j^2) / (gamma_{j+1} + gamma_j), which has no cancellation, so
//     the face velocities keep FP32 relative accuracy (the direct difference of two
//     Lorentz factors near 1 would lose four digits).
#pragma once
#include <cuda_runtime.h>

#include "amr.hpp"
#include "vx_kernels.hpp"

namespace vx {

using P32 = PatchT<float>;

// Quotients and square roots of the FP32 kernels use the hardware approximations
// (__fdividef: within 2 ulp for divisors below 2^126, which every divisor here is; and
// s * rsqrtf(s) for s >= 1); the precision form's stated error includes them.
__device__ __forceinline__ float sqrt_ge1(float s) { return s * rsqrtf(s); }

// WENO-type face value (Rectangle.cpp:980-1030) with the regulariser `mm`: the
// reference's 1e-10 carried into the scaled units of the smoothness indicators, floored
// at 1e-30 so that it stays a normal FP32 number (it only matters where f vanishes).
__device__ __forceinline__ float weno32(float f1, float f2, float f3, float f4, bool right, float mm) {
    const float c6 = 1.0f / 6.0f;
    const float c43 = 4.0f / 3.0f;
    float fL = c6 * (-f1 + 5.0f * f2 + 2.0f * f3);
    float fR = c6 * (2.0f * f2 + 5.0f * f3 - f4);
    float AL = f1 - 2.0f * f2 + f3;
    float BL = f3 - f1;
    float AR = f2 - 2.0f * f3 + f4;
    float BR = f4 - f2;
    float bL = c43 * (AL * AL) + 0.5f * AL * BL + 0.25f * (BL * BL);
    float bR = c43 * (AR * AR) - 0.5f * AR * BR + 0.25f * (BR * BR);
    // oL / (oL + oR) with o = 0.5 / (mm + b)^2, as a ratio that cannot underflow
    float rr = __fdividef(mm + bL, mm + bR);
    float wL = __fdividef(1.0f, 1.0f + rr * rr);  // rr^2 = inf gives wL = 0, its limit
    float wR = 1.0f - wL;
    float wL0 = wL * (0.75f + wL * (wL - 0.5f));
    float wR0 = wR * (0.75f + wR * (wR - 0.5f));
    float pick = right ? fmaxf(wL0, wR0) : fminf(wL0, wR0);
    float fwl = __fdividef(pick, wL0 + wR0);  // wL0 + wR0 >= 0.75
    return fwl * fL + (1.0f - fwl) * fR;
}

// Dimensionless momentum of p-face j, q^2 A^2 / (m c)^2 at the finest face under x-face
// i, and q times the rtb-average of E_x under coarse cell i (Rectangle::GetEfield,
// Rectangle.cpp:1055-1067), all from FP32 copies.
__device__ __forceinline__ float mom32(const P32 &P, int j) { return fmaf(P.dpnf, (float)(j + P.p_pos), P.pminf); }
__device__ __forceinline__ float asq32(const P32 &P, const RunFields &F, int i) {
    int x = P.rtb * (i + P.x_pos);
    x = x < 0 ? 0 : (x > F.n ? F.n : x);
    return P.a2nf * F.asq32[x];
}

__device__ __forceinline__ bool active32(const P32 &P, int i, int j) {
    return i >= P.xm && i < P.xp && j >= P.pm && j < P.pp;
}

// ---------------------------------------------------------------- streaming sub-steps
// The cell-wise sub-steps move whole planes with 128-bit accesses: a thread owns four
// consecutive p cells (j .. j+3) of one row, a tile is tile_i rows by 128 p cells.  Tiles
// start at j0 = -2 + 128 k, so j + 2 is a multiple of 4 and, with the pitch a multiple of
// 8 and every plane 16-byte aligned, each thread's four cells are one aligned float4.  The
// p neighbours past the four (j - 1, j + 4) are scalar loads, made only when a valid cell
// needs them (they are then inside the row).  Each body handles the thread (tx, row) of
// tile t: lane tx of the tile's 32 columns of four cells, row `row` of its tile_i rows.
#define VX_VTILE32                                        \
    const P32 &P = patches[t.patch];                      \
    const int i = t.i0 + row;                             \
    const int j = t.j0 + 4 * tx;                          \
    if (i > P.nx + 1 || j > P.np + 1) return;             \
    const int pit = P.pitch;                              \
    const int id = pidx(i, j, pit);

struct V4 {
    float v[4];
};
__device__ __forceinline__ V4 ld4(const float *p) {
    const float4 q = *reinterpret_cast<const float4 *>(p);
    return {{q.x, q.y, q.z, q.w}};
}
// Stores the elements e with lo <= j + e < hi (one 128-bit store when all four are).
__device__ __forceinline__ void st4(float *p, const V4 &x, int j, int lo, int hi) {
    if (j >= lo && j + 3 < hi) {
        *reinterpret_cast<float4 *>(p) = make_float4(x.v[0], x.v[1], x.v[2], x.v[3]);
        return;
    }
#pragma unroll
    for (int e = 0; e < 4; e++)
        if (j + e >= lo && j + e < hi) p[e] = x.v[e];
}

// RK flux combination (Rectangle.cpp:1396-1517): DS over the padded block.
__device__ __forceinline__ void ds_32(const P32 *patches, const TileRef t, int tx, int row, const float *params, int s) {
    VX_VTILE32
    const float *a = params + param_base(P.run, s);
    const float asum = a[6];
    V4 hx = ld4(P.FxH[0] + id), hp = ld4(P.FpH[0] + id);
#pragma unroll
    for (int e = 0; e < 4; e++) {
        hx.v[e] = a[0] * hx.v[e];
        hp.v[e] = a[0] * hp.v[e];
    }
    for (int k = 1; k <= s; k++) {
        if (s == 5 && k == 1) continue;  // b_1 = 0 (Rectangle.cpp:1494)
        const V4 gx = ld4(P.FxH[k] + id), gp = ld4(P.FpH[k] + id);
        const float ak = a[k];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            hx.v[e] += ak * gx.v[e];
            hp.v[e] += ak * gp.v[e];
        }
    }
    const V4 lx = ld4(P.FxL + id), lp = ld4(P.FpL + id);
    V4 dx, dp;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        dx.v[e] = hx.v[e] - __fmul_rn(asum, lx.v[e]);
        dp.v[e] = hp.v[e] - __fmul_rn(asum, lp.v[e]);
    }
    st4(P.FxDS + id, dx, j, -2, P.np + 2);
    st4(P.FpDS + id, dp, j, -2, P.np + 2);
}

// min(1, Q / P) for P > 0, else 0 (Q >= 0: a stencil extremum minus the centre value).
// Q >= P gives 1 without a quotient; otherwise the hardware reciprocal (within 2 ulp),
// except for a subnormal P, where it is not defined and IEEE division is used.
__device__ __forceinline__ float limiter_ratio(float Q, float P) {
    if (!(P > 0.0f)) return 0.0f;
    if (Q >= P) return 1.0f;
    return fminf(1.0f, P >= 1.17549435e-38f ? __fdividef(Q, P) : Q / P);
}

// ---- sub-steps that read neighbours in x and p
// One warp per row of a tile, four p cells per lane.  The p neighbours past a lane's four
// cells come from the next lanes; only the tile's two edge lanes load theirs (every lane
// loading its own cost as much in L1 as five more planes, and L1 bounded these kernels: 38.6
// M cells, C and update in one pass 335 us per stage against 137 us for its six planes).
// Walking several rows with one warp, each row of a plane loaded once, needs 72 to 86
// registers and was slower (limiter R 199 against 186 us, 27 against 16 us on 2.8 M cells).
#define VX_ROW32                                                  \
    const P32 &P = patches[t.patch];                              \
    const int i = t.i0 + row; /* warp-uniform */                  \
    const int j = t.j0 + 4 * lane, pit = P.pitch;                 \
    const bool col = j <= P.np + 1; /* four cells inside a row */ \
    const unsigned full = 0xffffffffu;

__device__ __forceinline__ V4 ld4_if(bool ok, const float *p) { return ok ? ld4(p) : V4{{0.0f, 0.0f, 0.0f, 0.0f}}; }
__device__ __forceinline__ V4 max4(const V4 &a, const V4 &b) {
    V4 r;
#pragma unroll
    for (int e = 0; e < 4; e++) r.v[e] = fmaxf(a.v[e], b.v[e]);
    return r;
}
__device__ __forceinline__ V4 min4(const V4 &a, const V4 &b) {
    V4 r;
#pragma unroll
    for (int e = 0; e < 4; e++) r.v[e] = fminf(a.v[e], b.v[e]);
    return r;
}

// Low-order solution (Rectangle.cpp:1518-1534) on the interior.  It needs only the step's
// stage-0 fluxes: after stage 0 it and the ghost cells it feeds are formed beside the
// stage's field work, off the chain from the solve to the update.
__device__ __forceinline__ void f2_32(const P32 *patches, const TileRef t, int lane, int row, const float *params, int s) {
    VX_ROW32
    if (i < 0 || i >= P.nx) return;
    const int id = pidx(i, j, pit);
    const float asum = params[param_base(P.run, s) + 6];
    const V4 lx = ld4_if(col, P.FxL + id), lp = ld4_if(col, P.FpL + id);
    const V4 f0 = ld4_if(col, P.f0 + id), lxn = ld4_if(col, P.FxL + id + pit);
    float lp4 = __shfl_down_sync(full, lp.v[0], 1);
    if (lane == 31) lp4 = (j + 3 < P.np) ? P.FpL[id + 4] : 0.0f;  // j + 4 <= np
    // the cell's own low-order fluxes are shared with its neighbours in the row: rounded once
    V4 lsx, lsp, f2;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        lsx.v[e] = __fmul_rn(asum, lx.v[e]);
        lsp.v[e] = __fmul_rn(asum, lp.v[e]);
    }
    const bool ai = i >= P.xm && i < P.xp, an = i + 1 >= P.xm && i + 1 < P.xp;
    const int lo = P.pm - j, hi = P.pp - j;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const bool aj = e >= lo && e < hi, ajn = e + 1 >= lo && e + 1 < hi;
        float v = f0.v[e];
        if (ai && aj) v += lsx.v[e];
        if (ai && aj) v += lsp.v[e];
        if (ai && ajn) v = e < 3 ? v - lsp.v[e + 1] : __fmaf_rn(-asum, lp4, v);
        if (an && aj) v = __fmaf_rn(-asum, lxn.v[e], v);
        f2.v[e] = v;
    }
    if (col) st4(P.f2 + id, f2, j, 0, P.np);
}

// Zalesak R+ and R- (Rectangle.cpp:1536-1582), cells i in [-1, nx], j in [-1, np].
__device__ __forceinline__ void limR32(const P32 *patches, const TileRef t, int lane, int row) {
    VX_ROW32
    if (i < -1 || i > P.nx) return;
    const int id = pidx(i, j, pit);
    const float *DX = P.FxDS, *DP = P.FpDS, *f0 = P.f0, *f2 = P.f2;
    const V4 dxi = ld4_if(col, DX + id), dxn = ld4_if(col, DX + id + pit), dpi = ld4_if(col, DP + id);
    // the cell beyond the tile's edge that lane 0 (j - 1) and lane 31 (j + 4) need
    const bool edge = (lane == 0 && j >= -1) || (lane == 31 && j + 3 <= P.np);
    const float edp = (edge && lane == 31) ? DP[id + 4] : 0.0f;
    float dp4 = __shfl_down_sync(full, dpi.v[0], 1);
    if (lane == 31) dp4 = edp;
    V4 Pp, Pm, rp, rm;
    bool some = false;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const float dpn = e < 3 ? dpi.v[e + 1] : dp4;
        Pp.v[e] = fmaxf(0.0f, dxi.v[e]) - fminf(0.0f, dxn.v[e]) + fmaxf(0.0f, dpi.v[e]) - fminf(0.0f, dpn);
        Pm.v[e] = fmaxf(0.0f, dxn.v[e]) - fminf(0.0f, dxi.v[e]) + fmaxf(0.0f, dpn) - fminf(0.0f, dpi.v[e]);
        some = some || Pp.v[e] > 0.0f || Pm.v[e] > 0.0f;
        rp.v[e] = rm.v[e] = 0.0f;
    }
    // nothing flows in or out of any of the warp's cells (empty phase space): R is 0
    if (__any_sync(full, some)) {
        const V4 a0 = ld4_if(col, f0 + id), c2 = ld4_if(col, f2 + id);
        const V4 u0 = ld4_if(col, f0 + id + pit), u2 = ld4_if(col, f2 + id + pit);
        const V4 d0 = ld4_if(col, f0 + id - pit), d2 = ld4_if(col, f2 + id - pit);
        float e0 = 0.0f, e2 = 0.0f;
        if (edge) {
            const int eoff = lane == 0 ? -1 : 4;
            e0 = f0[id + eoff];
            e2 = f2[id + eoff];
        }
        const V4 mxc = max4(a0, c2), mnc = min4(a0, c2);
        float lmx = __shfl_up_sync(full, mxc.v[3], 1), lmn = __shfl_up_sync(full, mnc.v[3], 1);
        float rmx = __shfl_down_sync(full, mxc.v[0], 1), rmn = __shfl_down_sync(full, mnc.v[0], 1);
        if (lane == 0) {
            lmx = fmaxf(e0, e2);
            lmn = fminf(e0, e2);
        }
        if (lane == 31) {
            rmx = fmaxf(e0, e2);
            rmn = fminf(e0, e2);
        }
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const float wMax = fmaxf(fmaxf(mxc.v[e], fmaxf(fmaxf(u0.v[e], u2.v[e]), fmaxf(d0.v[e], d2.v[e]))),
                                     fmaxf(e < 3 ? mxc.v[e + 1] : rmx, e > 0 ? mxc.v[e - 1] : lmx));
            const float wMin = fminf(fminf(mnc.v[e], fminf(fminf(u0.v[e], u2.v[e]), fminf(d0.v[e], d2.v[e]))),
                                     fminf(e < 3 ? mnc.v[e + 1] : rmn, e > 0 ? mnc.v[e - 1] : lmn));
            rp.v[e] = limiter_ratio(wMax - c2.v[e], Pp.v[e]);
            rm.v[e] = limiter_ratio(-wMin + c2.v[e], Pm.v[e]);
        }
    }
    if (!col) return;
    st4(P.Rp + id, rp, j, -1, P.np + 1);
    st4(P.Rm + id, rm, j, -1, P.np + 1);
}

// Face coefficients C (Rectangle.cpp:1583-1594) over the padded block: 1 outside
// i in [1, nx), j in [0, np).
__device__ __forceinline__ void limC32(const P32 *patches, const TileRef t, int tx, int row) {
    VX_VTILE32
    V4 cx{{1.0f, 1.0f, 1.0f, 1.0f}}, cp{{1.0f, 1.0f, 1.0f, 1.0f}};
    if (i >= 1 && i < P.nx && j + 3 >= 0 && j < P.np) {
        const float *Rp = P.Rp, *Rm = P.Rm;
        const V4 rpi = ld4(Rp + id), rmi = ld4(Rm + id), rpd = ld4(Rp + id - pit), rmd = ld4(Rm + id - pit);
        const V4 dx = ld4(P.FxDS + id), dp = ld4(P.FpDS + id);
        const bool lo_ok = j >= 0;
        const float rpl = lo_ok ? Rp[id - 1] : 0.0f, rml = lo_ok ? Rm[id - 1] : 0.0f;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            if (j + e < 0 || j + e >= P.np) continue;
            const float rpm = e > 0 ? rpi.v[e - 1] : rpl, rmm = e > 0 ? rmi.v[e - 1] : rml;
            cx.v[e] = dx.v[e] > 0.0f ? fminf(rpi.v[e], rmd.v[e]) : fminf(rpd.v[e], rmi.v[e]);
            cp.v[e] = dp.v[e] > 0.0f ? fminf(rpi.v[e], rmm) : fminf(rpm, rmi.v[e]);
        }
    }
    st4(P.Cx + id, cx, j, -2, P.np + 2);
    st4(P.Cp + id, cp, j, -2, P.np + 2);
}

// Antidiffusive update (Rectangle.cpp:1595-1612), interior cells.
__device__ __forceinline__ void update32(const P32 *patches, const TileRef t, int tx, int row) {
    VX_VTILE32
    if (i < 0 || i >= P.nx || j + 3 < 0 || j >= P.np) return;
    const V4 f2 = ld4(P.f2 + id), cx = ld4(P.Cx + id), dx = ld4(P.FxDS + id), cp = ld4(P.Cp + id),
             dp = ld4(P.FpDS + id);
    const V4 cxn = ld4(P.Cx + id + pit), dxn = ld4(P.FxDS + id + pit);
    const bool hi_ok = j + 3 < P.np;  // element 3 valid: j + 4 <= np
    const float cp4 = hi_ok ? P.Cp[id + 4] : 0.0f, dp4 = hi_ok ? P.FpDS[id + 4] : 0.0f;
    V4 out;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const int je = j + e;
        float v = f2.v[e];
        if (active32(P, i, je)) v += cx.v[e] * dx.v[e];
        if (active32(P, i, je)) v += cp.v[e] * dp.v[e];
        if (active32(P, i, je + 1)) v -= (e < 3 ? cp.v[e + 1] : cp4) * (e < 3 ? dp.v[e + 1] : dp4);
        if (active32(P, i + 1, je)) v -= cxn.v[e] * dxn.v[e];
        out.v[e] = v;
    }
    st4(P.f1 + id, out, j, 0, P.np);
}

// The two above in one pass, for the cells beside which no limiter exchange takes place: C
// of a cell's four faces is formed from R where it is used, so neither C plane is written
// or read (six planes moved instead of twelve).  Cells of the exchange (cmask) keep their C
// values for it and are updated after it (late_update32).  Where no flux is left to limit
// (empty phase space, smooth regions at rest) R is not read.
__device__ __forceinline__ void cupdate32(const P32 *patches, const TileRef t, int lane, int row) {
    VX_ROW32
    if (i > P.nx + 1) return;
    const int id = pidx(i, j, pit), np = P.np;
    unsigned mask = 0;
    if (P.cmask && col) mask = *reinterpret_cast<const unsigned *>(P.cmask + id);  // four cells' bytes
    const V4 one{{1.0f, 1.0f, 1.0f, 1.0f}};
    V4 cx = one, cp = one;  // C is 1 outside the interior
    // C of a face between two cells, from R of the upper (p, m) and the lower (l, lm) and its flux
    auto face = [](float flux, float p, float m, float l, float lm) {
        const bool up = flux > 0.0f;
        return fminf(up ? p : l, up ? lm : m);
    };
    if (i >= 0 && i < P.nx) {
        const float *Rp = P.Rp, *Rm = P.Rm, *DX = P.FxDS, *DP = P.FpDS;
        const bool in = i >= 1, inn = i + 1 < P.nx;  // rows i and i + 1 have faces between cells
        V4 dx = ld4_if(col, DX + id), dxn = ld4_if(col, DX + id + pit), dp = ld4_if(col, DP + id);
        const V4 f2 = ld4_if(col, P.f2 + id);
        float edp = 0.0f;
        if (lane == 31 && j + 3 < np) edp = DP[id + 4];
        // fluxes outside the face window count as zero
        const bool ai = i >= P.xm && i < P.xp, an = i + 1 >= P.xm && i + 1 < P.xp;
        const int lo = P.pm - j, hi = P.pp - j;
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const bool aj = e >= lo && e < hi;
            if (!(ai && aj)) dx.v[e] = 0.0f;
            if (!(an && aj)) dxn.v[e] = 0.0f;
            if (!(ai && aj)) dp.v[e] = 0.0f;
        }
        float dp4 = __shfl_down_sync(full, dp.v[0], 1);
        if (lane == 31) dp4 = (ai && 4 >= lo && 4 < hi) ? edp : 0.0f;
        bool some = mask != 0 || dp4 != 0.0f;
#pragma unroll
        for (int e = 0; e < 4; e++) some = some || dx.v[e] != 0.0f || dxn.v[e] != 0.0f || dp.v[e] != 0.0f;
        if (!__any_sync(full, some)) {
            if (col) st4(P.f1 + id, f2, j, 0, np);
            return;
        }
        const V4 rpc = ld4_if(col, Rp + id), rmc = ld4_if(col, Rm + id);
        const V4 rpd = ld4_if(col && in, Rp + id - pit), rmd = ld4_if(col && in, Rm + id - pit);
        const V4 rpn = ld4_if(col && inn, Rp + id + pit), rmn = ld4_if(col && inn, Rm + id + pit);
        // R beyond the tile's edge: lane 0 the cell j - 1, lane 31 the cell j + 4
        float ep = 0.0f, em = 0.0f;
        if ((lane == 0 && j >= 0) || (lane == 31 && j + 4 < np)) {
            const int eoff = lane == 0 ? -1 : 4;
            ep = Rp[id + eoff];
            em = Rm[id + eoff];
        }
        float lp = __shfl_up_sync(full, rpc.v[3], 1), lm = __shfl_up_sync(full, rmc.v[3], 1);
        if (lane == 0) {
            lp = ep;
            lm = em;
        }
        V4 cxn = one;
        if (in) {
#pragma unroll
            for (int e = 0; e < 4; e++) {
                cx.v[e] = face(dx.v[e], rpc.v[e], rmc.v[e], rpd.v[e], rmd.v[e]);
                const float c = face(dp.v[e], rpc.v[e], rmc.v[e], e > 0 ? rpc.v[e - 1] : lp, e > 0 ? rmc.v[e - 1] : lm);
                cp.v[e] = j + e < np ? c : 1.0f;
            }
        }
        if (inn) {
#pragma unroll
            for (int e = 0; e < 4; e++) cxn.v[e] = face(dxn.v[e], rpn.v[e], rmn.v[e], rpc.v[e], rmc.v[e]);
        }
        float cp4 = __shfl_down_sync(full, cp.v[0], 1);
        if (lane == 31) cp4 = (in && j + 4 < np) ? face(edp, ep, em, rpc.v[3], rmc.v[3]) : 1.0f;
        // a p face between two cells of the four: its product is rounded once and used twice
        V4 w, out;
#pragma unroll
        for (int e = 0; e < 4; e++) w.v[e] = __fmul_rn(cp.v[e], dp.v[e]);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            float v = __fmaf_rn(cx.v[e], dx.v[e], f2.v[e]);
            v = e > 0 ? v + w.v[e] : __fmaf_rn(cp.v[0], dp.v[0], v);
            v = e < 3 ? v - w.v[e + 1] : __fmaf_rn(-cp4, dp4, v);
            out.v[e] = __fmaf_rn(-cxn.v[e], dxn.v[e], v);
        }
        if (col) st4(P.f1 + id, out, j, 0, np);
    }
    if (mask) {
#pragma unroll
        for (int e = 0; e < 4; e++)
            if (((mask >> (8 * e)) & kCStore) && j + e < np + 2) {
                const bool out = j + e < 0 || j + e >= np;
                P.Cx[id + e] = out ? 1.0f : cx.v[e];
                P.Cp[id + e] = out ? 1.0f : cp.v[e];
            }
        // Row j = 0 at the lower momentum edge: its faces move nothing, but the exchange passes
        // their C on to finer faces that do, by the branch of the true flux.  Formed again for
        // these alone: with the fluxes kept as loaded for every C the step of 38.6 M cells took
        // 10.57 ms instead of 10.32.
        const int e = -j;
        if (e >= 0 && e < 4 && P.pm > 0 && ((mask >> (8 * e)) & kCStore) && i >= 1 && i < P.nx) {
            const int k = id + e;
            const float rp = P.Rp[k], rm = P.Rm[k];
            P.Cx[k] = face(P.FxDS[k], rp, rm, P.Rp[k - pit], P.Rm[k - pit]);
            P.Cp[k] = face(P.FpDS[k], rp, rm, P.Rp[k - 1], P.Rm[k - 1]);
        }
    }
}
#undef VX_ROW32

// The update of a cell beside an exchanged face, from the C planes; rounded as the passes
// above round the cell of its place in the four (e = (j + 2) mod 4).
__device__ __forceinline__ void late_update32(const P32 *patches, const CellOp *ops, int k) {
    const CellOp op = ops[k];
    const P32 &P = patches[op.patch];
    const int i = op.i, j = op.j, pit = P.pitch, id = pidx(i, j, pit), e = (j + 2) & 3;
    float v = P.f2[id];
    if (active32(P, i, j)) v = __fmaf_rn(P.Cx[id], P.FxDS[id], v);
    if (active32(P, i, j))
        v = e > 0 ? v + __fmul_rn(P.Cp[id], P.FpDS[id]) : __fmaf_rn(P.Cp[id], P.FpDS[id], v);
    if (active32(P, i, j + 1))
        v = e < 3 ? v - __fmul_rn(P.Cp[id + 1], P.FpDS[id + 1]) : __fmaf_rn(-P.Cp[id + 1], P.FpDS[id + 1], v);
    if (active32(P, i + 1, j)) v = __fmaf_rn(-P.Cx[id + pit], P.FxDS[id + pit], v);
    P.f1[id] = v;
}

// f0 = f1 over the padded block (Rectangle.cpp:1614-1621).
__device__ __forceinline__ void copy10_32(const P32 *patches, const TileRef t, int tx, int row) {
    VX_VTILE32
    st4(P.f0 + id, ld4(P.f1 + id), j, -2, P.np + 2);
}
#undef VX_VTILE32

// ---------------------------------------------------------------- fused face + flux
// One warp per strip tile: Lorentz factors, face velocities and WENO values are formed in
// registers and consumed there (neighbours through shuffles), so the FP32 form has no
// gamma or face planes at all.  The fluxes are the FP64 path's (k64_faces + k64_flux) in
// FP32; face values outside the reference's face ranges (x: i in [0, nx], j in [-1, np];
// p: i in [-1, nx], j in [0, np]) count as zero.  All 32 lanes of the warp call a strip
// body together (it shuffles across the warp).

// The descriptor and field-block values the p-direction body uses, read once into
// registers: its row loop stores to global memory, after which the compiler would
// otherwise reload every descriptor field it cannot prove unchanged (measured: the p
// kernel 32.5 -> 29.8 us on the 4096 x 512 case; the x kernel, with fewer fields in its
// loop, ran slower with the same change and keeps the descriptor reads).
struct FluxView {
    int nx, np, pit, rtb, x_pos, n;
    float dpnf, pminf, kpf, dpif, weno_eps, a2nf, qf, inv_rtb;
    const float *f, *asq, *efin;
    const uint8_t *ifp;
    float *FH, *FL;
    __device__ __forceinline__ FluxView(const P32 &P, const RunFields &F, int step, int use_f0) {
        nx = P.nx;
        np = P.np;
        pit = P.pitch;
        rtb = P.rtb;
        x_pos = P.x_pos;
        n = F.n;
        dpnf = P.dpnf;
        pminf = P.pminf;
        kpf = P.kpf;
        dpif = P.dpif;
        weno_eps = P.weno_eps;
        a2nf = P.a2nf;
        qf = P.qf;
        inv_rtb = 1.0f / (float)P.rtb;  // rtb is a power of two
        f = use_f0 ? P.f0 : P.f1;
        asq = F.asq32;
        efin = F.efin32;
        ifp = P.ifp;
        FH = P.FpH[step];
        FL = P.FpL;
    }
    // dimensionless momentum of p-face j (P.p_pos folded into the caller's j)
    __device__ __forceinline__ float mom(int jg) const { return fmaf(dpnf, (float)jg, pminf); }
    // q^2 A^2 / (m c)^2 at the finest face under x-face i
    __device__ __forceinline__ float asq_at(int i) const {
        int x = rtb * (i + x_pos);
        x = x < 0 ? 0 : (x > n ? n : x);
        return a2nf * asq[x];
    }
    // q times the rtb-average of E_x under coarse cell i (Rectangle::GetEfield,
    // Rectangle.cpp:1055-1067), periodic in x
    __device__ __forceinline__ float qe_at(int i) const {
        const int x = rtb * (i + x_pos);
        float t = 0.0f;
        for (int k = 0; k < rtb; k++) {
            int y = x + k;
            y = (y > -1) ? y : (y + n);
            y = (y < n) ? y : (y - n);
            t += efin[y];
        }
        return qf * (t * inv_rtb);
    }
};

// Empty phase space.  f underflows to 0 in FP32 thirteen thermal widths from its centre and
// is 0 outside the plasma, so on most of a base patch (83 % of the cells of the 0.5 keV
// wakefield case's, 60 % at 1 keV) every f a warp's row reads is 0, and with it the
// face values and the fluxes.  One vote per row finds that out, and the row's Lorentz
// factors, velocities and weights — the bulk of these issue-bound kernels — are not formed.

// x direction: a warp covers kXCols output columns j0 .. j0+29 (its 32 lanes hold the
// face values of j0-1 .. j0+30) over `strip` rows; rows are independent in x, and the
// four rows of f a face reads (i-2 .. i+1) slide down the strip, one new load per row.
__device__ __forceinline__ void xflux32(const P32 *patches, const TileRef t, int lane, const RunFields *fields,
                                       int step, int use_f0, int strip) {
    const P32 &P = patches[t.patch];
    const int pit = P.pitch;
    const float *f = use_f0 ? P.f0 : P.f1;
    const RunFields &F = fields[P.run];
    const int jj = t.j0 - 1 + lane;
    const bool col_ok = jj >= -1 && jj <= P.np;
    const float p0 = mom32(P, jj), p1 = mom32(P, jj + 1);
    const float w3 = 1.0f / 48.0f;
    const unsigned full = 0xffffffffu;
    // f at rows i-2, i-1, i of the first row (i0 >= 0, so all inside the padded block)
    float fa = 0.0f, fb = 0.0f, fc = 0.0f;
    if (col_ok) {
        const int id = pidx(t.i0, jj, pit);
        fa = f[id - 2 * pit];
        fb = f[id - pit];
        fc = f[id];
    }
    // q^2 A^2 / (m c)^2 of row i0 + k, formed once by lane k and taken by shuffle
    const float a_l = asq32(P, F, t.i0 + lane);
    // whether any lane's f of the four rows is not zero (bit k: row i - 2 + k)
    unsigned live = (__any_sync(full, fa != 0.0f) ? 1u : 0u) | (__any_sync(full, fb != 0.0f) ? 2u : 0u) |
                    (__any_sync(full, fc != 0.0f) ? 4u : 0u);
    for (int r = 0; r < strip; r++, live >>= 1) {
        const int i = t.i0 + r;
        if (i > P.nx) break;  // warp-uniform
        const int id = pidx(i, jj, pit);
        float am = 0.0f, fv = 0.0f, fd = 0.0f;
        if (col_ok) fd = f[id + pit];  // row i+1 <= nx+1
        if (__any_sync(full, fd != 0.0f)) live |= 8u;
        if (!live) {
            if (lane >= 1 && lane <= kXCols && col_ok && !(P.ifx && P.ifx[id])) {
                P.FxH[step][id] = 0.0f;
                if (step == 0) P.FxL[id] = 0.0f;
            }
            fa = fb;
            fb = fc;
            fc = fd;
            continue;
        }
        const float a = __shfl_sync(full, a_l, r);
        if (col_ok) {
            const float g0 = sqrt_ge1(1.0f + p0 * p0 + a), g1 = sqrt_ge1(1.0f + p1 * p1 + a);
            am = P.kxf * __fdividef(P.dpnf * (p1 + p0), g1 + g0);
            fv = weno32(fa, fb, fc, fd, am > 0.0f, P.weno_eps);
        }
        const float am1 = __shfl_up_sync(full, am, 1), ap1 = __shfl_down_sync(full, am, 1);
        const float fm1 = __shfl_up_sync(full, fv, 1), fp1 = __shfl_down_sync(full, fv, 1);
        if (lane >= 1 && lane <= kXCols && col_ok && !(P.ifx && P.ifx[id])) {
            P.FxH[step][id] = P.dxif * (fv * am + w3 * (fp1 - fm1) * (ap1 - am1));
            if (step == 0) P.FxL[id] = P.dxif * ((am > 0.0f ? fb : fc) * am);  // f[i-1] or f[i]
        }
        fa = fb;
        fb = fc;
        fc = fd;
    }
}

// p direction: a warp covers 32 columns over `strip` output rows, walking down with
// the face values of the previous and next rows in registers.  Face row i reads a^2 and
// gamma at x-faces i and i+1; the i+1 pair is the next row's i pair, so it is carried.
struct PRow {
    float a, g;  // q^2 A^2 / (m c)^2 and gamma at the row's lower x-face
};
__device__ __forceinline__ void pface32(const FluxView &V, int i, int j, bool col_ok, const PRow &lo,
                                        const PRow &hi, float qe, float &am, float &fv) {
    am = 0.0f;
    fv = 0.0f;
    const bool ok = col_ok && i >= -1 && i <= V.nx;
    float f1 = 0.0f, f2 = 0.0f, f3 = 0.0f, f4 = 0.0f;
    if (ok) {
        const float *f = V.f + pidx(i, j, V.pit);
        f1 = f[-2];
        f2 = f[-1];
        f3 = f[0];
        f4 = f[1];
        am = qe - V.kpf * __fdividef(hi.a - lo.a, hi.g + lo.g);
    }
    const bool live = __any_sync(0xffffffffu, f1 != 0.0f || f2 != 0.0f || f3 != 0.0f || f4 != 0.0f);
    if (live && ok) fv = weno32(f1, f2, f3, f4, am > 0.0f, V.weno_eps);
}

// The row quantities — q^2 A^2 / (m c)^2 at x-faces i0-1 .. i0+rows+1 and q<E_x> of rows
// i0-1 .. i0+rows — are the same for every lane: lane k forms those of row i0-1+k once
// (k <= strip + 2 < 32) and each row takes them by shuffle, instead of every lane
// forming every row's (their index clamping and the periodic E_x average were most of the
// kernel's integer instructions).
__device__ __forceinline__ void pflux32(const P32 *patches, const TileRef t, int lane, const RunFields *fields,
                                       int step, int use_f0, int strip) {
    const unsigned full = 0xffffffffu;
    const P32 &P = patches[t.patch];
    const FluxView V(P, fields[P.run], step, use_f0);
    const int j = t.j0 + lane;
    const bool col_ok = j >= 0 && j <= V.np;
    const float p = V.mom(j + P.p_pos);
    const float w3 = 1.0f / 48.0f;
    const int ir = t.i0 - 1 + lane;
    const float a_l = V.asq_at(ir);
    const float qe_l = (ir >= -1 && ir <= V.nx) ? V.qe_at(ir) : 0.0f;
    auto prow = [&](int i) {  // i - (i0 - 1) in 0 .. strip + 2
        const float a = __shfl_sync(full, a_l, i - (t.i0 - 1));
        return PRow{a, sqrt_ge1(1.0f + p * p + a)};
    };
    auto qe = [&](int i) { return __shfl_sync(full, qe_l, i - (t.i0 - 1)); };
    PRow r0 = prow(t.i0 - 1), r1 = prow(t.i0), r2 = prow(t.i0 + 1);
    float amA, fvA, amB, fvB;  // rows i-1 and i
    pface32(V, t.i0 - 1, j, col_ok, r0, r1, qe(t.i0 - 1), amA, fvA);
    pface32(V, t.i0, j, col_ok, r1, r2, qe(t.i0), amB, fvB);
    const int rows = min(strip, V.nx + 1 - t.i0);
    for (int r = 0; r < rows; r++) {
        const int i = t.i0 + r;
        const PRow r3 = prow(i + 2);
        float amC, fvC;  // row i+1
        pface32(V, i + 1, j, col_ok, r2, r3, qe(i + 1), amC, fvC);
        const int id = pidx(i, j, V.pit);
        if (col_ok && !(V.ifp && V.ifp[id])) {
            V.FH[id] = V.dpif * (fvB * amB + w3 * (fvC - fvA) * (amC - amA));
            if (step == 0) V.FL[id] = V.dpif * ((amB > 0.0f ? V.f[id - 1] : V.f[id]) * amB);
        }
        amA = amB;
        fvA = fvB;
        amB = amC;
        fvB = fvC;
        r2 = r3;
    }
}

}  // namespace vx
