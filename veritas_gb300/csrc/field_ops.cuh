// Device bodies of the field-side stage work (one cell per call): the assembly of rho and
// J and the Maxwell RK stage.  Shared by fields64.cu (FP64 runs, compiled without
// contraction, so every expression keeps the reference's operation order) and stage32.cu
// (runs of the FP32 precision form, whose fields are FP64 too, compiled with contraction).
#pragma once
#include <cuda_runtime.h>

#include "div64.cuh"
#include "vx_kernels.hpp"

namespace vx {

// ---------------------------------------------------------------- assembly
// Level::CollectRhoAndJ + EMFieldSolver::AssembleRhoAndJ (Level.cpp:19-62,
// EMSolver.cpp:104-122): per level, chargeL[x] = 0 + (patch values in patch order);
// charges_s[x] = 0 + level sums finest->coarsest; J sums species then levels;
// charge[x] = 0 + species sums.  CG: the column sums are read through L2 only (the
// pipelined solve reads them while the moment blocks that write them still run; see
// k64_moments_poisson).
template <bool CG = false>
__device__ __forceinline__ void assemble_cell(const AsmLaunch &A, int run, int x) {
    const int n = A.run_n[run];
    if (x >= n) return;
    const int ns = A.run_ns[run], nl = A.run_nl[run];
    const int *lp = A.lvl_ptr + A.lvl_off[run];
    const PatchT<double> *patches = (const PatchT<double> *)A.patches;
    double J = 0.0, charge = 0.0;
    for (int s = 0; s < ns; s++) {
        double cs = 0.0;
        for (int l = 0; l < nl; l++) {
            double lc = 0.0, lj = 0.0;
            for (int e = lp[s * nl + l]; e < lp[s * nl + l + 1]; e++) {
                const PatchT<double> &P = patches[A.lvl_patch[e]];
                int c = x - P.x_pos * P.rtb;
                if (c >= 0 && c < P.nx * P.rtb) {
                    if (A.pairs) {  // FP32 moments: (hi, lo) of the column sum, then its scale
                        const float2 qc = reinterpret_cast<const float2 *>(P.chargeR)[c];
                        const float2 qj = reinterpret_cast<const float2 *>(P.currentR)[c];
                        lc += ((double)qc.x + (double)qc.y) * P.msc_rho;
                        lj += ((double)qj.x + (double)qj.y) * P.msc_j;
                    } else if (CG) {
                        lc += __ldcg(P.chargeR + c);
                        lj += __ldcg(P.currentR + c);
                    } else {
                        lc += P.chargeR[c];
                        lj += P.currentR[c];
                    }
                }
            }
            cs += lc;
            J += lj;
        }
        charge += cs;
    }
    RunFields &F = A.fields[run];
    F.charge[x] = charge;
    F.J[x] = J;
}

// ---------------------------------------------------------------- Maxwell
// The six fields By, Bz, Ey, Ez, Ay, Az are formed by threads of their own (q = 0 .. 5) and
// the two components of a^2 by neighbouring lanes: the stage is a few chains of FP64
// operations, each of which occupies a sub-partition's unit for about 64 cycles per warp
// whatever its lanes do, so it is as long as the warps sharing a unit are many.  One thread
// per cell put all of n = 8192 on a fifth of the GPU's 608 units, two warps each: right-hand
// side, combination and a^2 took 20.5 us, 9.7 now (n = 1062: 19.1, 8.7).
// Every sum and product is rounded by itself (mul, add, sub), so that all forms, compiled
// with contraction or without, agree bit for bit.
constexpr int kMxFields = 6;
constexpr int kMxThreads = 128;  // a warp per sub-partition

__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }

__device__ __forceinline__ double *mx_field(const RunFields &F, int q) {
    double *const X[kMxFields] = {F.By, F.Bz, F.Ey, F.Ez, F.Ay, F.Az};
    return X[q];
}

// Right-hand side of field q into slot step+2 from slot 1 (EMSolver.cpp:479-553).
__device__ __forceinline__ void mx_rhs_cell(const MaxwellLaunch &L, int run, int i, int q) {
    RunFields &F = L.fields[run];
    const int nf = F.nf;
    if (i >= nf) return;
    const double dx_inv = L.dxinv[run];
    const double eps0_inv = kEps0Inv, mu_inv = kMuInv;
    const int pre = F.pre, n = F.n;
    const bool first = i == 0, second = first || i < pre || (i >= pre + n && i < nf - 2);
    double r = 0;
    if (second || (i >= pre && i < pre + n)) {
        if (q >= 4) {
            r = q == 4 ? -F.Ey[nf + i] : -F.Ez[nf + i];
        } else if (q < 2) {
            const double *E = (q == 0 ? F.Ez : F.Ey) + nf;
            const double d = q == 0 ? dx_inv : -dx_inv;
            if (second) {
                r = mul(d, sub(E[i + 1], E[i]));
            } else {
                const double c1 = -1.0 / 24;
                const double c2 = 9.0 / 8.0;
                r = mul(d, add(mul(c1, sub(E[i + 2], E[i - 1])), mul(c2, sub(E[i + 1], E[i]))));
            }
        } else {
            const double *B = (q == 2 ? F.Bz : F.By) + nf;
            const double d = q == 2 ? -dx_inv : dx_inv;
            if (second) {  // left of the first cell: the boundary value
                const double bm = first ? L.params[param_base(run, L.step) + (q == 2 ? 17 : 16)] : B[i - 1];
                r = mul(mul(mul(d, sub(B[i], bm)), eps0_inv), mu_inv);
            } else {
                const double c1 = -1.0 / 24;
                const double c2 = 9.0 / 8.0;
                const double A = (q == 2 ? F.Ay : F.Az)[nf + i], Jv = F.J[i - pre];
                const double curl = mul(d, add(mul(c1, sub(B[i + 1], B[i - 2])), mul(c2, sub(B[i], B[i - 1]))));
                r = sub(mul(mul(curl, eps0_inv), mu_inv), mul(mul(eps0_inv, Jv), A));
            }
        }
    }
    mx_field(F, q)[(L.step + 2) * nf + i] = r;
}

// Stage combination (EMSolver.cpp:204-338).  coef[0..5] are the dt-scaled weights of
// slots 2..7; the last stage writes slot 0 from slot 1 and copies it back to slot 1.
__device__ __forceinline__ void mx_update_cell(const MaxwellLaunch &L, int run, int i, int q) {
    RunFields &F = L.fields[run];
    const int nf = F.nf, step = L.step;
    if (i >= nf) return;
    const double *c = L.params + param_base(run, step) + 8;
    double *X = mx_field(F, q) + i;
    double v = step < 5 ? X[0] : X[nf];
    double x[6];
#pragma unroll
    for (int k = 0; k < 6; k++) x[k] = k <= step ? X[(k + 2) * nf] : 0.0;
#pragma unroll
    for (int k = 0; k < 6; k++)
        if (k <= step) v = add(v, mul(c[k], x[k]));
    if (step == 5) X[0] = v;
    X[nf] = v;
}

// WENO-weighted (unmapped) face value of A (EMSolver.cpp:555-619).
__device__ __forceinline__ double face_a(double f1, double f2, double f3, double f4) {
    const double c6 = 1.0 / 6;
    const double c43 = 4.0 / 3;
    const double fL = mul(c6, add(add(-f1, mul(5, f2)), mul(2, f3)));
    const double fR = mul(c6, sub(add(mul(2, f2), mul(5, f3)), f4));
    const double AL = add(sub(f1, mul(2, f2)), f3);
    const double BL = sub(f3, f1);
    const double AR = add(sub(f2, mul(2, f3)), f4);
    const double BR = sub(f4, f2);
    const double bL = add(add(mul(c43, mul(AL, AL)), mul(mul(0.5, AL), BL)), mul(0.25, mul(BL, BL)));
    const double bR = add(sub(mul(c43, mul(AR, AR)), mul(mul(0.5, AR), BR)), mul(0.25, mul(BR, BR)));
    const double mm = 1.0e-10;
    const double dL = mul(add(mm, bL), add(mm, bL)), dR = mul(add(mm, bR), add(mm, bR));
    // dL, dR are at least about 1e-20; below 2^600 (A below 1e45) the quotients take the short
    // form with the rounding of `/`
    double wL, wR;
    bool gen = !(__double2hiint(dL) < 0x65700000 && __double2hiint(dR) < 0x65700000);
    if (!gen) {
        const double oL = div_rn(0.5, dL, rcp_ulp(dL), gen), oR = div_rn(0.5, dR, rcp_ulp(dR), gen);
        const double o = add(oL, oR), y = rcp_ulp(o);
        wL = div_rn(oL, o, y, gen);
        wR = div_rn(oR, o, y, gen);
    }
    if (gen) {
        const double oL = div_call(0.5, dL), oR = div_call(0.5, dR);
        wL = div_call(oL, add(oL, oR));
        wR = div_call(oR, add(oL, oR));
    }
    return add(mul(wL, fL), mul(wR, fR));
}

// Component c (0: y, 1: z) of A at the face left of cell i of the box.
__device__ __forceinline__ double mx_face_a(const RunFields &F, int i, int c) {
    const double *A = (c ? F.Az : F.Ay) + F.nf + F.pre + i;
    return face_a(A[-2], A[-1], A[0], A[1]);
}

// a^2 there from the two, and (f32) the per-cell A^2 of field cell x that the next stage's
// FP32 moments read (as acell32_cell), unfused.
__device__ __forceinline__ void mx_asq_store(const MaxwellLaunch &L, const RunFields &F, int i, double a_y, double a_z) {
    const double a = add(mul(a_y, a_y), mul(a_z, a_z));
    F.asq[i] = a;
    if (L.asq32_out) F.asq32[i] = (float)a;
}
__device__ __forceinline__ void mx_acell(const RunFields &F, int x) {
    const double ay = F.Ay[F.nf + x], az = F.Az[F.nf + x];
    F.acell32[x] = (float)add(mul(ay, ay), mul(az, az));
}

// One thread per cell of the field grid.
__device__ __forceinline__ void mx_asq_cell(const MaxwellLaunch &L, int run, int x) {
    const RunFields &F = L.fields[run];
    if (x >= F.nf) return;
    if (L.f32) mx_acell(F, x);
    const int i = x - F.pre;
    if (i >= 0 && i < F.n) mx_asq_store(L, F, i, mx_face_a(F, i, 0), mx_face_a(F, i, 1));
}

// Two lanes per cell, t = 2 x + component (whole warps).
__device__ __forceinline__ void mx_asq_pair(const MaxwellLaunch &L, int run, int t) {
    const RunFields &F = L.fields[run];
    const int x = t >> 1, c = t & 1, i = x - F.pre;
    const bool face = i >= 0 && i < F.n;
    const double mine = face ? mx_face_a(F, i, c) : 0.0;
    const double other = __shfl_xor_sync(0xffffffffu, mine, 1);
    if (c == 0 && face) mx_asq_store(L, F, i, mine, other);
    if (c == 1 && L.f32 && x < F.nf) mx_acell(F, x);
}

}  // namespace vx
