// Device bodies of the AMR op batches built in amr.cpp (ghost fills, coarse/fine
// interface fluxes, limiter coefficient exchange; one op per call) and the coarse-level
// interpolation, shared by amr64.cu (FP64 patches, compiled without contraction, so every
// expression keeps the reference's operation order) and stage32.cu (FP32 patches of the
// precision form).
#pragma once
#include <cuda_runtime.h>

#include "amr.hpp"
#include "vx_kernels.hpp"

namespace vx {

template <class T>
__device__ __forceinline__ T *slot_plane(const PatchT<T> &P, int slot) {
    return slot == 0 ? P.f0 : (slot == 1 ? P.f1 : P.f2);
}

template <class T>
__device__ __forceinline__ T dmin(T a, T b) { return (b < a) ? b : a; }  // std::min

// Rectangle::GetInterpolantsREF (Rectangle.cpp:121-137): r values from five cells.
template <class T>
__device__ __forceinline__ void interp_ref(const double *c, int r, T f1, T f2, T f3, T f4, T f5, T *out) {
    const T m0 = (T)0.104166666666667, m1 = (T)-0.708333333333334, m2 = (T)0.708333333333334,
            m3 = (T)-0.104166666666667;
    const T m4 = (T)0.117647058823529, m5 = (T)0.029411764705882, m6 = (T)0.029411764705882,
            m7 = (T)0.117647058823529;
    const T m8 = (T)-0.083333333333333, m9 = (T)0.166666666666667, m10 = (T)-0.166666666666667,
            m11 = (T)0.083333333333334;
    f5 -= f3;
    f4 -= f3;
    f2 -= f3;
    f1 -= f3;
    T a1 = m0 * f1 + m1 * f2 + m2 * f4 + m3 * f5;
    T a2 = m4 * f1 + m5 * f2 + m6 * f4 + m7 * f5;
    T a3 = m8 * f1 + m9 * f2 + m10 * f4 + m11 * f5;
    for (int i = 0; i < r; i++) out[i] = (T)c[3 * i] * a1 + (T)c[3 * i + 1] * a2 + (T)c[3 * i + 2] * a3 + f3;
}

constexpr int kMaxR = 8;

// Rectangle::GetWenoValueFromCoarseLevel (Rectangle.cpp:343-415): the corrected r x r
// interpolants of coarse cell (ic, jc), out[kx * r + kp] for x sub-cell kx, p sub-cell kp.
// R: the refinement ratio when known at compile time (its arrays are then registers; with
// the general bound they are 104 words of local memory per thread), 0 otherwise.
template <int R, class T>
__device__ __forceinline__ void interp_block_r(const PatchT<T> &C, const T *f, int ic, int jc, T *out) {
    const int r = R ? R : C.r;
    const int pit = C.pitch;
    T temps[5][R ? R : kMaxR];
#pragma unroll
    for (int k = -2; k < 3; k++)
        interp_ref(C.refc, r, f[pidx(ic - 2, jc + k, pit)], f[pidx(ic - 1, jc + k, pit)], f[pidx(ic, jc + k, pit)],
                   f[pidx(ic + 1, jc + k, pit)], f[pidx(ic + 2, jc + k, pit)], temps[k + 2]);
    T sum = 0;
#pragma unroll
    for (int k = 0; k < r; k++) {
        interp_ref(C.refc, r, temps[0][k], temps[1][k], temps[2][k], temps[3][k], temps[4][k], out + k * r);
        for (int l = 0; l < r; l++) sum += out[k * r + l];
    }
    // 1 / r^2: r^2 is an exact small integer (the reference's std::pow(r, 2) gives it)
    T correction = f[pidx(ic, jc, pit)] - (T)1 / (T)(r * r) * sum;
#pragma unroll
    for (int q = 0; q < r * r; q++) out[q] += correction;
}
template <class T>
__device__ void interp_block(const PatchT<T> &C, const T *f, int ic, int jc, T *out) {
    if (C.r == 2) interp_block_r<2>(C, f, ic, jc, out);
    else interp_block_r<0>(C, f, ic, jc, out);
}

// Entry `sub` of interp_block.
template <class T>
__device__ __noinline__ T coarse_interp_any(const PatchT<T> &C, const T *f, int ic, int jc, int sub) {
    T out[kMaxR * kMaxR];
    interp_block_r<0>(C, f, ic, jc, out);
    return out[sub];
}
template <class T>
__device__ __forceinline__ T coarse_interp(const PatchT<T> &C, const T *f, int ic, int jc, int sub) {
    if (C.r != 2) return coarse_interp_any(C, f, ic, jc, sub);
    T out[4];
    interp_block_r<2>(C, f, ic, jc, out);
    return sub == 0 ? out[0] : sub == 1 ? out[1] : sub == 2 ? out[2] : out[3];
}

template <class T>
__device__ __forceinline__ void ghost_op(const PatchT<T> *patches, const GhostOp *ops, int k, int slot) {
    const GhostOp op = ops[k];
    const PatchT<T> &D = patches[op.dst];
    T v = 0;
    if (op.kind == kGhostCopy) {
        const PatchT<T> &S = patches[op.src];
        v = slot_plane(S, slot)[pidx(op.si, op.sj, S.pitch)];
    } else if (op.kind == kGhostInterp) {
        const PatchT<T> &S = patches[op.src];
        v = coarse_interp(S, slot_plane(S, slot), op.si, op.sj, op.sub);
    }
    slot_plane(D, slot)[pidx(op.di, op.dj, D.pitch)] = v;
}

// FP64, refinement ratio 2: a warp's ops (valid: this lane has one).  The four sub-cells of
// a coarse cell are consecutive ops, and each alone would form all of its r x r block: 270
// FP64 operations, and an FP64 instruction takes 64 cycles of its sub-partition's unit
// whatever its lanes do.  Four lanes that find each other (any position in the warp) share
// them: a row of the stencil each, the fifth row together, then each its x sub-cell:
// 120 operations in the same order.  Ops on their own take the single form.  Ghost fill
// of 50 x 38 in two levels 14.7 -> 9.2 us, of 4096 x 512 27.1 -> 16.3 us.
__device__ __forceinline__ void ghost_op_warp(const PatchT<double> *patches, const GhostOp *ops, int k, bool valid,
                                              int slot) {
    const unsigned full = 0xffffffffu;
    GhostOp op{};
    if (valid) op = ops[k];
    const bool interp = valid && op.kind == kGhostInterp && patches[op.src].r == 2;
    // the coarse cell: patch, and its cell by offset in the padded block (lanes without one: their own)
    unsigned long long key = (1ull << 63) | (unsigned)(threadIdx.x & 31);
    if (interp) key = ((unsigned long long)op.src << 32) | (unsigned)pidx(op.si, op.sj, patches[op.src].pitch);
    const unsigned mates = __match_any_sync(full, key);
    const unsigned upper = __ballot_sync(full, (op.sub >> 1) != 0) & mates, lower = mates & ~upper;
    const bool four = interp && __popc(mates) == 4 && upper && lower;
    double v = 0.0;
    if (__any_sync(full, four)) {
        // the mates in lane order; lanes of no group take part in the shuffles alone
        const int rank = __popc(mates & ((1u << (threadIdx.x & 31)) - 1));
        unsigned rest = four ? mates : full;
        int lane[4];
#pragma unroll
        for (int t = 0; t < 4; t++) {
            lane[t] = __ffs(rest) - 1;
            rest &= rest - 1;
        }
        double row[2] = {0.0, 0.0}, last[2] = {0.0, 0.0}, centre = 0.0;
        const PatchT<double> &C = patches[four ? op.src : 0];
        if (four) {
            const double *f = slot_plane(C, slot);
            const int pit = C.pitch, i = op.si, j = op.sj;
            auto form = [&](int c, double *out) {
                interp_ref(C.refc, 2, f[pidx(i - 2, c, pit)], f[pidx(i - 1, c, pit)], f[pidx(i, c, pit)],
                           f[pidx(i + 1, c, pit)], f[pidx(i + 2, c, pit)], out);
            };
            form(j - 2 + rank, row);
            form(j + 2, last);
            centre = f[pidx(i, j, pit)];
        }
        const bool up = op.sub >> 1;
        double x[4];
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const double a = __shfl_sync(full, row[0], lane[t]), b = __shfl_sync(full, row[1], lane[t]);
            x[t] = up ? b : a;
        }
        double out[2] = {0.0, 0.0};
        if (four) interp_ref(C.refc, 2, x[0], x[1], x[2], x[3], up ? last[1] : last[0], out);
        const int l0 = four ? __ffs(lower) - 1 : 0, l1 = four ? __ffs(upper) - 1 : 0;
        const double o00 = __shfl_sync(full, out[0], l0), o01 = __shfl_sync(full, out[1], l0);
        const double o10 = __shfl_sync(full, out[0], l1), o11 = __shfl_sync(full, out[1], l1);
        if (four) {
            double sum = 0.0;
            sum += o00;
            sum += o01;
            sum += o10;
            sum += o11;
            v = ((op.sub & 1) ? out[1] : out[0]) + (centre - 0.25 * sum);
        }
    }
    if (four) {
        const PatchT<double> &D = patches[op.dst];
        slot_plane(D, slot)[pidx(op.di, op.dj, D.pitch)] = v;
    } else if (valid) {
        ghost_op(patches, ops, k, slot);
    }
}

// A row of restrictions (Rectangle::GetValueFromFinerLevel, Rectangle.cpp:314-327), by one
// warp: neighbouring lanes take neighbouring cells.
template <class T>
__device__ __forceinline__ void restrict_row(const PatchT<T> *patches, const GhostOp *rows, int k, int lane, int slot) {
    const GhostOp op = rows[k];
    const PatchT<T> &D = patches[op.dst];
    const PatchT<T> &S = patches[op.src];
    const int r = D.r, pit = S.pitch;
    const T *f = slot_plane(S, slot) + pidx(op.si, op.sj, pit);
    T *d = slot_plane(D, slot) + pidx(op.di, op.dj, D.pitch);
    // std::pow(r, 2.0) of the reference, an exact integer; for a power of two the
    // product with its exact reciprocal is the same correctly rounded value
    if (r == 2 && (reinterpret_cast<uintptr_t>(f) | pit * sizeof(T)) % (2 * sizeof(T)) == 0) {
        // a block is two pairs (a patch starts on a whole coarse cell, so they are aligned): the
        // ghost fill of 38.6 M cells in three levels 64.8 -> 39.4 us
        struct alignas(2 * sizeof(T)) Pair {
            T a, b;
        };
#pragma unroll 4
        for (int c = lane; c < op.sub; c += 32) {
            const Pair u = *reinterpret_cast<const Pair *>(f + 2 * c);
            const Pair w = *reinterpret_cast<const Pair *>(f + pit + 2 * c);
            d[c] = (((u.a + u.b) + w.a) + w.b) * (T)0.25;
        }
        return;
    }
    const bool pow2 = (r & (r - 1)) == 0;
    const T inv = (T)(1.0f / (float)(r * r));
    for (int c = lane; c < op.sub; c += 32) {
        T t = 0;
        for (int a = 0; a < r; a++)
            for (int b = 0; b < r; b++) t += f[a * pit + c * r + b];
        if (pow2) t *= inv;
        else t /= (T)(r * r);
        d[c] = t;
    }
}
// Op batch as one launch: ops one per thread, then rows one per warp (thread index e).
template <class T>
__device__ __forceinline__ void ghost_work(const PatchT<T> *patches, const GhostOp *ops, int n, const GhostOp *rows,
                                           int nrows, long long e, int slot) {
    const long long pad = ((long long)n + 31) / 32 * 32;
    if (e < pad) {
        if constexpr (sizeof(T) == 8) ghost_op_warp(patches, ops, (int)e, e < n, slot);
        else if (e < n) ghost_op(patches, ops, (int)e, slot);
    } else if ((e - pad) / 32 < nrows) {
        restrict_row(patches, rows, (int)((e - pad) / 32), (int)(e & 31), slot);
    }
}

// Coarse faces on a coarse/fine interface: the mean of the finer patch's fluxes through
// the r fine faces (CalculateFluxToCoarse*, Rectangle.hpp:132-178).  The high-order mean
// uses the fine patch's stage fluxes; the stage-0 low-order mean recomputes each fine
// donor-cell flux the way RGKGetFluxXL/PL do, (dx_inv * f) * a (Rectangle.cpp:1216-1253).
// FP64: the face's antidiffusive stage flux (what the flux kernels form for all other
// faces) follows from its stage fluxes so far; the FP32 form has a pass for it.
template <class T>
__device__ __forceinline__ T stage_flux(T *const *H, int id, const double *a, int step, T low) {
    T h = a[0] * H[0][id];
    for (int k = 1; k <= step; k++) {
        if (step == 5 && k == 1) continue;  // b_1 = 0 (Rectangle.cpp:1494)
        h = h + a[k] * H[k][id];
    }
    return h - a[6] * low;
}

template <class T>
__device__ __forceinline__ void iface_op(const PatchT<T> *patches, const IfaceOp *ops, int k, int step,
                                         const double *params) {
    const IfaceOp op = ops[k];
    const PatchT<T> &C = patches[op.coarse];
    const PatchT<T> &F = patches[op.fine];
    const int r = C.r;
    const int cid = pidx(op.ci, op.cj, C.pitch);
    const T scale = (T)(1.0 / (r * r));
    const T *f = F.f1;
    const T dxi = (T)F.dx_inv, dpi = (T)F.dp_inv;
    if (op.dir == 0) {
        T t = 0;
        for (int q = 0; q < r; q++) t += F.FxH[step][pidx(op.fi, op.fj + q, F.pitch)];
        C.FxH[step][cid] = t * scale;
        if (step == 0) {
            T tl = 0;
            for (int q = 0; q < r; q++) {
                const int fid = pidx(op.fi, op.fj + q, F.pitch);
                T lo;
                // the FP32 form keeps no face-velocity plane; its FxL is this value
                if (sizeof(T) == 4 || (F.ifx && F.ifx[fid])) lo = F.FxL[fid];
                else {
                    const T am = F.ex[fid];
                    lo = dxi * (am > (T)0 ? f[fid - F.pitch] : f[fid]) * am;
                }
                tl += lo;
            }
            C.FxL[cid] = tl * scale;
        }
        if (sizeof(T) == 8) C.FxDS[cid] = stage_flux(C.FxH, cid, params + param_base(C.run, step), step, C.FxL[cid]);
    } else {
        T t = 0;
        for (int q = 0; q < r; q++) t += F.FpH[step][pidx(op.fi + q, op.fj, F.pitch)];
        C.FpH[step][cid] = t * scale;
        if (step == 0) {
            T tl = 0;
            for (int q = 0; q < r; q++) {
                const int fid = pidx(op.fi + q, op.fj, F.pitch);
                T lo;
                if (sizeof(T) == 4 || (F.ifp && F.ifp[fid])) lo = F.FpL[fid];
                else {
                    const T am = F.ep[fid];
                    lo = dpi * (am > (T)0 ? f[fid - 1] : f[fid]) * am;
                }
                tl += lo;
            }
            C.FpL[cid] = tl * scale;
        }
        if (sizeof(T) == 8) C.FpDS[cid] = stage_flux(C.FpH, cid, params + param_base(C.run, step), step, C.FpL[cid]);
    }
}

// Limiter coefficient exchange (Rectangle.cpp:1625-1917).
template <class T>
__device__ __forceinline__ void csync_op(const PatchT<T> *patches, const CSyncOp *ops, int k) {
    const CSyncOp op = ops[k];
    const PatchT<T> &N = patches[op.nb];
    const PatchT<T> &R = patches[op.caller];
    const int t = op.t;
    const bool xf = t < 2;
    T *NC = xf ? N.Cx : N.Cp;
    T *RC = xf ? R.Cx : R.Cp;
    const T *NDS = xf ? N.FxDS : N.FpDS;
    const T *RDS = xf ? R.FxDS : R.FpDS;
    const int nid = pidx(op.ni, op.nj, N.pitch);
    const int cid = pidx(op.ci, op.cj, R.pitch);
    const int nprev = xf ? nid - N.pitch : nid - 1;  // (ni-1, nj) or (ni, nj-1)
    const int cprev = xf ? cid - R.pitch : cid - 1;
    const T zero = 0;
    if (op.kind == kCSame) {  // SetCFromSameLevel
        T v;
        if (t == 0 || t == 2)
            v = NDS[nid] > zero ? dmin(R.Rp[cid], N.Rm[nprev]) : dmin(N.Rp[nprev], R.Rm[cid]);
        else
            v = NDS[nid] > zero ? dmin(R.Rm[cprev], N.Rp[nid]) : dmin(N.Rm[nid], R.Rp[cprev]);
        NC[nid] = v;
        RC[cid] = v;
    } else if (op.kind == kCUpdate) {  // UpdateCFromSameLevel
        T v = dmin(NC[nid], RC[cid]);
        NC[nid] = v;
        RC[cid] = v;
    } else {  // SetCFromDifferentLevel
        const int r = N.r;
        T v = NC[nid];
        for (int q = 0; q < r; q++) {
            const int fid = xf ? cid + q : cid + q * R.pitch;
            const int fprev = xf ? fid - R.pitch : fid - 1;
            if (t == 0 || t == 2) v = dmin(v, RDS[fid] > zero ? R.Rp[fid] : R.Rm[fid]);
            else v = dmin(v, RDS[fid] > zero ? R.Rm[fprev] : R.Rp[fprev]);
        }
        if (t == 0 || t == 2) v = dmin(v, NDS[nid] > zero ? N.Rm[nprev] : N.Rp[nprev]);
        else v = dmin(v, NDS[nid] > zero ? N.Rp[nid] : N.Rm[nid]);
        for (int q = 0; q < r; q++) RC[xf ? cid + q : cid + q * R.pitch] = v;
        NC[nid] = v;
    }
}

}  // namespace vx
