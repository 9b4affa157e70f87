// FP64 field-side kernels: momentum moments (Rectangle::CalculateRhoAndJ, MKL path
// Rectangle.cpp:157-237), finest-grid assembly (Level.cpp:19-62, EMSolver.cpp:104-122),
// Poisson solve with the precomputed LU factors (EMSolver.cpp:156-192), the transverse
// Maxwell RK stage with face interpolation of A (EMSolver.cpp:194-619) and the CFL bound
// (EMSolver.cpp:631-664).
//
// Compiled with --fmad=false so each double expression keeps the reference's operations
// and evaluation order.
#include <cuda_runtime.h>
#include <algorithm>
#include "div64.cuh"
#include "field_ops.cuh"
#include "poisson_lu.hpp"
#include "vx_kernels.hpp"

namespace vx {

using P64 = PatchT<double>;

// Interpolated value of f on the finest sub-cells of coarse cell (i, j), rtb > 1, with the
// conservative correction (Rectangle.cpp:139-155 and :183-204; the reference's fixed
// 12-entry interpolation matrix, Rectangle.cpp:76-89).  rel_shared forms what all
// sub-cells share — f3, the interpolation coefficients, the correction cor from the sum
// over every sub-cell's value — and sub-cell k's value is rel_pick(k) + cor, in the
// reference's operations and order.
__device__ __forceinline__ void rel_shared(const P64 &P, const double *f, int i, int j, double &f3, double &a1,
                                           double &a2, double &a3, double &cor) {
    const int pit = P.pitch;
    f3 = f[pidx(i, j, pit)];
    const double m0 = 0.104166666666667, m1 = -0.708333333333334, m2 = 0.708333333333334, m3 = -0.104166666666667;
    const double m4 = 0.117647058823529, m5 = 0.029411764705882, m6 = 0.029411764705882, m7 = 0.117647058823529;
    const double m8 = -0.083333333333333, m9 = 0.166666666666667, m10 = -0.166666666666667, m11 = 0.083333333333334;
    double g1 = f[pidx(i - 2, j, pit)] - f3;
    double g2 = f[pidx(i - 1, j, pit)] - f3;
    double g4 = f[pidx(i + 1, j, pit)] - f3;
    double g5 = f[pidx(i + 2, j, pit)] - f3;
    a1 = m0 * g1 + m1 * g2 + m2 * g4 + m3 * g5;
    a2 = m4 * g1 + m5 * g2 + m6 * g4 + m7 * g5;
    a3 = m8 * g1 + m9 * g2 + m10 * g4 + m11 * g5;
    double te = 0.0;
    for (int q = 0; q < P.rtb; q++) {
        double v = P.relc[3 * q] * a1 + P.relc[3 * q + 1] * a2 + P.relc[3 * q + 2] * a3 + f3;
        te += v;
    }
    cor = f3 - P.rtb_inv * te;
}
__device__ __forceinline__ double rel_pick(const P64 &P, int k, double a1, double a2, double a3, double f3) {
    return P.relc[3 * k] * a1 + P.relc[3 * k + 1] * a2 + P.relc[3 * k + 2] * a3 + f3;
}
// The same two for the fast FP64 form: multiply-adds fused (this file is otherwise
// compiled without contraction).
__device__ __forceinline__ void rel_shared_fma(const P64 &P, const double *f, int i, int j, double &f3, double &a1,
                                               double &a2, double &a3, double &cor) {
    const int pit = P.pitch;
    f3 = f[pidx(i, j, pit)];
    const double m0 = 0.104166666666667, m1 = -0.708333333333334, m2 = 0.708333333333334, m3 = -0.104166666666667;
    const double m4 = 0.117647058823529, m5 = 0.029411764705882, m6 = 0.029411764705882, m7 = 0.117647058823529;
    const double m8 = -0.083333333333333, m9 = 0.166666666666667, m10 = -0.166666666666667, m11 = 0.083333333333334;
    const double g1 = f[pidx(i - 2, j, pit)] - f3, g2 = f[pidx(i - 1, j, pit)] - f3;
    const double g4 = f[pidx(i + 1, j, pit)] - f3, g5 = f[pidx(i + 2, j, pit)] - f3;
    a1 = __fma_rn(m3, g5, __fma_rn(m2, g4, __fma_rn(m1, g2, m0 * g1)));
    a2 = __fma_rn(m7, g5, __fma_rn(m6, g4, __fma_rn(m5, g2, m4 * g1)));
    a3 = __fma_rn(m11, g5, __fma_rn(m10, g4, __fma_rn(m9, g2, m8 * g1)));
    double te = 0.0;
    for (int q = 0; q < P.rtb; q++)
        te += __fma_rn(P.relc[3 * q + 2], a3, __fma_rn(P.relc[3 * q + 1], a2, __fma_rn(P.relc[3 * q], a1, f3)));
    cor = __fma_rn(-P.rtb_inv, te, f3);
}
__device__ __forceinline__ double rel_pick_fma(const P64 &P, int k, double a1, double a2, double a3, double f3) {
    return __fma_rn(P.relc[3 * k + 2], a3, __fma_rn(P.relc[3 * k + 1], a2, __fma_rn(P.relc[3 * k], a1, f3)));
}

__device__ __forceinline__ double cell_asq(const RunFields &F, int x) {
    int i = x + F.pre;
    i = i > -1 ? i : 0;
    i = i < F.nf ? i : F.nf - 1;
    double ay = F.Ay[F.nf + i], az = F.Az[F.nf + i];
    return (ay * ay) + (az * az);
}

// One warp per coarse column i, a unit's kMomCols columns of one patch (or a third of them)
// per block; a warp forms its column's finest sub-columns k in pairs, the f stencil and the interpolation's
// shared part once per cell for the pair.  The warp walks p in windows of 32 lanes
// covering j0-1 .. j0+30: every lane computes the Lorentz factor at its p-face once
// (shared with the neighbouring face through shuffles instead of the reference's four
// Gamma calls per cell), the log ratio
//   L(j) = c2 * ln((g_{j+1} + c1 p_{j+1}) / (g_j + c1 p_j))
// (the reference's gm; gm1 and gp1 are L(j-1) and L(j+1), the same expressions), the
// interpolated f and the cell's charge/current contributions.  The window's 29
// contributions per sub-column then go through shared memory to the block's last warp,
// whose lanes each add one sub-column's in ascending j, which keeps the reference's
// accumulation order (Rectangle.cpp:207-255) exactly.  The serial sums thus take one
// FP64 warp instruction per cell for up to 30 sub-columns at once (an FP64 warp
// instruction occupies the sub-partition's FP64 unit for tens of cycles whatever the
// number of active lanes), and with two window buffers they run while the column warps
// form the next window.
// The coarse-column list is padded per patch to a multiple of kMomCols (padding: patch
// -1), so the warps of a block share n_p and rtb and step through the windows together.
constexpr int kMomOut = kMomWindow;  // outputs per window: j0 .. j0+28
constexpr int kMomSmallPart = 5;     // columns per block of k64_moments for small sets

// Two window buffers: the column warps fill one while the summing warp adds the other.
template <int PART>
struct MomSmem {
    double cc[2][PART][2][32], cj[2][PART][2][32];
    int redo;
};

// One window of column i's sub-columns k0 .. k0+kg-1 (kg <= 2): lane L covers the p index
// j = j0 - 1 + L; lanes 1 .. kMomOut return the charge and current contributions cc[q],
// cj[q] of their cell (zero where the cell is not used) and set `use`.  All 32 lanes
// take part (shuffles).  a[q]: q^2 A^2 of sub-column k0+q.
// ln(Gn / G) for the fast FP64 form.  Neighbouring nodes of a p grid differ by a factor
// 1 + dp / gamma, so z = (Gn - G) / (Gn + G) is small and ln(Gn / G) = 2 atanh(z) =
// 2 z (1 + z^2/3 + z^4/5 + z^6/7) to within z^8 / 9 < 1.2e-17 relative for |z| <= 0.01;
// otherwise the logarithm of the quotient.
__device__ __forceinline__ double fast_log_ratio(double Gn, double G) {
    const double s = Gn + G;
    // tests on the high words (a zero or a subnormal has exponent 0): no FP64 compares
    constexpr unsigned kExp = 0x7ff00000u, kHundredth = 0x3f847ae1u;  // high word of 0.01
    if (((unsigned)__double2hiint(G) & kExp) != 0 && ((unsigned)__double2hiint(s) & kExp) != 0) {
        const double z = (Gn - G) * rcp_ulp(s);
        if (((unsigned)__double2hiint(z) & 0x7fffffffu) < kHundredth) {
            const double z2 = z * z;
            const double poly = __fma_rn(z2, __fma_rn(z2, __fma_rn(z2, 1.0 / 7.0, 0.2), 1.0 / 3.0), 1.0);
            return (2.0 * z) * poly;
        }
        return log(Gn * rcp_ulp(G));
    }
    return log(Gn / G);
}

// FAST (the fast FP64 form): multiply-adds fused and the node ratio's logarithm as above;
// the same formulas, not the reference's rounding.
template <bool FAST>
__device__ __forceinline__ void mom_window(const P64 &P, const double *f, bool real, int i, int j0, int k0, int kg,
                                           const double a[2], double c1, double c2, int lane, double cc[2],
                                           double cj[2], bool &use) {
    const unsigned full = 0xffffffffu;
    const double c3 = 1 / 48.0;
    const int np = P.np, rtb = P.rtb, pit = P.pitch;
    const int j = j0 - 1 + lane;  // this lane's p index
    double p = 0.0, f3 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0, cor = 0.0;
    use = false;
    if (real) {
        p = FAST ? __fma_rn(P.dp, (double)(j + P.p_pos), P.pmin) : P.pmin + P.dp * (double)(j + P.p_pos);
        if (j <= np) {
            if (rtb == 1) f3 = f[pidx(i, j, pit)];
            else if (FAST) rel_shared_fma(P, f, i, j, f3, a1, a2, a3, cor);
            else rel_shared(P, f, i, j, f3, a1, a2, a3, cor);
        }
        use = lane >= 1 && lane <= kMomOut && j < np && !(P.nested && P.nested[pidx(i, j, pit)]);
    }
    for (int q = 0; q < kg; q++) {
        cc[q] = 0.0;
        cj[q] = 0.0;
        if (real) {
            double G = 1.0, V = 0.0;  // 1 past the last node: those lanes' logarithms are not used
            if (j <= np + 1) {
                const double x = FAST ? __fma_rn(__fma_rn(p, p, a[q]), P.g2, 1.0) : 1.0 + ((p * p) + a[q]) * P.g2;
                bool hard = false;
                const double g = sqrt_rn(x, hard);
                G = FAST ? __fma_rn(c1, p, g) : g + c1 * p;
                // after its first use, which covers the test; the fast form does without
                if (!FAST && hard) G = sqrt_call(x) + c1 * p;
            }
            if (j <= np) V = rtb == 1 ? f3 : (FAST ? rel_pick_fma(P, k0 + q, a1, a2, a3, f3) : rel_pick(P, k0 + q, a1, a2, a3, f3)) + cor;
            const double Gn = __shfl_down_sync(full, G, 1);
            // valid for lanes 0..30 (lane 31's Gn is its own G)
            double L;
            if (FAST) {
                L = c2 * fast_log_ratio(Gn, G);
            } else {
                bool hard = (unsigned)(exp_bits(G) - 963) > 120u;  // G beyond 2^-60 .. 2^60, or 0
                L = c2 * log(div_rn(Gn, G, rcp_ulp(G), hard));
                if (hard) L = c2 * log(Gn / G);  // likewise
            }
            const double Lm = __shfl_up_sync(full, L, 1);
            const double Lp = __shfl_down_sync(full, L, 1);
            const double Vm = __shfl_up_sync(full, V, 1);
            const double Vp = __shfl_down_sync(full, V, 1);
            if (use) {
                cc[q] = V;
                cj[q] = FAST ? __fma_rn(V, L, c3 * (Lp - Lm) * (Vp - Vm)) : V * L + c3 * (Lp - Lm) * (Vp - Vm);
            }
        }
    }
}

// ---- windows that cannot change a sum
// Most of a base patch's momentum range holds values many orders below the column's bulk
// (a thermal f falls by 2^96 within 12 thermal widths; cells under a finer patch count for
// nothing at all), and forming their contributions was most of the moments' work: about a
// hundred FP64 instructions per cell and sub-column.  k64_mom_screen bounds |f| per window
// and column, and a window whose every column lies 2^96 below its own largest value that
// counts (or is zero, or nested) is not formed.  That alone would be an approximation; what makes it
// exact is the summing lane, which carries lower and upper bounds through the sum.  Added
// to a sum more than 2^55 times larger, a skipped window's contributions leave it bit for
// bit as it is; otherwise they widen the bounds by more than they could ever move the sum
// (each rounded addition moves it by at most twice its addend), and, rounding being
// monotone, the exact sum stays between the two when the same contributions are added to
// both.  Once they meet (within a window of the bulk's first cells, where the sum has
// outgrown what was skipped below it) they are the reference's sum; a column where they
// do not (charge that cancels, a bulk of one cell) has its unit formed in full.  What is
// skipped is below 2^-87 of the sum, an ulp 2^-52 of it: by chance that happens to one sum
// in 2^34.
// Contributions are bounded from F >= |f| over the window's cells and stencil: charge
// |V| <= 8 F with the sub-cell interpolation (its weights sum to less than 7), F without;
// current |V L + (L+ - L-)(V+ - V-) / 48| <= 1.09 |V| max|L| with |L| <= dp (the logarithm
// of the node ratio grows by c1 dp / gamma per cell).  As computed, the ratio's cancellation
// at negative p puts 4 gamma^2 2^-53 on top: below gamma = 1e6 that is lost in the bound's
// margin, and beyond it (where the ratio comes to 1 / 0, too) every window is formed.
struct MomSum {
    double lo0 = 0.0, hi0 = 0.0, lo1 = 0.0, hi1 = 0.0;
    __device__ __forceinline__ bool split() const { return !(lo0 == hi0 && lo1 == hi1); }
    // a skipped window whose contributions are at most e in size each
    static __device__ __forceinline__ void widen(double &lo, double &hi, double e) {
        if (e == 0.0 || (lo == hi && e < fabs(lo) * 0x1p-55)) return;
        lo = __dadd_rd(lo, -(2 * kMomOut + 4) * e);
        hi = __dadd_ru(hi, (2 * kMomOut + 4) * e);
    }
    // kMomOut contributions in ascending p (both: the bounds have not met)
    template <class A, class B>
    __device__ __forceinline__ void add(bool both, bool two, A a, B b) {
        if (!both) {
            if (two) {
#pragma unroll
                for (int t = 1; t <= kMomOut; t++) {
                    lo0 += a(t);
                    lo1 += b(t);
                }
            } else {
#pragma unroll
                for (int t = 1; t <= kMomOut; t++) lo0 += a(t);
            }
            hi0 = lo0;
            hi1 = lo1;
        } else {
            for (int t = 1; t <= kMomOut; t++) {
                const double v = a(t);
                lo0 += v;
                hi0 += v;
                if (two) {
                    const double w = b(t);
                    lo1 += w;
                    hi1 += w;
                }
            }
        }
    }
};

// What a summing lane adds: of a pair of sub-columns, lane = 2 column + sub-column takes
// the charge and the current; of a single one (rtb = 1), lanes 0 .. kMomCols-1 take the
// charges and the next kMomCols the currents, so that one FP64 instruction adds both.
struct MomLane {
    bool on, two, cur;
    int w, q;
    double f0, f1;  // bounds of one contribution over F
    // of the unit's columns c0 .. c0 + nc - 1 alone
    __device__ __forceinline__ MomLane(const P64 &P, int kg, int lane, int c0 = 0, int nc = kMomCols) {
        two = kg == 2;
        cur = !two && lane >= nc;
        w = c0 + (two ? lane >> 1 : (cur ? lane - nc : lane));
        on = lane < 2 * nc;
        if (!on) w = c0;
        q = two ? lane & 1 : 0;
        const double c = P.rtb > 1 ? 8.0 : 1.0, j = (P.rtb > 1 ? 10.0 : 1.25) * P.dp;
        f0 = on ? (cur ? j : c) : 0.0;
        f1 = on && two ? j : 0.0;
    }
    __device__ __forceinline__ void store(const MomLaunch &M, const P64 &P, int col0, int k0, const MomSum &s) const {
        if (!on || M.colpatch[col0 + w] < 0) return;
        const int cl = M.colidx[col0 + w] + k0 + q;  // i_w * rtb + k
        const double qc = P.q;
        if (!cur) P.chargeR[cl] = s.lo0 * (P.dp * qc);
        if (two || cur) P.currentR[cl] = (two ? s.lo1 : s.lo0) * (-qc * qc / P.mass);
    }
};

__device__ __forceinline__ int mom_windows(int np) { return (np + kMomOut - 1) / kMomOut; }

// Per unit and window: a bound F >= |f| for each column over the window's cells and the
// column's stencil, as the high word of a double (0: the column's contributions are all
// zero), and in word kMomCols whether the window is formed.  One block per unit, a warp per
// row of f: reads f once (4 rows of halo with the sub-cell interpolation).  Loads of
// kScreenWin windows are in flight together: 22 MB of the 4096 x 512 two-level workload
// took 48 us with eight warps that waited for each window, 16 us now.
constexpr int kScreenRows = kMomCols + 4, kScreenWin = 6;
__global__ void __launch_bounds__(kScreenRows * 32) k64_mom_screen(MomLaunch M) {
    VX_PDL_WAIT();
    extern __shared__ unsigned s_bound[];  // [row][window], bit 31 on a column's own row: none of its cells count
    __shared__ unsigned s_max[kMomCols];   // per column: largest |f| of the cells that count
    __shared__ int s_field[kMomCols];
    const unsigned full = 0xffffffffu;
    const int col0 = blockIdx.x * kMomCols, lane = threadIdx.x & 31, r = threadIdx.x >> 5;
    const P64 &P = ((const P64 *)M.patches)[M.colpatch[col0]];
    const int np = P.np, rtb = P.rtb, nwin = mom_windows(np), halo = rtb > 1 ? 2 : 0;
    // real columns: consecutive i, the padding at the end
    const int ncol = __popc(__ballot_sync(full, lane < kMomCols && M.colpatch[col0 + min(lane, kMomCols - 1)] >= 0));
    const int i0 = M.colidx[col0] / rtb;
    if (r < ncol + 2 * halo) {
        const int i = i0 - halo + r;
        const bool own = r >= halo && r < halo + ncol, nest = own && P.nested;
        const double *f = P.f1 + pidx(i, 0, P.pitch);
        const uint8_t *nested = nest ? P.nested + pidx(i, 0, P.pitch) : nullptr;
        unsigned top = 0;
        for (int w0 = 0; w0 < nwin; w0 += kScreenWin) {
            double v[kScreenWin];
            bool counts[kScreenWin];
#pragma unroll
            for (int k = 0; k < kScreenWin; k++) {
                const int j = kMomOut * (w0 + k) - 1 + lane;
                v[k] = j <= np ? f[j] : 0.0;  // windows past the last: nothing
                counts[k] = nest && lane >= 1 && lane <= kMomOut && j < np && !nested[j];
            }
#pragma unroll
            for (int k = 0; k < kScreenWin; k++) {
                const unsigned h = (unsigned)__double2hiint(v[k]) & 0x7fffffffu;
                const unsigned e = (h | (unsigned)__double2loint(v[k])) ? min(h + 1u, 0x7fffffffu) : 0u;
                unsigned m = __reduce_max_sync(full, e);
                if (nest) {
                    top = max(top, __reduce_max_sync(full, counts[k] ? e : 0u));
                    if (!__any_sync(full, counts[k])) m |= 0x80000000u;
                } else {
                    top = max(top, m);
                }
                if (lane == 0 && w0 + k < nwin) s_bound[r * nwin + w0 + k] = m;
            }
        }
        if (own && lane == 0) s_max[r - halo] = top;
    }
    if (threadIdx.x < ncol) {
        // gamma^2 - 1 < 1e12 over the column's nodes (false for a field that is not a number)
        const double pe = fmax(fabs(P.pmin + P.dp * (P.p_pos - 1)), fabs(P.pmin + P.dp * (P.p_pos + np + 1)));
        bool fin = true;
        for (int k = 0; k < rtb; k++)
            fin = fin && (pe * pe + P.qq * cell_asq(M.fields[P.run], (i0 + (int)threadIdx.x + P.x_pos) * rtb + k)) * P.g2 < 1e12;
        s_field[threadIdx.x] = fin;
    }
    __syncthreads();
    constexpr unsigned kFar = 96u << 20;  // 2^96 in the exponent of a high word
    unsigned *out = M.screen + (size_t)blockIdx.x * M.maxnwin * kMomScreen;
    // sixteen lanes per window: a column each
    for (int w0 = 2 * r; w0 < nwin; w0 += 2 * kScreenRows) {
        const int w = w0 + (lane >> 4), c = lane & 15;
        unsigned b = 0;
        bool form = false;
        if (w < nwin && c < ncol && !(s_bound[(c + halo) * nwin + w] & 0x80000000u)) {
            for (int q = c; q <= c + 2 * halo; q++) b = max(b, s_bound[q * nwin + w] & 0x7fffffffu);
            form = !s_field[c] || (b && !(s_max[c] < 0x7ff00000u && b + kFar <= s_max[c]));
        }
        const unsigned any = __ballot_sync(full, form) & (0xffffu << (lane & 16));
        if (w < nwin) out[w * kMomScreen + c] = c < kMomCols ? b : any != 0;
    }
}

void launch_mom_screen64(const MomLaunch &M) {
    if (M.ncols == 0) return;
    const int smem = (kMomCols + 4) * M.maxnwin * (int)sizeof(unsigned);
    if (smem > 200 * 1024) {  // n_p beyond 78000: every window formed
        cudaMemsetAsync(M.screen, 1, (size_t)(M.ncols / kMomCols) * M.maxnwin * kMomScreen * sizeof(unsigned), M.stream);
        return;
    }
    if (smem > 48 * 1024) vx_allow_smem(k64_mom_screen);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(M.ncols / kMomCols);
    cfg.blockDim = dim3(kScreenRows * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = M.stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributePriority;  // beside the face kernels of the other stream
    attr[0].val.priority = M.priority;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_launch_pdl ? 2 : 1;
    cudaLaunchKernelEx(&cfg, k64_mom_screen, M);  // errors surface through cudaGetLastError
}

// One part of a unit: PART of the kMomCols columns of a unit of the padded column list, from
// c0, formed by a warp each and summed by warp PART.  A block of all fifteen keeps every
// FP64 unit of its SM in four warps' hands; where there are not enough units for every SM
// (a set of at most two per SM), three blocks of five spread a unit over three SMs: 50 x 38
// 63 -> 44 us, 2048 x 256 74 -> 61 us with the screen, but 6.65 -> 6.71 ms per step for the
// 657 units of 4096 x 512 in two levels (the summing warps do the same for fewer columns).
template <bool FAST, int PART>
__global__ void __launch_bounds__((PART + 1) * 32, PART == kMomCols ? 2 : 5) k64_moments(MomLaunch M) {
    VX_PDL_WAIT();
    constexpr int kParts = kMomCols / PART, nc = PART;
    static_assert(kMomCols % PART == 0, "parts of equal size");
    __shared__ MomSmem<PART> S;
    const int unit = blockIdx.x / kParts, c0 = (blockIdx.x % kParts) * PART;
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int col0 = unit * kMomCols;
    if (M.colpatch[col0 + c0] < 0) return;  // padding alone
    const bool summer = wid == PART;
    const int col = col0 + c0 + wid;
    const bool real = !summer && M.colpatch[col] >= 0;  // warp-uniform
    const P64 &P = ((const P64 *)M.patches)[M.colpatch[col0]];  // the unit's patch
    const int rtb = P.rtb, nwin = mom_windows(P.np);
    const int i = real ? M.colidx[col] / rtb : 0;
    const RunFields &F = M.fields[P.run];
    const unsigned *screen = M.screen + (size_t)unit * M.maxnwin * kMomScreen;
    const double minv = 1 / P.mass;
    const double c1 = minv * kCInv;
    const double c2 = 1 / c1;
    const double *f = P.f1;
    const unsigned full = 0xffffffffu;
    for (int k0 = 0; k0 < rtb; k0 += 2) {  // unit-uniform
        const int kg = rtb - k0 < 2 ? rtb - k0 : 2;
        double a[2] = {0.0, 0.0};
        for (int q = 0; q < kg; q++)
            if (real) a[q] = P.qq * cell_asq(F, (i + P.x_pos) * rtb + k0 + q);
        const MomLane ml(P, kg, lane, c0, nc);
        for (int pass = 0; pass < 2; pass++) {  // pass 1: every window, where pass 0 did not settle
            MomSum s;
            bool both = false;
            int next = 0;  // the summing warp's next window
            // the skipped windows before `w`, then window w from buffer bf
            auto add_to = [&](int w, int bf) {
                for (; next < w; next++) {
                    const double b = __hiloint2double((int)screen[next * kMomScreen + ml.w], 0);
                    MomSum::widen(s.lo0, s.hi0, b * ml.f0);
                    MomSum::widen(s.lo1, s.hi1, b * ml.f1);
                }
                if (w == nwin) return;
                both = __any_sync(full, s.split());
                const int k = ml.w - c0;
                const double *pc = ml.cur ? S.cj[bf][k][0] : S.cc[bf][k][ml.q], *pj = S.cj[bf][k][ml.q];
                s.add(both, ml.two, [&](int t) { return pc[t]; }, [&](int t) { return pj[t]; });
                next = w + 1;
            };
            int bf = 0, prev = -1;
            for (int w = 0; w < nwin; w++) {
                if (!pass && !screen[w * kMomScreen + kMomCols]) continue;  // unit-uniform
                if (!summer) {
                    double cc[2], cj[2];
                    bool use;
                    mom_window<FAST>(P, f, real, i, w * kMomOut, k0, kg, a, c1, c2, lane, cc, cj, use);
                    for (int q = 0; q < kg; q++) {
                        S.cc[bf][wid][q][lane] = cc[q];
                        S.cj[bf][wid][q][lane] = cj[q];
                    }
                } else if (prev >= 0) {
                    add_to(prev, bf ^ 1);  // the previous window, in ascending j
                }
                prev = w;
                bf ^= 1;
                __syncthreads();
            }
            if (summer) {
                if (prev >= 0) add_to(prev, bf ^ 1);
                add_to(nwin, 0);
                const bool redo = !pass && __any_sync(full, ml.on && M.colpatch[col0 + ml.w] >= 0 && s.split());
                if (lane == 0) S.redo = redo;
                if (!redo) ml.store(M, P, col0, k0, s);
            }
            __syncthreads();  // the next pair's first window reuses the buffers
            if (!S.redo) break;
            __syncthreads();
        }
    }
}

void launch_moments64(const MomLaunch &M) {
    if (M.ncols == 0) return;
    launch_mom_screen64(M);
    const int units = M.ncols / kMomCols;  // the list is padded per patch
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (units <= 2 * sms) {
        auto kern = M.fast ? k64_moments<true, kMomSmallPart> : k64_moments<false, kMomSmallPart>;
        vx_launch(kern, units * (kMomCols / kMomSmallPart), (kMomSmallPart + 1) * 32, 0, M.stream, M);
    } else {
        auto kern = M.fast ? k64_moments<true, kMomCols> : k64_moments<false, kMomCols>;
        vx_launch(kern, units, (kMomCols + 1) * 32, 0, M.stream, M);
    }
}

// ---------------------------------------------------------------- separable initial f
// Interior cells of an FP32 patch's slots 0 and 1: (float)(((dx_sum[i] dp_sum[j]) inv) fn),
// the host quadrature's product in its order (this file keeps IEEE multiplies unfused).
__global__ void k_fill_separable(float *f0, float *f1, int pitch, int nx, int np, const double *dx_sum,
                                 const double *dp_sum, double inv, double fn) {
    VX_PDL_WAIT();
    const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
    if (j >= np || i >= nx) return;
    const double v = dx_sum[i] * dp_sum[j] * inv;
    const float x = (float)(v * fn);
    const int id = pidx(i, j, pitch);
    f0[id] = x;
    f1[id] = x;
}

void launch_fill_separable(float *f0, float *f1, int pitch, int nx, int np, const double *dx_sum,
                           const double *dp_sum, double inv, double fn, cudaStream_t s) {
    vx_launch(k_fill_separable, dim3((np + 255) / 256, nx), 256, 0, s, f0, f1, pitch, nx, np, dx_sum, dp_sum, inv, fn);
}

// Rectangle::InitializeDistribution (Rectangle.cpp:616-665) for a problem whose
// InitialDistribution is a sum of product terms, f(x, p) = sum_t (X_t(x) * P_t(p)) / C_t.
// The host evaluates the hook's factors at every sample point (X over the patch's n_x *
// nvals x samples, P over its n_p * nvals p samples, with its own exp / sin); each
// thread forms one cell's nvals^2 samples in the reference's loop order and operation
// order (--fmad=false: no contraction), so the cell averages equal the host loop's bits.
__global__ void k64_quadrature(double *f0, double *f1, int pitch, int nx, int np, int nvals, int terms,
                               const double *X, const double *Pf, const double *C, double scale) {
    VX_PDL_WAIT();
    const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
    if (j >= np || i >= nx) return;
    const double *xr = X + (size_t)i * nvals, *pr = Pf + (size_t)j * nvals;
    const size_t xstride = (size_t)nx * nvals, pstride = (size_t)np * nvals;
    double temp = 0.0;
    for (int k = 0; k < nvals; k++) {
        for (int l = 0; l < nvals; l++) {
            double v = (xr[k] * pr[l]) / C[0];
            for (int t = 1; t < terms; t++) v = v + (xr[t * xstride + k] * pr[t * pstride + l]) / C[t];
            temp = temp + v;
        }
    }
    const double f = temp * scale;
    const int id = pidx(i, j, pitch);
    f0[id] = f;
    f1[id] = f;
}

void launch_quadrature64(double *f0, double *f1, int pitch, int nx, int np, int nvals, int terms, const double *X,
                         const double *Pf, const double *C, double scale, cudaStream_t s) {
    vx_launch(k64_quadrature, dim3((np + 127) / 128, nx), 128, 0, s, f0, f1, pitch, nx, np, nvals, terms, X, Pf, C,
              scale);
}

// ---------------------------------------------------------------- assembly
// FP64 runs; runs of the FP32 form go to launch_assemble32 (stage32.cu).
__global__ void k_assemble(AsmLaunch A) {
    VX_PDL_WAIT();
    const int run = blockIdx.y;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (run >= A.nruns) return;
    assemble_cell(A, run, x);
}

void launch_assemble(const AsmLaunch &A) {
    if (A.pairs) {
        launch_assemble32(A);
        return;
    }
    dim3 g((A.maxn + 255) / 256, A.nruns);
    vx_launch(k_assemble, g, 256, 0, A.stream, A);
}

// ---------------------------------------------------------------- Poisson
__device__ __forceinline__ double efield_at(const double *phi, int n, double fcoef, double ex0, int i) {
    int ip1 = i + 1, im1 = i - 1, ip2 = i + 2, im2 = i - 2;
    ip1 = (ip1 > -1) ? ip1 : (ip1 + n);
    im1 = (im1 > -1) ? im1 : (im1 + n);
    ip2 = (ip2 > -1) ? ip2 : (ip2 + n);
    im2 = (im2 > -1) ? im2 : (im2 + n);
    ip1 = (ip1 < n) ? ip1 : (ip1 - n);
    im1 = (im1 < n) ? im1 : (im1 - n);
    ip2 = (ip2 < n) ? ip2 : (ip2 - n);
    im2 = (im2 < n) ? im2 : (im2 - n);
    return -fcoef * (8 * (phi[ip1] - phi[im1]) - phi[ip2] + phi[im2]) + ex0;
}

// One block per run.  The triangular solves are linear recurrences; to keep the
// reference's rounding they run in the order of the column-oriented dgetrs (entries
// ascending in column for L, descending for U), one warp each, chunk by chunk of 256 rows
// staged in shared memory by the other warps.  FP64 dependent latency (~65 cycles per
// add/mul/fma, ~550 per IEEE division on this part, 37 per 64-bit shuffle) makes the chain
// length the cost, so the factors are stored in band form (exact zeros where the factor
// has none — subtracting a zero product never changes a partial sum, which is never -0
// here) and only the operations that need the previous row's value sit on the chain.
constexpr int kPoisRows = kPoisRowsHost;     // rows per chunk
constexpr int kPoisLA = 4;                   // look-ahead rows staged with each chunk
constexpr int kPoisBuf = kPoisRows + kPoisLA;

// Lower factor: staged rows of one chunk.
struct PoisFwdChunk {
    int a;                                    // first staged row
    double c[4][kPoisBuf];                    // band coefficients, c[d-1][row - a]
    double slotc[4][kPoisBuf];                // accumulator-lane coefficients per step
    int sload[4][kPoisBuf];                   // row taken up by each slot at each step
    int take[kPoisBuf];                       // slot finishing row step+4
};
// Upper factor: rows r0 - kPoisLA .. of a chunk starting at row r0 (zeros below row 0).
struct PoisBwdChunk {
    double2 c[4][kPoisBuf];                   // {u_{d+1}, d == 0 ? y : 1} of each row; c[3][0] = {0, 1}
    float2 lo[kPoisBuf];                      // FP32 {yl, u1}
    double diag[kPoisRows], rhs[kPoisRows];   // u_ii and the right-hand sides
};
union PoisChunk {
    PoisFwdChunk f;
    PoisBwdChunk b;
};

// Stage rows [a, b) (clamped to [0, n)) of the lower factor into B with threads
// t, t + nt, ...
__device__ void pois_stage_fwd(PoisFwdChunk &B, const BandFactor &F, int a, int b, int n, int t, int nt) {
    a = max(a, 0);
    b = min(b, n);
    const int cnt = b - a;
    if (t == 0) B.a = a;
    for (int k = t; k < cnt; k += nt) {
        const int r = a + k;
        B.c[0][k] = F.band[4 * r];
        B.c[1][k] = F.band[4 * r + 1];
        B.c[2][k] = F.band[4 * r + 2];
        B.c[3][k] = F.band[4 * r + 3];
        for (int sl = 0; sl < F.nslots; sl++) {
            B.slotc[sl][k] = F.slot_coef[(size_t)sl * n + r];
            B.sload[sl][k] = F.slot_load[(size_t)sl * n + r];
        }
        if (F.take) B.take[k] = F.take[r];
    }
    // buffer rows past n: neutral entries, so that a look-ahead read past the matrix's end
    // finds a zero coefficient and no row index
    for (int k = cnt + t; k < kPoisBuf; k += nt) {
        B.c[0][k] = B.c[1][k] = B.c[2][k] = B.c[3][k] = 0.0;
        for (int sl = 0; sl < 4; sl++) {  // every accumulator row of the buffer
            B.slotc[sl][k] = 0.0;
            B.sload[sl][k] = -1;
        }
        B.take[k] = -1;
    }
}

// Right-hand side of row r with its far entries subtracted in summation order.
__device__ __forceinline__ double pois_far(const BandFactor &F, const double *x, int r) {
    double s = x[r];
    for (int e = F.fptr[r]; e < F.fptr[r + 1]; e++) s = s - x[F.fcol[e]] * F.fval[e];
    return s;
}

// Rows lo .. hi-1 of a factor one after another on one thread, every operation as dgetrs
// has it: the upper factor's first rows, a chunk whose quotients did not all come out
// (far = false: the far entries are subtracted already), and factors whose far entries do
// not fit the sweeps' forms.
template <bool UPPER>
__device__ __noinline__ void pois_rows_plain(const BandFactor &F, int lo, int hi, int n, double *x, bool far) {
    for (int q = 0; q < hi - lo; q++) {
        const int i = UPPER ? hi - 1 - q : lo + q;
        double s = far ? pois_far(F, x, i) : x[i];
        for (int d = 4; d >= 1; d--) {
            const int c = UPPER ? i + d : i - d;
            if (c >= 0 && c < n) s = s - x[c] * F.band[4 * i + d - 1];
        }
        x[i] = UPPER ? s / F.diag[i] : s;
    }
}

// Stage the factors of rows [r0, r1) of the upper factor (they need no solution value):
// threads t of nt.
__device__ void pois_stage_bwd(PoisBwdChunk &B, const BandFactor &F, int r0, int r1, int t, int nt) {
    const int base = r0 - kPoisLA, rows = r1 - base;
    for (int k = t; k < rows; k += nt) {
        double v[kBwdCols] = {0.0, 0.0, 0.0, 0.0, 0.0};
        if (base + k >= 0)
            for (int c = 0; c < kBwdCols; c++) v[c] = F.sweep[(size_t)(base + k) * kBwdCols + c];
        B.c[0][k] = make_double2(v[0], v[3]);
        B.c[1][k] = make_double2(v[1], 1.0);
        B.c[2][k] = make_double2(v[2], 1.0);
        B.lo[k] = make_float2(__int_as_float(__double2loint(v[4])), __int_as_float(__double2hiint(v[4])));
        if (k >= kPoisLA) B.diag[k - kPoisLA] = F.diag[base + k];
    }
    if (t == 0) B.c[3][0] = make_double2(0.0, 1.0);
}
// Their right-hand sides with the far terms subtracted (the solution values of the last
// rows, which are known): threads t of nt, t < 0 takes no part.
__device__ void pois_rhs_bwd(PoisBwdChunk &B, const BandFactor &F, int r0, int r1, double *x, int t, int nt) {
    if (t < 0) return;
    for (int k = t; k < r1 - r0; k += nt) {
        const double v = pois_far(F, x, r0 + k);
        x[r0 + k] = v;
        B.rhs[k] = v;
    }
}

// The last rows of the upper factor, where its far columns lie: the triangle in dense form.
constexpr int kPoisTail = PoissonLU::Band::kTail;
struct PoisTail {
    double u[kPoisTail][kPoisTail], diag[kPoisTail], y[kPoisTail];  // y: rounded 1 / diag
};
__device__ void pois_stage_tail(PoisTail &T, const BandFactor &F, int t0, int t) {
    if (t >= kPoisTail) return;
    const int i = t0 + t;
    for (int c = 0; c < kPoisTail; c++) T.u[t][c] = 0.0;
    for (int d = 1; d <= 4 && t + d < kPoisTail; d++) T.u[t][t + d] = F.band[4 * i + d - 1];
    for (int e = F.fptr[i]; e < F.fptr[i + 1]; e++) T.u[t][F.fcol[e] - t0] = F.fval[e];
    T.diag[t] = F.diag[i];
    T.y[t] = F.sweep[(size_t)i * kBwdCols + 3];
}
// Solved by warp 0, a row per lane: column by column from the last, which subtracts every
// row's terms in descending column order as dgetrs does (a zero where the factor has no
// entry changes nothing).  The quotients on the way are short ones; each lane then checks
// its own against IEEE division, and if one differs the rows are solved again one by one.
// One thread with its operands in global memory took 8 us.
__device__ void pois_tail(const PoisTail &T, const BandFactor &F, int t0, double *x) {
    constexpr unsigned act = (1u << kPoisTail) - 1;
    const int l = threadIdx.x & 31;
    if (l >= kPoisTail) return;
    double s = x[t0 + l], mine = 0.0, num = 0.0;
    const double diag = T.diag[l], y = T.y[l];
    for (int c = kPoisTail - 1; c >= 0; c--) {
        const double u = T.u[l][c], q = div_short(s, diag, y);
        const double xc = __shfl_sync(act, q, c);
        if (l == c) {
            mine = q;
            num = s;
        }
        s = s - xc * u;
    }
    if (!__any_sync(act, __double_as_longlong(num / diag) != __double_as_longlong(mine))) x[t0 + l] = mine;
    else if (l == 0) pois_rows_plain<true>(F, t0, t0 + kPoisTail, t0 + kPoisTail, x, true);
}

// Forward sweep of one chunk, software-pipelined on lanes 0..7 of warp 0.  Row i's sum is
// ((((Fb - x4 c4) - x3 c3) - x2 c2) - x1 c1), x_d the solution d rows back, Fb the
// right-hand side minus its far entries (finished by the accumulator lanes 4..7).  Lane L <
// 4 holds the partial sum of row i+L, already reduced by every term but the one with
// x_{i-1}; when that value arrives, each lane subtracts its own product in the same two
// warp instructions, lane 0's result is x_i, and the partials shift down one lane while
// lane 3 takes up the next row's right-hand side.  On this part each FP64 warp instruction
// occupies the sub-partition's FP64 unit for tens of cycles whatever the number of active
// lanes, so the lanes carry the independent work for free.  Each lane walks its own
// coefficient stream with a pointer, the shift and the slot hand-over are one shuffle with
// a per-lane source, and no branch depends on the lane.  The operands of the next row are
// loaded at the top of each row, ahead of its multiply: the warp issues in order, and a
// load placed after the previous row's shuffle-dependent store would add its shared-memory
// latency to every row of the chain.  The look-ahead reads at most two rows past the
// chunk: the staged look-ahead rows, or past n the neutral entries pois_stage_fwd writes
// there (zero coefficients, no slot row).  198 cycles per row (204 rolled, 206 and 204 unrolled by
// three and four).
__device__ void pois_fwd_fast(const PoisFwdChunk &B, const BandFactor &F, int r0, int cnt, int n, double *x,
                              double &V, double &w1) {
    // Only lanes 0..7 (band lanes 0..3, accumulator lanes 4..7) run the recurrence.
    constexpr unsigned act = 0xffu;
    const int lane = threadIdx.x & 31;
    if (lane >= 8) return;
    const int slot = lane - 4;
    const bool is_slot = slot >= 0 && slot < F.nslots;
    const bool has_coef = lane < 4 || is_slot;
    const int k0 = r0 - B.a;
    // coefficient stream of this lane (lanes without a role read slot 0's and use zero)
    const double *cp = lane < 4 ? &B.c[lane][k0 + lane] : &B.slotc[is_slot ? slot : 0][k0];
    const int cstep = has_coef ? 1 : 0;
    // row indices the slot takes up, read two rows ahead so that x[row] is one row ahead
    const int *lp = &B.sload[is_slot ? slot : 0][k0];
    const int lstep = is_slot ? 1 : 0;
    const int base_src = lane < 3 ? lane + 1 : lane;
    // rows past the end of the matrix get a zero coefficient
    const int lim = lane < 4 ? n - 1 - lane - r0 : cnt;  // q > lim: row i+lane >= n
    double coef = (0 > lim || !has_coef) ? 0.0 : *cp;
    cp += cstep;
    int ld = is_slot ? *lp : -1;
    lp += lstep;
    int ldn = is_slot ? *lp : -1;
    lp += lstep;
    double vld = ld >= 0 ? x[ld] : 0.0;
    int tk = B.take[k0];
    double fb = (lane == 3 && r0 + 4 < n) ? x[r0 + 4] : 0.0;
#pragma unroll 2
    for (int q = 0; q < cnt; q++) {
        const int i = r0 + q;
        // row q+1's operands; a slot's row r >= step + 4 and the right-hand side x[i + 5]
        // are not yet overwritten by the sweep.  Rows past the chunk read the staged
        // look-ahead rows, or past n the neutral entries pois_stage_fwd leaves there.
        double coef_n = *cp;
        cp += cstep;
        if (q + 1 > lim || !has_coef) coef_n = 0.0;
        const int tk_n = B.take[k0 + q + 1];
        const double fb_n = (lane == 3 && i + 5 < n) ? x[i + 5] : 0.0;
        const double vld_n = ldn >= 0 ? x[ldn] : 0.0;
        const int ldnn = is_slot ? *lp : -1;
        lp += lstep;
        if (ld >= 0) V = vld;  // a slot takes up a new row's right-hand side
        const double nv = V - w1 * coef;
        const double xi = __shfl_sync(act, nv, 0, 8);
        const int src = (lane == 3 && tk >= 0) ? 4 + tk : base_src;  // tk < kMaxSlots = 4
        const double sh = __shfl_sync(act, nv, src, 8);
        V = (lane == 3 && tk < 0) ? fb : sh;
        if (lane == 0) x[i] = xi;
        w1 = xi;
        coef = coef_n;
        tk = tk_n;
        fb = fb_n;
        vld = vld_n;
        ld = ldn;
        ldn = ldnn;
    }
}

// FP32 neighbours of doubles, on the integer units: d2f truncates a double (its exponent is
// taken modulo 2^8: garbage beyond FP32's range), f2d is exact for normal floats.
__device__ __forceinline__ float d2f_bits(double d) {
    const unsigned hi = __double2hiint(d), lo = __double2loint(d);
    const unsigned w = __funnelshift_l(lo, hi, 3) ^ 0x40000000u;
    return __uint_as_float((w & 0x7fffffffu) | (hi & 0x80000000u));
}
__device__ __forceinline__ double f2d_bits(float f) {
    const unsigned u = __float_as_uint(f);
    return __hiloint2double((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u), u << 29);
}

// Backward sweep of one chunk: rows r0 + cnt - 1 down to r0, on lanes 0..7 of warp 0.
// Row k is x_k = a_k / u0, a_k = ((B_k - u3 x_{k+3}) - u2 x_{k+2}) - u1 x_{k+1} (the upper
// factor has three columns beside the diagonal).  Lane L < 3 holds the partial sum of row
// k - L, already reduced by every term but the one with x_{k+1}; each lane subtracts its
// own product in the same two warp instructions, and a third, fma(a, y, t), makes lane 0's
// sum x_k (y the rounded reciprocal of u0) and leaves the others as they are (y = 1, t =
// -0); one shuffle spreads x_k, one moves the partials down a lane.  t is a_k times the
// reciprocal's low part, at most half an ulp of x_k; ten of its digits are enough, so it
// is formed in FP32 from the truncated s_k - u1 x_{k+1}, on units the chain does not use,
// while the product and the difference run.  The quotient is then within 2^-20 ulp of the
// true one before its rounding (FP32's range holds t down to x = 1e-21: below, above FP32's
// range and at 0 it is simply wrong; a solution of zeros is not swept); the block checks every row against IEEE division
// afterwards and has the chunk redone if any differs, so the result is always the dgetrs
// rounding.  What bounds it is latency: three dependent FP64 instructions (63 cycles each)
// and the shuffles behind them, 250 cycles per row (an fma more for t, and its lane 0
// select: 320).
__device__ void pois_bwd_fast(const PoisBwdChunk &B, int r0, int cnt, double *x) {
    constexpr unsigned act = 0xffu;
    const int lane = threadIdx.x & 31;
    if (lane >= 8) return;
    const int k0 = r0 + cnt - 1, q0 = cnt - 1 + kPoisLA;  // first row and its buffer row
    const bool is0 = lane == 0, is2 = lane == 2;
    const int src = lane < 7 ? lane + 1 : 7;
    const double2 *pc = lane < 3 ? &B.c[lane][q0 - lane] : &B.c[3][0];
    const int sc = lane < 3 ? 1 : 0;
    // lane 2: the right-hand sides, from row k0 - 2 down (rows below the chunk are not read);
    // the others: the FP32 pair of the row
    const double *pl = is2 ? x + k0 - 2 : reinterpret_cast<const double *>(&B.lo[q0]);
    int left = is2 ? cnt - 2 : 0x7fffffff;
    double X = x[k0 + 1], V = 0.0;
    {
        const double x2 = x[k0 + 2], x3 = x[k0 + 3];
        if (is0) V = (x[k0] - x3 * B.c[2][q0].x) - x2 * B.c[1][q0].x;
        if (lane == 1 && cnt > 1) V = x[k0 - 1] - x2 * B.c[2][q0 - 1].x;
        if (is2 && cnt > 2) V = x[k0 - 2];
    }
    double2 c = *pc;
    double l = left > 0 ? *pl : 0.0;
#pragma unroll 2
    for (int q = cnt - 1; q >= 0; q--) {
        pc -= sc;
        pl--;
        left--;
        const double2 c_n = *pc;
        const double l_n = left > 0 ? *pl : 0.0;
        const double m = __dmul_rn(X, c.x);
        const float yl = __int_as_float(__double2loint(l)), u1 = __int_as_float(__double2hiint(l));
        const float tf = yl * (d2f_bits(V) - u1 * d2f_bits(X));
        const double t = is0 ? f2d_bits(tf) : -0.0;
        const double a = __dsub_rn(V, m);
        const double r = __fma_rn(a, c.y, t);
        X = __shfl_sync(act, r, 0, 8);
        const double down = __shfl_sync(act, r, src, 8);
        V = is2 ? l_n : down;
        if (is0) x[r0 + q] = r;
        c = c_n;
        l = l_n;
    }
}

constexpr int kPoisSmemMaxN = 16384;  // solution vector kept in shared memory up to this n

// ---- pipelined form: the solve follows the moment units of its run (k64_moments_poisson)
constexpr unsigned kPipeMaxPolls = 1u << 25;  // second bound of a wait (>= 64 ns per poll)

__device__ __forceinline__ unsigned long long pipe_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ unsigned pipe_ld_acquire(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ int pipe_ld_relaxed(const int *p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void pipe_bar(int bar, int nt) {
    asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(nt) : "memory");
}

// Waits until done counter ci has every unit it expects.  A wait that runs out records
// itself in *err and returns; so does every later wait at once (the step's values are
// then not valid, but every index stays what the host tables say: nothing goes out of
// bounds).
__device__ void pipe_wait(const PipeLaunch &K, int ci) {
    const unsigned need = (unsigned)K.need[ci] + (unsigned)K.phantom;
    const unsigned *p = K.state + kPipeDone + ci;
    if (pipe_ld_acquire(p) >= need) return;
    if (pipe_ld_relaxed(K.err) != 0) return;
    const unsigned long long t0 = pipe_ns();
    for (unsigned poll = 0;; poll++) {
        __nanosleep(32);
        if (pipe_ld_acquire(p) >= need) break;
        if ((poll & 63u) == 63u && pipe_ld_relaxed(K.err) != 0) break;
        if (poll >= kPipeMaxPolls || pipe_ns() - t0 > K.limit_ns) {
            atomicCAS(K.err, 0, 1 + ci);
            break;
        }
    }
    __threadfence();
}

// Rows that forward chunk c reads first: one thread waits for the chunk's moment units,
// then threads t = 0 .. nt-1 (barrier bar) assemble rho and J at each row's x position
// perm[k] and form its right-hand side as the unpipelined solve does
// (tmp[i] = (te * (charge[i] + neut[i])) * w, then x[k] = tmp[perm[k]]).  off_sp0: while
// warp 0 runs the sweep, the FP64 work stays off its sub-partition (warps 4m), whose FP64
// unit the sweep's dependent chain needs.
__device__ void pipe_rows(const PipeLaunch &K, int run, int c, double *x, int t, int nt, int bar, bool off_sp0) {
    if (t == 0) {
        if (K.trace && run == 0 && c == 0) K.trace[0] = pipe_ns();
        pipe_wait(K, K.run_ctr[run] + c);
        if (K.trace && run == 0) K.trace[1 + c] = pipe_ns();
    }
    pipe_bar(bar, nt);
    const int *gp = K.gptr + K.run_gptr[run];
    RunFields &F = K.P.fields[run];
    const int *perm = K.P.lu[run].perm;
    const double te = kEps0Inv;
    const double w = K.P.w[run];
    if (off_sp0) {  // warps 1..31 of the block: the 24 that are not 4m
        const int wg = (int)threadIdx.x >> 5;
        if ((wg & 3) == 0) return;
        t = ((wg >> 2) * 3 + (wg & 3) - 1) * 32 + ((int)threadIdx.x & 31);
        nt = 24 * 32;
    }
    for (int e = gp[c] + t; e < gp[c + 1]; e += nt) {
        const int k = K.grow[e], i = perm[k];
        assemble_cell<true>(K.A, run, i);
        const double v = te * (F.charge[i] + F.neut[i]);
        x[k] = v * w;
    }
}

// The solve with the solution vector x in shared memory (XS) or in phi itself.  The two
// instantiations let the compiler see x's address space: with one pointer chosen at run
// time its loads and stores in the sweeps go through generic addressing.
template <bool XS, bool PIPE>
__device__ __forceinline__ void poisson_solve(const PoissonLaunch &L, int run, unsigned char *smem_raw, double *x,
                                              const PipeLaunch *K) {
    PoisChunk *buf = (PoisChunk *)smem_raw;  // two chunk buffers, then the solution vector
    __shared__ int s_bad;
    __shared__ PoisTail s_tail;
    RunFields &F = L.fields[run];
    const LUDev &lu = L.lu[run];
    const int n = F.n;
    constexpr bool in_smem = XS;
    double *tmp = F.efin;  // scratch until E_x is recomputed at the end
    const double te = kEps0Inv;
    const double w = L.w[run];
    const bool fwd_chunks = PIPE || lu.L.nslots >= 0;
    if (fwd_chunks) pois_stage_fwd(buf[0].f, lu.L, 0, kPoisBuf, n, threadIdx.x, blockDim.x);  // needs no moments
    if (PIPE) {
        pipe_rows(*K, run, 0, x, threadIdx.x, blockDim.x, 0, false);  // chunk 0's rows, all threads
    } else {
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            double v = te * (F.charge[i] + F.neut[i]);
            tmp[i] = v * w;
        }
        __syncthreads();
        // Row interchanges of dgetrs applied as one gather: b'[k] = b[perm[k]].
        for (int k = threadIdx.x; k < n; k += blockDim.x) x[k] = tmp[lu.perm[k]];
    }
    const int nchunks = (n + kPoisRows - 1) / kPoisRows;
    unsigned long long *trace = (L.trace && run == 0 && threadIdx.x == 0) ? L.trace : nullptr;
    // clock64 (cycles) alone; globaltimer (ns) when pipelined, to compare with the moment units
    auto tick = [] { return PIPE ? pipe_ns() : (unsigned long long)clock64(); };
    if (trace) trace[0] = tick();
    if (PIPE && K->trace && run == 0 && threadIdx.x == 0) K->trace[1 + 2 * K->trace_nch] = clock64();
    const int lane = threadIdx.x & 31;
    // ---- forward: rows ascending; chunk c stages rows [c*R, c*R + R + LA)
    const int t0 = lu.U.sweep ? lu.U.far_pre_col : 0;
    const bool tail = t0 > 0;
    if (!fwd_chunks) {
        __syncthreads();
        if (threadIdx.x == 0) pois_rows_plain<false>(lu.L, 0, n, n, x, true);
        if (tail) {
            pois_stage_tail(s_tail, lu.U, t0, threadIdx.x);
            pois_stage_bwd(buf[nchunks & 1].b, lu.U, max(t0 - kPoisRows, 0), t0, threadIdx.x, blockDim.x);
        }
        __syncthreads();
    } else {
        double V = 0.0, w1 = 0.0;
        __syncthreads();
        if (threadIdx.x < 32 && lane < 4 && lane < n) V = pois_far(lu.L, x, lane);
        // warp 0 sweeps, the others stage the next chunk (pipelined: and gather its rows):
        // two loops with one block barrier per chunk each, so that the sweep's loop holds
        // only the sweep's values (the host pipelines only factors with accumulator lanes)
        if (threadIdx.x < 32) {
            for (int c = 0; c < nchunks; c++) {
                const int r0 = c * kPoisRows;
                pois_fwd_fast(buf[c & 1].f, lu.L, r0, min(kPoisRows, n - r0), n, x, V, w1);
                __syncthreads();
                if (trace) trace[1 + c] = tick();
            }
        } else {
            for (int c = 0; c + 1 < nchunks; c++) {
                const int r1 = (c + 1) * kPoisRows;
                pois_stage_fwd(buf[(c + 1) & 1].f, lu.L, r1, r1 + kPoisBuf, n, threadIdx.x - 32, blockDim.x - 32);
                // the rows chunk c+1 reads first, while warp 0 sweeps chunk c (it reads
                // and writes only rows first read by chunks up to c)
                if (PIPE) pipe_rows(*K, run, c + 1, x, threadIdx.x - 32, blockDim.x - 32, 1, true);
                __syncthreads();
            }
            if (tail) {  // beside the last chunk: what the backward sweep starts from
                pois_stage_tail(s_tail, lu.U, t0, threadIdx.x - 32);
                pois_stage_bwd(buf[nchunks & 1].b, lu.U, max(t0 - kPoisRows, 0), t0, threadIdx.x - 32, blockDim.x - 32);
            }
            __syncthreads();  // the last chunk's
        }
    }
    if (PIPE && K->trace && run == 0 && threadIdx.x == 0) K->trace[2 + 2 * K->trace_nch] = clock64();
    // ---- backward: the last rows (all of them, one by one, if their far columns reach
    // further down), then chunks of R rows, descending
    {
        if (!tail && threadIdx.x == 0) pois_rows_plain<true>(lu.U, 0, n, n, x, true);
        if (tail && threadIdx.x < 32) pois_tail(s_tail, lu.U, t0, x);
        if (threadIdx.x == 0) s_bad = 0;
        __syncthreads();
        // A neutral state leaves 0 everywhere: the rows are 0 / u_ii, and the sweep, whose FP32
        // term is wrong at 0, is not run (every chunk would be redone row by row: 6.7 ms instead
        // of 0.97 at n = 4096).
        bool some = false;
        for (int i = threadIdx.x; i < n; i += blockDim.x)
            some = some || (i < t0 ? __double_as_longlong(x[i]) != 0 : x[i] != 0.0);
        const bool sweep = __syncthreads_or(some);
        if (!sweep)
            for (int i = threadIdx.x; i < t0; i += blockDim.x) x[i] = copysign(0.0, lu.U.diag[i]);
        const int nbwd = sweep ? (t0 + kPoisRows - 1) / kPoisRows : 0;
        // chunk c's rows and buffer; the first chunk's factors are staged already
        auto first = [&](int c) { return max(t0 - (c + 1) * kPoisRows, 0); };
        auto rows = [&](int c) { return t0 - c * kPoisRows - first(c); };
        auto buffer = [&](int c) -> PoisBwdChunk & { return buf[(c + nchunks) & 1].b; };
        // every row of a swept chunk with IEEE division, from the rows above it
        auto check = [&](int c, int t, int nt) {
            const PoisBwdChunk &B = buffer(c);
            const int r0 = first(c), cnt = rows(c);
            for (int q = t; q < cnt; q += nt) {
                const double *xr = x + r0 + q;
                const int e = q + kPoisLA;
                double s = B.rhs[q] - xr[3] * B.c[2][e].x;
                s = s - xr[2] * B.c[1][e].x;
                s = s - xr[1] * B.c[0][e].x;
                if (__double_as_longlong(s / B.diag[q]) != __double_as_longlong(xr[0])) s_bad = 1;
            }
        };
        // chunk c in IEEE division, row by row
        auto redo = [&](int c) {
            const PoisBwdChunk &B = buffer(c);
            const int r0 = first(c), cnt = rows(c);
            for (int q = threadIdx.x; q < cnt; q += blockDim.x) x[r0 + q] = B.rhs[q];
            __syncthreads();
            if (threadIdx.x == 0) {
                pois_rows_plain<true>(lu.U, r0, r0 + cnt, n, x, false);
                s_bad = 0;
            }
            __syncthreads();
        };
        // FP64 work of the other warps stays off warp 0's sub-partition (warps 4m)
        const int wg = (int)threadIdx.x >> 5, others = (int)blockDim.x - 32;
        const int t2 = (wg & 3) == 0 ? -1 : ((wg >> 2) * 3 + (wg & 3) - 1) * 32 + lane;
        const int nt2 = ((int)blockDim.x >> 7) * 3 * 32;
        if (nbwd > 0) pois_rhs_bwd(buffer(0), lu.U, first(0), first(0) + rows(0), x, t2, nt2);
        __syncthreads();
        // While warp 0 sweeps chunk c, the others check chunk c - 1 and then, in the buffer that
        // leaves, stage chunk c + 1 (the check between the sweeps took 1.2 us of a chunk's 34).
        // A chunk that fails is redone, and the sweep of the next one, which began from it.
        int settled = -1;  // the last chunk done in IEEE division: not checked again
        for (int c = 0; c < nbwd; c++) {
            if (threadIdx.x < 32) {
                pois_bwd_fast(buffer(c), first(c), rows(c), x);
            } else {
                if (c > 0 && c - 1 != settled && t2 >= 0) check(c - 1, t2, nt2);
                pipe_bar(1, others);
                if (c + 1 < nbwd && !s_bad) {
                    pois_stage_bwd(buffer(c + 1), lu.U, first(c + 1), first(c), threadIdx.x - 32, others);
                    pois_rhs_bwd(buffer(c + 1), lu.U, first(c + 1), first(c), x, t2, nt2);
                }
            }
            __syncthreads();
            if (s_bad) {  // uniform
                __syncthreads();
                redo(c - 1);
                for (int q = threadIdx.x; q < rows(c); q += blockDim.x) x[first(c) + q] = buffer(c).rhs[q];
                __syncthreads();
                settled = --c;
                continue;
            }
            if (trace) trace[1 + nchunks + c] = tick();
        }
        if (nbwd > 0) {
            check(nbwd - 1, threadIdx.x, blockDim.x);
            __syncthreads();
            if (s_bad) {
                __syncthreads();
                redo(nbwd - 1);
            }
        }
        if (trace)
            for (int c = nbwd; c < nchunks; c++) trace[1 + nchunks + c] = tick();
    }
    if (in_smem)
        for (int i = threadIdx.x; i < n; i += blockDim.x) F.phi[i] = x[i];
    if (threadIdx.x == 0) {
        double ex0 = *F.ex0;
        double e_m1 = efield_at(x, n, L.fcoef[run], ex0, -1);
        double e_0 = efield_at(x, n, L.fcoef[run], ex0, 0);
        *F.ex0 = ex0 + -(e_m1 + e_0) * 0.5;
    }
    __syncthreads();
    const double ex0 = *F.ex0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) F.efin[i] = efield_at(x, n, L.fcoef[run], ex0, i);
}

__global__ void __launch_bounds__(1024, 1) k_poisson(PoissonLaunch L) {
    VX_PDL_WAIT();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int run = blockIdx.x;
    if (L.x_in_smem) poisson_solve<true, false>(L, run, smem_raw, (double *)(smem_raw + 2 * sizeof(PoisChunk)), nullptr);
    else poisson_solve<false, false>(L, run, smem_raw, L.fields[run].phi, nullptr);
}

// ---- workers of the pipelined launch
// One item: column warp wid forms window j0 of its column's sub-columns k0, k0+1 (those
// the patch has) and writes the contributions of lanes 1 .. kMomOut to `out`.
template <bool FAST>
__device__ __forceinline__ void mom_item(const PipeLaunch &K, int u, int k0, int j0, int wid, int lane, double *out) {
    const MomLaunch &M = K.M;
    const int col0 = K.unit_col0[u];
    const bool real = M.colpatch[col0 + wid] >= 0;  // warp-uniform
    const P64 &P = ((const P64 *)M.patches)[M.colpatch[col0]];
    const int rtb = P.rtb;
    const int i = M.colidx[col0 + wid] / rtb;
    const RunFields &F = M.fields[P.run];
    const double2 c12 = K.unit_c12[u];
    const int kg = rtb - k0 < 2 ? rtb - k0 : 2;
    double a[2] = {0.0, 0.0};
    for (int q = 0; q < kg; q++)
        if (real) a[q] = P.qq * cell_asq(F, (i + P.x_pos) * rtb + k0 + q);
    double cc[2], cj[2];
    bool use;
    mom_window<FAST>(P, P.f1, real, i, j0, k0, kg, a, c12.x, c12.y, lane, cc, cj, use);
    if (lane >= 1 && lane <= kMomOut)
        for (int q = 0; q < kg; q++) {
            out[lane * 30 + wid * 2 + q] = cc[q];
            out[960 + lane * 30 + wid * 2 + q] = cj[q];
        }
}

// The windows of unit u that the screen left out, formed by one warp (rare: see MomSum).
template <bool FAST>
__device__ __noinline__ void mom_form_rest(const PipeLaunch &K, int u, int k0, int lane) {
    const unsigned *screen = K.M.screen + (size_t)(K.unit_col0[u] / kMomCols) * K.M.maxnwin * kMomScreen;
    const int nw = K.unit_nwin[u];
    for (int win = 0; win < nw; win++) {
        if (screen[win * kMomScreen + kMomCols]) continue;
        double *out = K.scratch + (size_t)(K.unit_item0[u] + (k0 / 2) * nw + win) * kPipeItemDoubles;
        for (int wid = 0; wid < kMomCols; wid++) mom_item<FAST>(K, u, k0, win * kMomOut, wid, lane, out);
    }
    __threadfence();
    __syncwarp();
}

// The column sums of unit u (one warp, lanes as MomLane has them): every formed window's
// contributions in ascending p.  A cell that is not used contributes +0.0, which leaves a
// sum that starts at +0.0 unchanged bit for bit (such a sum never becomes -0.0), so these
// are the sums of the used cells alone.  Then the unit counts as done for its chunk.
template <bool FAST>
__device__ __forceinline__ void mom_sum_unit(const PipeLaunch &K, int u, int lane) {
    const unsigned full = 0xffffffffu;
    const MomLaunch &M = K.M;
    const int col0 = K.unit_col0[u];
    const P64 &P = ((const P64 *)M.patches)[M.colpatch[col0]];
    const unsigned *screen = M.screen + (size_t)(col0 / kMomCols) * M.maxnwin * kMomScreen;
    const int rtb = P.rtb, nw = K.unit_nwin[u];
    for (int k0 = 0; k0 < rtb; k0 += 2) {
        const int kg = rtb - k0 < 2 ? rtb - k0 : 2;
        const MomLane ml(P, kg, lane);
        for (int pass = 0; pass < 2; pass++) {
            const double *src = K.scratch + (size_t)(K.unit_item0[u] + (k0 / 2) * nw) * kPipeItemDoubles +
                                (ml.cur ? 960 : 0) + ml.w * 2 + ml.q;
            MomSum s;
            for (int win = 0; win < nw; win++, src += kPipeItemDoubles) {
                if (pass || screen[win * kMomScreen + kMomCols]) {
                    s.add(__any_sync(full, s.split()), ml.two, [&](int t) { return __ldcg(src + t * 30); },
                          [&](int t) { return __ldcg(src + 960 + t * 30); });
                } else {
                    const double b = __hiloint2double((int)screen[win * kMomScreen + ml.w], 0);
                    MomSum::widen(s.lo0, s.hi0, b * ml.f0);
                    MomSum::widen(s.lo1, s.hi1, b * ml.f1);
                }
            }
            if (!pass && __any_sync(full, ml.on && M.colpatch[col0 + ml.w] >= 0 && s.split())) {
                mom_form_rest<FAST>(K, u, k0, lane);
                continue;
            }
            ml.store(M, P, col0, k0, s);
            break;
        }
    }
    __threadfence();  // the column sums, device-wide, before the count
    __syncwarp();
    if (lane == 0) {
        atomicAdd(K.state + kPipeDone + K.unit_sig[u], 1u);
        if (K.trace && K.unit_sig[u] < K.trace_nch) atomicMax(K.trace + 1 + K.trace_nch + K.unit_sig[u], pipe_ns());
    }
}

// A group of a worker block: kPipeCols column warps take parts of items until none are
// left; the warp that completes a unit (its part count reaches its total) appends the unit
// to the queue of completed units.  They never wait for anything but each other.
template <bool FAST>
__device__ void pipe_columns(const PipeLaunch &K, int *ticket, int g, int tid) {
    const int wid = tid >> 5, lane = tid & 31;
    const int bar = 1 + g, ncol = kPipeCols * 32, nparts = K.nitems * kPipeParts;
    unsigned *items_done = K.state + kPipeDone + K.ndone;      // per unit
    unsigned *queue = items_done + K.nunits;                    // completed units (u + 1), in order
    // a part of unit u is done: the last one queues the unit
    auto count = [&](int u) {
        const unsigned total = (unsigned)(K.unit_item0[u + 1] - K.unit_item0[u]) * kPipeParts;
        if (atomicAdd(items_done + u, 1u) + 1 == total) {
            __threadfence();  // every item's contributions before a summing warp reads them
            const unsigned slot = atomicAdd(K.state + kPipeQHead, 1u);
            atomicExch(queue + slot, (unsigned)u + 1);
        }
    };
    auto window = [&](int t, int u, int &kp) {
        const int loc = t - K.unit_item0[u], nw = K.unit_nwin[u];
        kp = loc / nw;
        return loc - kp * nw;
    };
    for (int it = 0;; it++) {
        if (tid == 0) {  // the next item whose window is formed
            int t;
            for (;;) {
                t = (int)atomicAdd(K.state + kPipeTicket, 1u);
                if (t >= nparts) break;
                const int u = K.item_unit[t / kPipeParts];
                int kp;
                const int w = window(t / kPipeParts, u, kp);
                if (K.M.screen[((size_t)(K.unit_col0[u] / kMomCols) * K.M.maxnwin + w) * kMomScreen + kMomCols]) break;
                count(u);
            }
            ticket[it & 1] = t;
        }
        pipe_bar(bar, ncol);
        const int tk = ticket[it & 1];
        if (tk >= nparts) break;
        const int t = tk / kPipeParts, c = (tk - t * kPipeParts) * kPipeCols + wid;
        const int u = K.item_unit[t];
        int kp;
        const int w = window(t, u, kp);
        if (c < kMomCols) mom_item<FAST>(K, u, 2 * kp, w * kMomOut, c, lane, K.scratch + (size_t)t * kPipeItemDoubles);
        __threadfence();  // this warp's contributions, device-wide, before the item counts
        pipe_bar(bar, ncol);
        if (tid == 0) count(u);
    }
}

// A summing warp (one per sub-partition of a summing block, so that its serial adds have
// the sub-partition's FP64 unit to themselves): takes completed units from the queue in
// order and forms their column sums.  It waits only for units, which the column warps
// always complete; a wait that runs out records itself and ends the warp.
template <bool FAST>
__device__ void pipe_summer(const PipeLaunch &K, int lane) {
    const unsigned full = 0xffffffffu;
    unsigned *queue = K.state + kPipeDone + K.ndone + K.nunits;
    for (;;) {
        int slot = 0;
        if (lane == 0) slot = (int)atomicAdd(K.state + kPipeQTail, 1u);
        slot = __shfl_sync(full, slot, 0);
        if (slot >= K.nunits) break;
        unsigned v = 0;
        if (lane == 0) {
            v = pipe_ld_acquire(queue + slot);
            if (!v) {
                const unsigned long long t0 = pipe_ns();
                for (unsigned poll = 0;; poll++) {
                    __nanosleep(64);
                    v = pipe_ld_acquire(queue + slot);
                    if (v) break;
                    if ((poll & 63u) == 63u && pipe_ld_relaxed(K.err) != 0) break;
                    if (poll >= kPipeMaxPolls || pipe_ns() - t0 > K.limit_ns) {
                        atomicCAS(K.err, 0, 1 + K.ndone);
                        break;
                    }
                }
            }
        }
        v = __shfl_sync(full, v, 0);
        if (!v) break;
        __threadfence();
        mom_sum_unit<FAST>(K, (int)v - 1, lane);
    }
}

// Moments, assembly and the exact solve in one launch, a block per SM.  A block solves one run
// (its forward sweep starts as soon as the moments of its first rows are summed, instead of
// after the whole moments kernel), carries four summing warps (pipe_summer), or up to
// kPipeGroups groups of column warps (pipe_columns).  Column warps wait for nothing outside
// their group, summing warps only for column warps, the solve only for summing warps; the
// blocks' order (pipe_block) lets every wait end on any number of SMs.  Same arithmetic as
// k64_moments + k_assemble + k_poisson.
// The fast form's workers are called, the exact form's inlined: the kernel has 64 registers a
// thread, and which way the sweeps keep theirs differs between the two (4096 x 512 in two
// levels per step: fast 13.64 ms inlined, 13.42 called; exact 13.78 and 14.29).
template <bool FAST>
__device__ __noinline__ void pipe_columns_call(const PipeLaunch &K, int *ticket, int g, int tid) {
    pipe_columns<FAST>(K, ticket, g, tid);
}
template <bool FAST>
__device__ __noinline__ void pipe_summer_call(const PipeLaunch &K, int lane) {
    pipe_summer<FAST>(K, lane);
}
template <bool FAST>
__global__ void __launch_bounds__(1024, 1) k64_moments_poisson(PipeLaunch K) {
    VX_PDL_WAIT();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const PipeBlock me = pipe_block((int)blockIdx.x, K.P.nruns, K.summers);
    if (me.role == kPipeSolver) {
        if (K.P.x_in_smem)
            poisson_solve<true, true>(K.P, me.run, smem_raw, (double *)(smem_raw + 2 * sizeof(PoisChunk)), &K);
        else poisson_solve<false, true>(K.P, me.run, smem_raw, K.P.fields[me.run].phi, &K);
    } else if (me.role == kPipeSummer) {
        if (threadIdx.x < 4 * 32) {  // warps 0..3: one per sub-partition
            if constexpr (FAST) pipe_summer_call<FAST>(K, (int)threadIdx.x & 31);
            else pipe_summer<FAST>(K, (int)threadIdx.x & 31);
        }
    } else {
        int *ticket = reinterpret_cast<int *>(smem_raw);
        const int g = (int)threadIdx.x / (kPipeCols * 32);
        const int tid = (int)threadIdx.x - g * kPipeCols * 32;
        if (g < K.groups) {
            if constexpr (FAST) pipe_columns_call<FAST>(K, ticket + 2 * g, g, tid);
            else pipe_columns<FAST>(K, ticket + 2 * g, g, tid);
        }
    }
    // the last block out zeroes the tickets, the queue, done and item counters for the next launch
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(K.state + kPipeLeave, 1u) + 1 == gridDim.x) {
            atomicExch(K.state + kPipeTicket, 0u);
            atomicExch(K.state + kPipeQHead, 0u);
            atomicExch(K.state + kPipeQTail, 0u);
            for (int i = 0; i < K.ndone + 2 * K.nunits; i++) atomicExch(K.state + kPipeDone + i, 0u);
            atomicExch(K.state + kPipeLeave, 0u);
            __threadfence();
        }
    }
}

void launch_poisson(const PoissonLaunch &L) {
    PoissonLaunch P = L;
    int max_smem = 0, dev = 0;  // per call: engines on several host threads may launch
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    // the solution vector joins the two chunk buffers in shared memory when it fits
    const int base = 2 * (int)sizeof(PoisChunk);
    P.x_in_smem = (L.maxn <= kPoisSmemMaxN && base + 8 * L.maxn <= max_smem) ? 1 : 0;
    const int smem = base + (P.x_in_smem ? 8 * L.maxn : 0);
    vx_allow_smem(k_poisson);
    // 1024 threads x 64 registers take a whole SM's register file: no block of the FP64
    // face kernels that run beside the solve shares the SM, whose FP64 unit would
    // otherwise delay the solve's dependent chain (step 32.4 -> 28.1 ms on 4096 x 512)
    vx_launch(k_poisson, L.nruns, 1024, smem, L.stream, P);
}

void launch_moments_poisson64(const PipeLaunch &K0) {
    PipeLaunch K = K0;
    int max_smem = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const int base = 2 * (int)sizeof(PoisChunk);
    K.P.x_in_smem = (K.P.maxn <= kPoisSmemMaxN && base + 8 * K.P.maxn <= max_smem) ? 1 : 0;
    const int smem_solve = base + (K.P.x_in_smem ? 8 * K.P.maxn : 0);
    const int smem = std::max(smem_solve, 2 * (int)sizeof(int) * kPipeGroups);
    auto kern = K.M.fast ? k64_moments_poisson<true> : k64_moments_poisson<false>;
    vx_allow_smem(kern);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(K.P.nruns + K.summers + K.workers);
    cfg.blockDim = dim3(1024);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = K.stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributePriority;
    attr[0].val.priority = K.priority;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_launch_pdl ? 2 : 1;
    cudaLaunchKernelEx(&cfg, kern, K);  // errors surface through cudaGetLastError
}

// E_x on the finest grid from phi and Ex0 (EMSolver::GetEfield), for states loaded from
// outside the step.
__global__ void k_efield(RunFields *fields, const double *fcoef, int nruns, int f32) {
    VX_PDL_WAIT();
    const int run = blockIdx.y;
    if (run >= nruns) return;
    RunFields &F = fields[run];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= F.n) return;
    const double e = efield_at(F.phi, F.n, fcoef[run], *F.ex0, i);
    F.efin[i] = e;
    if (f32) F.efin32[i] = (float)e;
}

void launch_efield(RunFields *fields, const double *fcoef, int nruns, int maxn, int f32, cudaStream_t s) {
    dim3 g((maxn + 255) / 256, nruns);
    vx_launch(k_efield, g, 256, 0, s, fields, fcoef, nruns, f32);
}

// ---------------------------------------------------------------- Maxwell
// FP64 runs; runs of the FP32 form go to launch_maxwell32 (stage32.cu).
__global__ void k_mx_rhs(MaxwellLaunch L) {
    VX_PDL_WAIT();
    const int run = blockIdx.y;
    if (run >= L.nruns) return;
    mx_rhs_cell(L, run, blockIdx.x * blockDim.x + threadIdx.x, blockIdx.z);
}
__global__ void k_mx_update(MaxwellLaunch L) {
    VX_PDL_WAIT();
    const int run = blockIdx.y;
    if (run >= L.nruns) return;
    mx_update_cell(L, run, blockIdx.x * blockDim.x + threadIdx.x, blockIdx.z);
}
__global__ void k_mx_asq(MaxwellLaunch L) {
    VX_PDL_WAIT();
    const int run = blockIdx.y;
    if (run >= L.nruns) return;
    mx_asq_pair(L, run, blockIdx.x * blockDim.x + threadIdx.x);
}

void launch_maxwell(const MaxwellLaunch &L) {
    if (L.f32) {
        launch_maxwell32(L);
        return;
    }
    const dim3 g((L.maxnf + kMxThreads - 1) / kMxThreads, L.nruns, kMxFields);
    vx_launch(k_mx_rhs, g, kMxThreads, 0, L.stream, L);
    vx_launch(k_mx_update, g, kMxThreads, 0, L.stream, L);
    vx_launch(k_mx_asq, dim3((2 * L.maxnf + kMxThreads - 1) / kMxThreads, L.nruns), kMxThreads, 0, L.stream, L);
}

// ---------------------------------------------------------------- CFL
// The maximum runs over non-negative doubles, so it is taken on their bit patterns:
// each block reduces its slice and folds it into out[run] with an integer atomicMax.
__global__ void k_cfl(CflLaunch L) {
    VX_PDL_WAIT();
    const int run = blockIdx.y;
    const RunFields &F = L.fields[run];
    const int ns = L.run_ns[run];
    const double *sp = L.spec + run * 25;  // up to 8 species x 3 + dpsMax
    const double dpsMax = sp[24];
    __shared__ double red[256];
    double pc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < F.n; i += gridDim.x * blockDim.x) {
        double Azv = F.Az[i], Ayv = F.Ay[i];
        double As = Ayv * Ayv + Azv * Azv;
        double temp = 0.0;
        for (int j = 0; j < ns; j++) {
            double aq = sp[3 * j], m = sp[3 * j + 1], dps = sp[3 * j + 2];
            double v = aq / m / sqrt(1 + As / ((m * kCs) * (m * kCs))) * dps;
            temp = (temp < v) ? v : temp;
        }
        double v = temp * fabs(Ayv * F.Bz[i] - Azv * F.By[i]) + dpsMax * fabs(F.efin[i]);
        pc = (pc < v) ? v : pc;
    }
    red[threadIdx.x] = pc;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) {
            double o = red[threadIdx.x + s];
            red[threadIdx.x] = (red[threadIdx.x] < o) ? o : red[threadIdx.x];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
        atomicMax((unsigned long long *)&L.out[run], (unsigned long long)__double_as_longlong(red[0]));
}

void launch_cfl(const CflLaunch &L) {
    cudaMemsetAsync(L.out, 0, (size_t)L.nruns * sizeof(double), L.stream);
    dim3 g(std::min(32, std::max(1, (L.maxn + 255) / 256)), L.nruns);
    vx_launch(k_cfl, g, 256, 0, L.stream, L);
}

__global__ void k_negate(double *dst, const double *src, int n) {
    VX_PDL_WAIT();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = -src[i];
}

void launch_negate(double *dst, const double *src, int n, cudaStream_t s) {
    vx_launch(k_negate, (n + 255) / 256, 256, 0, s, dst, src, n);
}

}  // namespace vx

namespace vx {
// Eight independent fused multiply-add chains per thread (register resident).  The
// result is stored so the chains are not eliminated.
__global__ void k_fp64_peak(double *out, int iters) {
    VX_PDL_WAIT();
    double a0 = threadIdx.x * 1e-9, a1 = a0 + 1e-9, a2 = a0 + 2e-9, a3 = a0 + 3e-9;
    double a4 = a0 + 4e-9, a5 = a0 + 5e-9, a6 = a0 + 6e-9, a7 = a0 + 7e-9;
    const double b = 0.999999, c = 1e-7;
    for (int k = 0; k < iters; k++) {
        a0 = fma(a0, b, c);
        a1 = fma(a1, b, c);
        a2 = fma(a2, b, c);
        a3 = fma(a3, b, c);
        a4 = fma(a4, b, c);
        a5 = fma(a5, b, c);
        a6 = fma(a6, b, c);
        a7 = fma(a7, b, c);
    }
    out[blockIdx.x * blockDim.x + threadIdx.x] = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
}

void launch_fp64_peak(double *out, int blocks, int threads, int iters, cudaStream_t s) {
    vx_launch(k_fp64_peak, blocks, threads, 0, s, out, iters);
}

// Dependent-chain latency on one lane: iters steps of the substitution's multiply-
// subtract, then the same with a 64-bit shuffle in the chain (clock64 cycles, into
// cyc[0] and cyc[1]; the chains' values into val so that they are not eliminated).
__global__ void k_fp64_latency(long long *cyc, double *val, int iters) {
    VX_PDL_WAIT();
    double x = 1.0 + threadIdx.x * 1e-3;
    const double c = 0.999999, v = 1e-7;
    long long t0 = clock64();
    for (int k = 0; k < iters; k++) x = v - x * c;
    long long t1 = clock64();
    double y = x;
    for (int k = 0; k < iters; k++) {
        y = v - y * c;
        y = __shfl_sync(0xffffffffu, y, 0);
    }
    long long t2 = clock64();
    if (threadIdx.x == 0) {
        cyc[0] = t1 - t0;
        cyc[1] = t2 - t1;
        val[0] = x + y;
    }
}

void launch_fp64_latency(long long *cyc, double *val, int iters, cudaStream_t s) {
    vx_launch(k_fp64_latency, 1, 32, 0, s, cyc, val, iters);
}
}  // namespace vx
