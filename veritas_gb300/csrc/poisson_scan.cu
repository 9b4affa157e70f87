// O(n) Poisson solve by prefix scans (EMFieldSolver::UpdatePotential,
// EMSolver.cpp:156-192): used by the FP32 precision form and, on request, by FP64 runs.
//
// The reference's LU solve sees M = P^T, P its row-major stencil matrix (EMSolver.cpp:
// 41-67).  Column 0 of M is e_0, so M = [[1, r^T], [0, B]]: phi[1:] = B^{-1} b[1:] and
// phi_0 = b_0 - (w1 phi_1 + w2 phi_2 + w2 phi_{n-2} + w1 phi_{n-1}).  B (m = n-1) is the
// pentadiagonal Toeplitz stencil T = (w2, w1, w3, w1, w2) plus the corner pair
// w2 (e_0 e_{m-1}^T + e_{m-1} e_0^T).  The stencil's symbol has the roots 1, 1, rho, 1/rho
// (rho = 7 - 4 sqrt 3), so T = c G G^T + (a 2x2 block at the top left) with
// G = (I - S)(I - rho S), c = w2 / rho.  Hence
//   B^{-1} v = z - Y K (z_0, z_1, z_{m-1}),   z = (1/c) G^{-T} G^{-1} v,
// with Y = (1/c) G^{-T} G^{-1} [e_0 e_1 e_{m-1}] and the 3x3 K precomputed on the host
// (Woodbury, poisson_fast.cpp).  G^{-1} and G^{-T} are two prefix sums and two decaying
// first-order recurrences.
//
// One thread-block cluster per run: the kPsCluster blocks of a cluster hold consecutive
// chunks of the vector in shared memory (T segments of L elements each, stored
// segment-minor so that a warp's threads walk their segments on different banks).  A
// pass runs every segment serially; its carry — the prefix sum of the preceding segment
// sums (a block scan plus the preceding blocks' totals read through distributed shared
// memory), or for the decaying recurrences the sum over preceding segment ends weighted by
// rho^{L (q-1)}, which drops below 1e-20 after a few segments (three for L >= 8, which the
// block size is chosen for) — is added as the next pass runs.  The cluster barriers are
// hardware barriers of co-scheduled blocks.
//
// FP64 throughout, with fused multiply-adds (E_x itself comes from k_efield, which keeps
// the reference's rounding).  The result is not the LU's rounding order; both have the
// error the discrete system's conditioning (~n^2) allows, about 1e-11 relative at
// n = 2048 and 1e-9 at n = 8192 against the exact solution.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <utility>

#include "field_ops.cuh"
#include "vx_kernels.hpp"

namespace vx {

namespace {

namespace cg = cooperative_groups;

constexpr int kPsMaxTerms = 24;  // carry-gather terms of a decaying pass (rho^24 < 1e-27)
constexpr int kPsGather = 4;     // of them, loaded together
// Threads beyond the T of the scans: they share the element-wise work (an FP64 instruction
// of a warp takes about 64 cycles of its sub-partition, so a block of one warp would use a
// quarter of the SM's units), and the last warp forms the values at the vector's ends.
constexpr int kPsMinThreads = 128;

// Per-block scratch of the passes.  Each pass has its own cells for what other blocks read
// (sa, s_tot), so that no cluster barrier is needed before the next pass writes.
struct ScanScratch {
    double sa[2][kPsMaxThreads];  // decaying passes: segment ends without carry (read across the cluster)
    double s_tot[2];              // prefix sums: block totals (read across the cluster)
    double sb[32];                // warp totals
    double pw[kPsMaxSeg];         // rho^(s+1)
    double wt[kPsMaxTerms];       // rho^(L q) carry weights
    double s_pre;                 // preceding blocks' totals
    int nterms;                   // carry terms of a decaying pass
};

// Carry into thread tid's segment of a prefix-sum pass: the preceding blocks' totals in scan
// order, plus the block's exclusive scan (thread order) of the segment sums y.
template <bool REV>
__device__ double sum_carry(cg::cluster_group &cl, ScanScratch &W, int T, double y) {
    const unsigned full = 0xffffffffu;
    constexpr int C = kPsCluster;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = T >> 5;
    const int rank = (int)cl.block_rank(), cpos = REV ? C - 1 - rank : rank;
    double x = y;
    if (wid < nw) {
        for (int o = 1; o < 32; o <<= 1) {
            const double p = __shfl_up_sync(full, x, o);
            if (lane >= o) x = x + p;
        }
        if (lane == 31) W.sb[wid] = x;
    }
    if (nw > 1) {
        __syncthreads();
        if (wid == 0) {
            double w = (lane < nw) ? W.sb[lane] : 0.0;
            for (int o = 1; o < nw; o <<= 1) {
                const double p = __shfl_up_sync(full, w, o);
                if (lane >= o) w = w + p;
            }
            W.sb[lane] = w;
            if (lane == nw - 1) W.s_tot[REV] = w;
        }
        __syncthreads();
    } else if (tid == 31) {
        W.s_tot[REV] = x;
    }
    auto arrival = cl.barrier_arrive();
    double ex = 0.0;
    if (wid < nw) {
        ex = __shfl_up_sync(full, x, 1);
        if (lane == 0) ex = 0.0;
        if (wid > 0) ex = W.sb[wid - 1] + ex;
    }
    cl.barrier_wait(std::move(arrival));
    if (tid == 0) {
        double v[C - 1];
#pragma unroll
        for (int q = 0; q < C - 1; q++) v[q] = q < cpos ? cl.map_shared_rank(W.s_tot, REV ? C - 1 - q : q)[REV] : 0.0;
        double pre = 0.0;
#pragma unroll
        for (int q = 0; q < C - 1; q++)
            if (q < cpos) pre = pre + v[q];
        W.s_pre = pre;
    }
    __syncthreads();
    return W.s_pre + ex;
}

// Carry into thread tid's segment of a decaying pass, from the segment ends y:
// sum_q rho^{L (q-1)} y_end(sp - q), terms below 1e-20 relative dropped.
template <bool REV>
__device__ double decay_carry(cg::cluster_group &cl, ScanScratch &W, int T, double y) {
    constexpr int C = kPsCluster;
    const int tid = threadIdx.x, rank = (int)cl.block_rank();
    if (tid < T) W.sa[REV][tid] = y;
    cl.sync();
    double carry = 0.0;
    if (tid < T) {
        const int sp = (REV ? C - 1 - rank : rank) * T + tid, nq = min(W.nterms, sp);
        for (int q0 = 1; q0 <= nq; q0 += kPsGather) {  // the remote reads of a group in flight together
            double v[kPsGather];
#pragma unroll
            for (int k = 0; k < kPsGather; k++) {
                const int src = sp - q0 - k;
                v[k] = q0 + k <= nq ? cl.map_shared_rank(W.sa[REV], REV ? C - 1 - src / T : src / T)[src % T] : 0.0;
            }
#pragma unroll
            for (int k = 0; k < kPsGather; k++)
                if (q0 + k <= nq) carry = carry + W.wt[q0 + k - 1] * v[k];
        }
    }
    return carry;
}

// phi of unknown g from its element of (c z) and the Woodbury coefficients t.
__device__ __forceinline__ double phi_value(const PoissonFastDev &D, int g, double v, const double t[3]) {
    const double z = v * D.c_inv;
    return z - (D.Y[3 * g] * t[0] + D.Y[3 * g + 1] * t[1] + D.Y[3 * g + 2] * t[2]);
}

// With P.assemble the launch forms rho and J from the moments too (one cell per thread),
// instead of a launch of its own before it.  Six cluster barriers: one per pass for its
// carries, one before the Woodbury entries are read, one before phi replaces the vector.
// The solve is latency from end to end (the FP64 units are idle most of the time): 13.4 us
// at n = 1062 and 22.7 us at n = 8192, against 21.4 and 26.9 us with eleven barriers, the
// remote reads one at a time and E_x read back from global memory.
__global__ void __cluster_dims__(kPsCluster, 1, 1) __launch_bounds__(kPsMaxThreads + 32)
    k_poisson_scan(PoissonFastLaunch P) {
    VX_PDL_WAIT();
    extern __shared__ double xs[];  // [L][T + 1]: element (segment s, offset o) at o (T + 1) + s
    __shared__ ScanScratch W;
    __shared__ double s_halo[4], s_phi0, s_ex0;
    cg::cluster_group cl = cg::this_cluster();
    const unsigned full = 0xffffffffu;
    const int T = P.scan_threads, NT = blockDim.x, stride = T + 1, tid = threadIdx.x;
    const int run = blockIdx.x / kPsCluster;
    const int rank = (int)cl.block_rank();
    RunFields &F = P.fields[run];
    const PoissonFastDev &D = P.pf[run];
    const int n = F.n, m = n - 1;
    const int L = (m + T * kPsCluster - 1) / (T * kPsCluster);
    const int g0 = rank * T * L;  // first unknown of this block's chunk
    const int cnt = max(0, min(T * L, m - g0));
    const double rho = D.rho;
    // right-hand side (dx^2 / eps0) (rho + rho_neutral), x_k = b_{k+1}
    const double te = kEps0Inv, w = P.w[run];
    for (int l = tid; l < cnt; l += NT) {
        if (P.assemble) assemble_cell(P.A, run, g0 + l + 1);
        const double r = te * (F.charge[g0 + l + 1] + F.neut[g0 + l + 1]);
        xs[(l % L) * stride + l / L] = r * w;
    }
    const bool ends = tid >= NT - 32;  // the last warp: the values at the ends of the vector
    const int lane = tid & 31;
    double b0 = 0.0, ex_old = 0.0;
    if (ends) {
        if (P.assemble && lane == 0) assemble_cell(P.A, run, 0);  // every block: the same values
        __syncwarp();
        const double r0 = te * (F.charge[0] + F.neut[0]);
        b0 = r0 * w;
        ex_old = *F.ex0;  // rewritten after the last barrier
    }
    if (tid == NT - 32) {  // powers by repeated products (a library pow is a long FP64 chain here)
        double x = rho;
        for (int q = 0; q < L; q++) {
            W.pw[q] = x;
            x = x * rho;
        }
        const double aL = W.pw[L - 1];
        x = 1.0;
        int q = 0;
        while (q < kPsMaxTerms && x > 1e-20) {
            W.wt[q++] = x;
            x = x * aL;
        }
        W.nterms = q;
    }
    __syncthreads();
    // Thread t < T owns segment t, in the descending passes segment T - 1 - t, so that thread
    // order is scan order either way; blocks are in scan order by rank.  Segments past the
    // end of the vector are short or empty; in scan order they come last (descending:
    // first), so no full-length weight ever crosses one.
    {  // (I - S)^{-1}, then (I - rho S)^{-1}, ascending
        double *seg = xs + tid;
        const int len = tid < T ? max(0, min(L, cnt - tid * L)) : 0;
        double y = 0.0;
        for (int s = 0; s < len; s++) {
            y = seg[s * stride] + y;
            seg[s * stride] = y;
        }
        const double c1 = sum_carry<false>(cl, W, T, y);
        y = 0.0;
        for (int s = 0; s < len; s++) {
            const double v = seg[s * stride] + c1;
            y = v + rho * y;
            seg[s * stride] = y;
        }
        const double c2 = decay_carry<false>(cl, W, T, y);
        for (int s = 0; s < len; s++) seg[s * stride] = seg[s * stride] + W.pw[s] * c2;
    }
    __syncthreads();
    {  // (I - rho S^T)^{-1}, then (I - S^T)^{-1}, descending
        double *seg = xs + (T - 1 - tid);
        const int len = tid < T ? max(0, min(L, cnt - (T - 1 - tid) * L)) : 0;
        double y = 0.0;
        for (int s = len - 1; s >= 0; s--) {
            y = seg[s * stride] + rho * y;
            seg[s * stride] = y;
        }
        const double c1 = decay_carry<true>(cl, W, T, y);
        y = 0.0;
        for (int s = len - 1; s >= 0; s--) {
            const double v = seg[s * stride] + W.pw[len - 1 - s] * c1;
            y = v + y;
            seg[s * stride] = y;
        }
        const double c2 = sum_carry<true>(cl, W, T, y);
        for (int s = len - 1; s >= 0; s--) seg[s * stride] = seg[s * stride] + c2;
    }
    cl.sync();  // every chunk final
    // the element of unknown g, from the block that holds it
    auto remote = [&](int g) {
        const int r = g / (T * L), l = g - r * T * L;
        return cl.map_shared_rank(xs, r)[(l % L) * stride + l / L];
    };
    // The block's cells: phi index p0 .. p1-1 (block 0 holds phi_0 too).
    const int p0 = rank == 0 ? 0 : g0 + 1, p1 = g0 + cnt + 1;
    double u[3];
#pragma unroll
    for (int k = 0; k < 3; k++) u[k] = remote(k == 2 ? m - 1 : k);
    // The last warp's lanes: phi at 1, 2, n - 3, n - 2, n - 1 (phi_0 and Ex0 come from them)
    // and at the two cells on either side of the block's (a block without cells has no sides:
    // its bounds lie past the vector's end).
    const int nends = cnt > 0 ? 9 : 5;
    int pe = 0;  // 0 .. n - 1
    double ve = 0.0;
    if (ends && lane < nends) {
        pe = lane < 2 ? lane + 1 : lane < 5 ? n - 5 + lane : lane < 7 ? p0 - 7 + lane : p1 - 7 + lane;
        pe = pe < 0 ? pe + n : pe >= n ? pe - n : pe;
        if (pe > 0) ve = remote(pe - 1);
    }
    auto arrival = cl.barrier_arrive();
    double t[3];
    for (int r = 0; r < 3; r++) {
        const double s0 = u[0] * D.c_inv, s1 = u[1] * D.c_inv, s2 = u[2] * D.c_inv;
        t[r] = D.K[3 * r] * s0 + D.K[3 * r + 1] * s1 + D.K[3 * r + 2] * s2;
    }
    const double fc = P.fcoef[run];
    double ex0 = 0.0;
    if (ends) {
        double ph = (lane < nends && pe > 0) ? phi_value(D, pe - 1, ve, t) : 0.0;
        const double q1 = __shfl_sync(full, ph, 0), q2 = __shfl_sync(full, ph, 1), z3 = __shfl_sync(full, ph, 2),
                     z2 = __shfl_sync(full, ph, 3), z1 = __shfl_sync(full, ph, 4);
        const double phi0 = b0 - (D.w1 * q1 + D.w2 * q2 + D.w2 * z2 + D.w1 * z1);
        const double e_m1 = -fc * (8 * (phi0 - z2) - q1 + z3) + ex_old;
        const double e_0 = -fc * (8 * (q1 - z1) - q2 + z2) + ex_old;
        ex0 = ex_old + -(e_m1 + e_0) * 0.5;
        if (lane >= 5 && lane < 9) s_halo[lane - 5] = pe > 0 ? ph : phi0;
        if (lane == 0) {
            s_phi0 = phi0;
            s_ex0 = ex0;
        }
    }
    cl.barrier_wait(std::move(arrival));  // no block reads another's vector any more
    for (int l = tid; l < cnt; l += NT) {
        double *p = &xs[(l % L) * stride + l / L];
        const double v = phi_value(D, g0 + l, *p, t);
        *p = v;
        F.phi[g0 + l + 1] = v;
    }
    if (rank == 0 && tid == NT - 32) {
        F.phi[0] = s_phi0;
        *F.ex0 = ex0;
    }
    __syncthreads();
    // E_x on the finest grid (EMFieldSolver::GetEfield)
    ex0 = s_ex0;
    auto phi = [&](int p) {  // p0 - 2 <= p <= p1 + 1
        if (p < p0) return s_halo[p - p0 + 2];
        if (p >= p1) return s_halo[p - p1 + 2];
        if (p == 0) return s_phi0;
        const int l = p - 1 - g0;
        return xs[(l % L) * stride + l / L];
    };
    if (rank > 0 && cnt == 0) return;
    for (int i = p0 + tid; i < p1; i += NT) {
        const double e = -fc * (8 * (phi(i + 1) - phi(i - 1)) - phi(i + 2) + phi(i - 2)) + ex0;
        F.efin[i] = e;
        if (P.f32) F.efin32[i] = (float)e;
    }
}

// Scan threads per block: segments of about 8 elements (a decaying pass then gathers three
// carry terms), 32 to kPsMaxThreads threads.
int scan_threads(int maxn) {
    const int m = maxn - 1;
    int t = 32;
    while (t < kPsMaxThreads && (long long)t * kPsCluster * 8 < m) t *= 2;
    return t;
}

}  // namespace

size_t poisson_scan_smem(int maxn) {
    const int m = maxn - 1, T = scan_threads(maxn);
    const int L = (m + T * kPsCluster - 1) / (T * kPsCluster);
    return (size_t)L * (T + 1) * sizeof(double);
}

void launch_poisson_fast(const PoissonFastLaunch &L) {
    if (L.nruns == 0) return;
    const size_t smem = poisson_scan_smem(L.maxn);
    PoissonFastLaunch P = L;
    P.scan_threads = scan_threads(L.maxn);
    vx_allow_smem(k_poisson_scan);
    vx_launch(k_poisson_scan, L.nruns * kPsCluster, std::max(P.assemble ? kPsMaxThreads : kPsMinThreads, P.scan_threads + 32), smem, L.stream, P);
}

}  // namespace vx
