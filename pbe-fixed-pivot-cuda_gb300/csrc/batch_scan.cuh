// =============================================================================
// batch_scan.cuh -- running sums over a cell's bins by a cluster of CTAs, and the
// launch of the per-cell prep kernels (batch_kernels.cu, batch_vjp.cu).
// =============================================================================
#pragma once

#include <cooperative_groups.h>

#include "agg_moments.cuh"
#include "batch_internal.cuh"

namespace pbe_gb300 {

namespace cg = cooperative_groups;

// The cell of a cluster of CTAs: its bins are split evenly over the CTAs, and a
// CTA's bins over its threads in contiguous runs.
struct CellPart {
    int rank, ranks;      // this CTA in the cell's cluster
    int r0, r1;           // its bins
    int t0, t1;           // this thread's bins
};
__device__ __forceinline__ CellPart cell_part(int n)
{
    const cg::cluster_group cl = cg::this_cluster();
    CellPart p;
    p.rank = static_cast<int>(cl.block_rank());
    p.ranks = static_cast<int>(cl.num_blocks());
    const int per = (n + p.ranks - 1) / p.ranks;
    p.r0 = min(n, p.rank * per);
    p.r1 = min(n, p.r0 + per);
    const int c = (p.r1 - p.r0 + static_cast<int>(blockDim.x) - 1) / static_cast<int>(blockDim.x);
    p.t0 = min(p.r1, p.r0 + c * static_cast<int>(threadIdx.x));
    p.t1 = min(p.r1, p.t0 + c);
    return p;
}

// Barrier over the CTAs of the cell.
__device__ __forceinline__ void cell_sync(const CellPart& part)
{
    if (part.ranks > 1) cg::this_cluster().sync(); else __syncthreads();
}

// Running sums over the cell's bins, from the first up (SUF = false) or from the
// last down (true), into pre: with m_q = {1/a, 1, a, a^2, x}_q and (y, z) = val(i)
//   pre[q stride + i]       = sum m_q y
//   pre[(5 + q) stride + i] = sum m_q z, bin j's z being relative to 2^E_j (SUF:
//                             2^-E_j), E_j the exponent of x_j; the sum to 2^E_i (2^-E_i)
// and, by the cluster's CTA 0, the sums of m_q y over all bins into mom[0..4]. Two
// passes over a thread's run (totals, then the running sums), a scan of the totals
// over lanes, warps and CTAs between them. Positions p count bins in the scan's
// direction. Fixed order for a fixed launch shape.
constexpr int kPrepMaxWarps = 8;
struct PrefixShared {
    double wt[kPrepMaxWarps][2 * kMomN];     // warp totals, then the warps' offsets
    int we[kPrepMaxWarps];                   // exponent after the warp's last bin
    double ct[2 * kMomN];                    // CTA totals (read by the cluster's other CTAs)
    int ce;
};

template <int K, bool SUF, class V>
__device__ void cell_scan(const double* __restrict__ x, const double* __restrict__ a,
                          const double* __restrict__ ia, V val, const CellPart& part, int n,
                          PrefixShared& sm, double* pre, long long stride, double* mom)
{
    const cg::cluster_group cl = cg::this_cluster();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    double P[kMomN], T[kMomN];
    auto bin = [&](int p) { return SUF ? n - 1 - p : p; };
    // a position's exponent, rising with it (down the grid -E does)
    auto ex = [&](int p) { const int E = exponent_of(__ldg(x + bin(p))); return SUF ? -E : E; };
    auto add = [&](int p, int& e) {
        const int i = bin(p), ei = ex(p);
        const double xi = __ldg(x + i);
        double y, z;
        val(i, xi, y, z);
        const double ai = (K >= 3) ? __ldg(a + i) : 0.0, iai = (K >= 3) ? __ldg(ia + i) : 0.0;
        const double ay = ai * y, az = ai * z;
        const double my[kMomN] = {iai * y, y, ay, (K >= 4) ? ai * ay : 0.0, xi * y};
        const double mz[kMomN] = {iai * z, z, az, (K >= 4) ? ai * az : 0.0, xi * z};
#pragma unroll
        for (int q = 0; q < kMomN; ++q) {
            if (!need_moment<K>(q)) continue;
            P[q] += my[q];
            T[q] = (ei != e ? scale_down(T[q], e - ei) : T[q]) + mz[q];
        }
        e = ei;
    };
#pragma unroll
    for (int q = 0; q < kMomN; ++q) { P[q] = 0.0; T[q] = 0.0; }
    const int eb = part.t0 > 0 ? ex(part.t0 - 1) : 0;   // before the run
    int e = part.t0 > 0 ? eb : ex(0);
    for (int p = part.t0; p < part.t1; ++p) add(p, e);
    // inclusive scan of the runs over the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int dE = __shfl_up_sync(0xffffffffu, e, o) - e;
#pragma unroll
        for (int q = 0; q < kMomN; ++q) {
            if (!need_moment<K>(q)) continue;
            const double p = __shfl_up_sync(0xffffffffu, P[q], o);
            const double t = __shfl_up_sync(0xffffffffu, T[q], o);
            if (lane >= o) { P[q] += p; T[q] += scale_down(t, dE); }
        }
    }
    if (lane == 31) {
        sm.we[w] = e;
#pragma unroll
        for (int q = 0; q < kMomN; ++q) { sm.wt[w][q] = P[q]; sm.wt[w][kMomN + q] = T[q]; }
    }
    // the runs before this lane's in the warp (their sum stands at exponent ep)
    const int eu = __shfl_up_sync(0xffffffffu, e, 1);
    const int ep = lane > 0 ? eu : eb;
#pragma unroll
    for (int q = 0; q < kMomN; ++q) {
        if (!need_moment<K>(q)) continue;
        const double p = __shfl_up_sync(0xffffffffu, P[q], 1);
        const double t = __shfl_up_sync(0xffffffffu, T[q], 1);
        P[q] = lane > 0 ? p : 0.0;
        T[q] = lane > 0 ? t : 0.0;
    }
    __syncthreads();
    // lanes 0 .. 2 kMomN - 1 of warp 0, one sum each: the warps' offsets in the CTA
    const bool weighted = lane >= kMomN;
    double acc = 0.0;
    int ea = 0;
    if (w == 0 && lane < 2 * kMomN) {
        for (int v = 0; v < nw; ++v) {
            const double t = sm.wt[v][lane];
            if (weighted && v > 0) acc = scale_down(acc, ea - sm.we[v]);
            ea = sm.we[v];
            acc += t;
        }
        sm.ct[lane] = acc;
        if (lane == 0) sm.ce = ea;
    }
    cell_sync(part);                                  // every CTA's totals are there
    if (w == 0 && lane < 2 * kMomN) {
        // the CTAs before this one, then the warps before each warp
        double base = 0.0;
        int be = 0;
        for (int r = 0; r < part.rank; ++r) {
            const int en = *cl.map_shared_rank(&sm.ce, r);
            if (weighted && r > 0) base = scale_down(base, be - en);
            base += *cl.map_shared_rank(&sm.ct[lane], r);
            be = en;
        }
        for (int v = 0; v < nw; ++v) {
            const double t = sm.wt[v][lane];
            sm.wt[v][lane] = base;                    // before warp v, at exponent be
            const int en = sm.we[v];
            __syncwarp((1u << (2 * kMomN)) - 1u);     // read by every lane
            if (lane == 0) sm.we[v] = be;
            if (weighted) base = scale_down(base, be - en);
            base += t;
            be = en;
        }
        if (part.rank == 0 && lane < kMomN) {
            double tot = sm.ct[lane];
            for (int r = 1; r < part.ranks; ++r) tot += *cl.map_shared_rank(&sm.ct[lane], r);
            mom[lane] = tot;
        }
    }
    __syncthreads();
    const int wb = sm.we[w];
#pragma unroll
    for (int q = 0; q < kMomN; ++q) {
        if (!need_moment<K>(q)) continue;
        P[q] += sm.wt[w][q];
        T[q] += scale_down(sm.wt[w][kMomN + q], wb - ep);
    }
    e = part.t0 > 0 ? ep : ex(0);
    for (int p = part.t0; p < part.t1; ++p) {
        add(p, e);
        const int i = bin(p);
#pragma unroll
        for (int q = 0; q < kMomN; ++q) {
            if (!need_moment<K>(q)) continue;
            pre[static_cast<long long>(q) * stride + i] = P[q];
            pre[static_cast<long long>(kMomN + q) * stride + i] = T[q];
        }
    }
}

// Prefix moments of y (AggWs::mloc's sums, over the whole cell).
template <int K>
__device__ __forceinline__ void cell_prefix(const double* __restrict__ x, const double* __restrict__ a,
                                            const double* __restrict__ ia, const double* y,
                                            const CellPart& part, int n, PrefixShared& sm, double* pre,
                                            long long stride, double* mom)
{
    cell_scan<K, false>(x, a, ia,
                        [&](int i, double xi, double& u, double& v) { u = y[i]; v = u * mantissa_of(xi); },
                        part, n, sm, pre, stride, mom);
}

// Launch of a per-cell prep kernel: a cluster of d.prep_ranks CTAs (prep_shape) of
// `threads` threads per cell.
template <class... P, class... A>
cudaError_t launch_prep(const BatchDev& d, void (*kern)(P...), int threads, cudaStream_t s, A... args)
{
    const unsigned ranks = static_cast<unsigned>(d.prep_ranks);
    return launch_result(launch_dep(kern, dim3(static_cast<unsigned>(d.n_cells) * ranks),
                                    static_cast<unsigned>(threads), 0, s, ranks, args...));
}

} // namespace pbe_gb300
