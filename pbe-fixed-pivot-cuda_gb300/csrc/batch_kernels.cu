// =============================================================================
// batch_kernels.cu -- batched-cell RHS and RK4 stage kernels (sm_103a, FP64).
//
// Per plan (once): batch_grid_kernel builds each grid's per-bin values, the
// beta-free per-lag tables and the geometric check; batch_frag_kernel builds
// the breakage fragment tables of each grid (brackets, weights, run starts).
//
// Per RHS evaluation (two launches):
//  * batch_prep_kernel, one cluster of CTAs per cell: the RK4 stage update of the
//    cell's state, the stage arrays (j-side factors carrying the cell's kernel
//    coefficients, S(x) N for breakage), the prefix moments over the bins (their
//    last sums are the death moments) and the sum of the cell's clipped pairs.
//  * batch_main_kernel: CTAs of 256 threads, each one "bundle" (largest first) of
//    256/T tasks (cell, first bin) that run side by side on groups of T threads;
//    T is chosen per section-count class by the plan (autotuned or by rule). A
//    task owns 31 bins of a cell: a warp's lanes hold their slots and the one
//    below (agg_slot.cuh), the group's warps split the pairs that the prefix
//    moments leave, and the group gathers the breakage term of its bins from S N
//    (a few fragments per bin and quadrature point), adds the clip sum and
//    writes its bins once: no atomics, and a fixed summation order for a fixed
//    schedule. The slot below the first bin is summed by two tasks (1 in 32), so
//    nothing is handed over between tasks.
// RK4 of plans of small cells: batch_cells_rk4_kernel, a CTA per cell that runs the
// bodies of both for all stages of its steps.
// =============================================================================
#include <type_traits>

#include "batch_internal.cuh"
#include "agg_slot.cuh"
#include "batch_scan.cuh"

namespace pbe_gb300 {
namespace {

constexpr int SW = kSlotBins;

// ---------------------------------------------------------------------------
// Grid tables: one CTA per grid. Per bin: a, 1/a, 1/dx; per lag d (= bin
// index): Bd = c_d * (1 or rho + 1/rho + 2), Sd = c_d (1 + rho)^3 with
// rho = (x_d / x_0)^(1/3), c_d = 1/2 for d = 0 (beta is applied per cell, on
// the j side); Ld = bracket of x_0 + x_d. Geometric check as the
// single-instance prep (max |ln(x_i/x_0) - i ln r| <= kGeoTol, x_1 <= 64 x_0).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
batch_grid_kernel(BatchDev d)
{
    dep_wait();
    __shared__ double sh[8];
    __shared__ int d0_s;
    BatchGridDev* gd = d.grids + blockIdx.x;
    const int n = gd->n;
    const double* x = d.gx + gd->off;
    if (threadIdx.x == 0) d0_s = n;
    __syncthreads();
    const bool brownian_like = (d.kernel >= 3);
    double dev = 0.0;
    int d0 = n;
    const double x0 = x[0];
    const double ax0 = cbrt(x0);
    const GeoFit fit = geo_fit(x0, x[n - 1], n);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double xi = x[i];
        const double ai = cbrt(xi);
        d.ga[gd->off + i] = ai;
        d.gia[gd->off + i] = 1.0 / ai;
        d.ginv_dx[gd->off + i] = (i < n - 1) ? 1.0 / (x[i + 1] - xi) : 0.0;
        const double c = (i == 0) ? 0.5 : 1.0;
        const double rho = ai / ax0;
        const double s = 1.0 + rho;
        d.gBd[gd->off + i] = brownian_like ? c * (rho + 1.0 / rho + 2.0) : c;
        d.gSd[gd->off + i] = c * (s * s) * s;
        d.gSl[gd->off + i] = (s * s) * s * (x0 / xi);
        const double v = x0 + xi;
        const int L = (dbits(v) >= dbits(x[n - 1])) ? kLagClipAll : bracket_from(x, n, v, i);
        d.gLd[gd->off + i] = L;
        if (L == i && i > 0) d0 = min(d0, i);   // lag 0 carries the pair 1/2: never separated
        // first j with fl(x_j + x_i) >= x_{i+1}: the prefix sums of slot i on a
        // grid that is not geometric (monotone in j, so a bisection)
        int jl = 0, jh = i;
        if (i < n - 1) {
            const long long top = dbits(x[i + 1]);
            while (jl < jh) {
                const int mid = (jl + jh) >> 1;
                if (dbits(x[mid] + xi) >= top) jh = mid; else jl = mid + 1;
            }
        }
        d.gJ0[gd->off + i] = jl;
        d.gJt[gd->off + i] = i < n - 1 ? slot_rows_end(x, i, i) : 0;
        if (n >= 2) {
            double e = geo_dev(fit, xi, i);
            if (!(e == e)) e = 1.0;
            dev = fmax(dev, e);
        }
    }
    atomicMin(&d0_s, d0);
    dev = warp_max(dev);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = dev;
    __syncthreads();
    if (threadIdx.x == 0) {
        double mx = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) mx = fmax(mx, sh[w]);
        const bool ratio_ok = n >= 2 && x[1] <= 64.0 * x[0];
        gd->geo = (n >= 2 && mx <= kGeoTol && ratio_ok) ? 1 : 0;
        gd->D0 = d0_s;
    }
}

// Breakage fragment tables: one CTA per grid, threads over (q, j). Fragment
// v = x_j t_q has the bracket lo = frag_bracket (-1: clipped to bin 0, n-1:
// clipped to bin n-1); its shares of bw_q are
// (bw_q/(x_{lo+1} - x_lo)) (x_{lo+1} - v) and (...) (v - x_lo), as the
// reference splits contrib (src/breakage_kernels.cuh:197-216).
__global__ void __launch_bounds__(256)
batch_frag_kernel(BatchDev d, const double* __restrict__ t_q, const double* __restrict__ bw_q)
{
    const int dep = dep_wait();
    t_q += dep; bw_q += dep;
    const BatchGridDev gd = d.grids[blockIdx.x];
    const int n = gd.n, nq = d.nq;
    const double* x = d.gx + gd.off;
    for (int idx = threadIdx.x; idx < n * nq; idx += blockDim.x) {
        const int q = idx / n, j = idx - q * n;
        const double tq = t_q[q], bw = bw_q[q];
        const double v = x[j] * tq;
        const int lo = frag_bracket(x, n, v);
        double wl = bw, wh = 0.0;
        if (lo >= 0 && lo < n - 1) {
            const double xl = x[lo], xh = x[lo + 1];
            const double qq = bw / (xh - xl);
            wl = qq * (xh - v);
            wh = qq * (v - xl);
        }
        d.bwlo[gd.woff + q * n + j] = wl;
        d.bwhi[gd.woff + q * n + j] = wh;
        d.blo[gd.woff + q * n + j] = lo;
        int* fq = d.bfirst + gd.foff + q * (n + 2);
        const int lo_prev = (j == 0) ? -2 : frag_bracket(x, n, x[j - 1] * tq);
        for (int m = max(lo_prev + 1, -1); m <= lo; ++m) fq[m + 1] = j;
        if (j == n - 1)
            for (int m = max(lo + 1, -1); m <= n; ++m) fq[m + 1] = n;
    }
}

// ---------------------------------------------------------------------------
// Stage prep: one CTA per cell.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double sel_value(int F, double v, double S0, double v_ref,
                                            double alpha, double v_min)
{
    switch (F) {
    case 0: return selection<0>(v, S0, v_ref, alpha, v_min);
    case 1: return selection<1>(v, S0, v_ref, alpha, v_min);
    case 2: return selection<2>(v, S0, v_ref, alpha, v_min);
    default: return selection<3>(v, S0, v_ref, alpha, v_min);
    }
}

// RK4 stage arithmetic of the reference examples (pbe_examples_utils.hpp:432-455)
// with every product and sum rounded separately, as the host code does:
// stage = N + (c dt) k, N_new = N + (dt/6) (((k1 + 2 k2) + 2 k3) + k4).
__device__ __forceinline__ double stage_update(int stage, double* N, const double* k, double* kacc,
                                               double* Y, int i, double c, double dt6)
{
    double y;
    if (stage == kStageRhs) {
        y = N[i];
    } else if (stage == kStageNext || stage == kStageFinish) {
        const double s = __dadd_rn(kacc[i], k[i]);
        y = __dadd_rn(N[i], __dmul_rn(dt6, s));
        N[i] = y;
    } else {
        const double ki = k[i];
        kacc[i] = (stage == kStageTwo) ? ki : __dadd_rn(kacc[i], __dmul_rn(2.0, ki));
        y = __dadd_rn(N[i], __dmul_rn(c, ki));
        Y[i] = y;
    }
    return y;
}

// Per-cell stage update of the per-cell launch loop (same arithmetic).
__global__ void __launch_bounds__(256)
cell_stage_kernel(double* N, const double* k, double* kacc, double* Y, int n, int stage,
                  double c, double dt6)
{
    const int dep = dep_wait();
    k += dep; n += dep;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) stage_update(stage, N, k, kacc, Y, i, c, dt6);
}

// Selection function of every cell bin for the given parameters: one thread
// per packed bin over the whole plan (its cell found by bisection of the
// cells' offsets), so that a large cell's transcendentals spread over all
// SMs instead of one CTA's; evaluated once per call instead of per stage.
__global__ void __launch_bounds__(256)
batch_sel_kernel(BatchDev d, const pbe_batch_cell_params_t* __restrict__ params,
                 double* __restrict__ Sx, long long total)
{
    const int dep = dep_wait();
    params += dep; Sx += dep;
    for (long long e = blockIdx.x * 256LL + threadIdx.x; e < total; e += 256LL * gridDim.x) {
        int lo = 0, hi = d.n_cells;          // cells[lo].off <= e < cells[hi].off
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (d.cells[mid].off <= e) lo = mid; else hi = mid;
        }
        const BatchCellDev cd = d.cells[lo];
        const pbe_batch_cell_params_t P = params[lo];
        const double* x = d.gx + d.grids[cd.grid].off;
        Sx[e] = sel_value(d.selection, x[e - cd.off], P.S0, P.v_ref, P.alpha, P.v_min);
    }
}

// One lane's part of the breakage gather of bin i (0 < i < n) of a cell:
// quadrature points q = q0, q0 + nqp, ..., each adding the hi-shares of the
// fragments bracketed at i-1 and the lo-shares of those at i. The nqp lanes of a
// bin then add their parts in a fixed butterfly.
__device__ __forceinline__ double brk_lane(const BatchDev& d, const BatchGridDev& gd,
                                           const double* SN, int n, int i, int q0, int nqp)
{
    const int ng = gd.n;
    double acc = 0.0;
    for (int q = q0; q < d.nq; q += nqp) {
        const int* fq = d.bfirst + gd.foff + q * (ng + 2);
        const double* wl = d.bwlo + gd.woff + q * ng;
        const double* wh = d.bwhi + gd.woff + q * ng;
        const int fa = min(max(fq[i], 0), n);         // first j with lo >= i-1
        const int fb = min(max(fq[i + 1], fa), n);    // first j with lo >= i
        const int fc = min(max(fq[i + 2], fb), n);    // first j with lo >= i+1
        for (int j = fa; j < fb; ++j) acc = fma(SN[j], wh[j], acc);
        for (int j = fb; j < fc; ++j) acc = fma(SN[j], wl[j], acc);
    }
    return acc;
}

// Bin 0 by one warp, its lanes over the parents: the lo-shares of the fragments
// clipped below x[0] and of those bracketed at 0 (with small table entries that is
// some hundred parents a point, 18 us for one lane at 128 sections an octave).
// Valid in every lane.
__device__ __forceinline__ double brk_bin0(const BatchDev& d, const BatchGridDev& gd, const double* SN, int n)
{
    const int ng = gd.n;
    double acc = 0.0;
    for (int q = 0; q < d.nq; ++q) {
        const int fc = min(max(d.bfirst[gd.foff + q * (ng + 2) + 2], 0), n);   // first j with lo >= 1
        const double* wl = d.bwlo + gd.woff + q * ng;
        for (int j = threadIdx.x & 31; j < fc; j += 32) acc = fma(SN[j], wl[j], acc);
    }
    return warp_sum(acc);
}

__device__ __forceinline__ int brk_lanes(int nq)
{
    int nqp = 1;
    while (nqp < nq && nqp < 32) nqp <<= 1;
    return nqp;
}

// Breakage term of the bins [r0, r1) of a cell (one CTA; the prep kernels without
// kBrkTasks), minus S_i N_i: a warp covers 32/nqp bins, nqp = the quadrature
// points rounded up to a power of two (<= 32) lanes per bin.
__device__ void cell_breakage(const BatchDev& d, const BatchGridDev& gd, const double* SN,
                              double* Bk, int n, int r0, int r1)
{
    const int nqp = brk_lanes(d.nq);
    const int per_warp = 32 / nqp;
    const int nw = blockDim.x >> 5, w = threadIdx.x >> 5, l = threadIdx.x & 31;
    for (int base = r0 + w * per_warp; base < r1; base += nw * per_warp) {   // uniform per warp
        const int i = base + l / nqp;
        double acc = (i < r1 && i > 0) ? brk_lane(d, gd, SN, n, i, l % nqp, nqp) : 0.0;
        for (int o = nqp >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (i < r1 && i > 0 && (l % nqp) == 0) Bk[i] = acc - SN[i];
    }
    if (r0 == 0 && w == nw - 1) {
        const double acc = brk_bin0(d, gd, SN, n);
        if (l == 0) Bk[0] = acc - SN[0];
    }
}

// The same term for the bins I .. I+SW-1 of a cell (those below n), by a
// task's group into out[0 .. SW) (kBrkTasks): the same lanes per bin, loops and
// butterfly, so the sums are bitwise those of cell_breakage.
template <class Group>
__device__ void tile_breakage(const BatchDev& d, const BatchGridDev& gd, const double* SN, int n,
                              int I, double* out, const Group& G)
{
    const int nqp = brk_lanes(d.nq);
    const int per_warp = 32 / nqp;
    const int nw = G.T >> 5, w = G.lane >> 5, l = G.lane & 31;
    for (int base = w * per_warp; base < SW; base += nw * per_warp) {   // uniform per warp
        const int t = base + l / nqp;
        const int i = I + t;
        const bool in = t < SW && i > 0 && i < n;
        double acc = in ? brk_lane(d, gd, SN, n, i, l % nqp, nqp) : 0.0;
        for (int o = nqp >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (t < SW && i > 0 && (l % nqp) == 0) out[t] = in ? acc - SN[i] : 0.0;
    }
    if (I == 0 && w == nw - 1) {
        const double acc = brk_bin0(d, gd, SN, n);
        if (l == 0) out[0] = acc - SN[0];
    }
}

__device__ __forceinline__ SlotGrid slot_grid(const BatchDev& d, const BatchGridDev& gd, int n,
                                              const pbe_batch_cell_params_t& P)
{
    return SlotGrid{d.gx + gd.off, d.ga + gd.off, d.gia + gd.off, d.ginv_dx + gd.off,
                    d.gBd + gd.off, d.gSd + gd.off, d.gLd + gd.off, d.gJ0 + gd.off,
                    n, gd.D0, gd.geo != 0, P.beta0, P.beta_br, P.beta_sh};
}

// The passes of a launch for the cell at packed offset off: the RHS at Y (one
// pass), or the Jacobian-vector product at d.A along Y (A with Y, Y with A).
template <int NP>
__device__ __forceinline__ void slot_passes(const BatchDev& d, const double* Y, int off, SlotPass* p)
{
    const double* y = Y + off;
    if constexpr (NP == 1) {
        p[0] = SlotPass{d.Nj + off, d.Hj + off, y, d.Hk + off, y, d.Hk + off};
    } else {
        const double* a = d.A + off;
        p[0] = SlotPass{d.Nj + off, d.Hj + off, a, d.Ha + off, y, d.Hk + off};
        p[1] = SlotPass{d.Nj2 + off, d.Hj2 + off, y, d.Hk + off, a, d.Ha + off};
    }
}

// ---------------------------------------------------------------------------
// Stage prep: one cluster per cell. Per bin: the stage update and the stage
// arrays (S N for the breakage gather of the pair tasks); then the prefix
// moments, and (after a cluster barrier, so the whole cell's arrays are
// visible) each CTA's part of the cell's clipped pairs (mom[10 + rank]) and of
// its breakage term.
// ---------------------------------------------------------------------------
struct PrepShared {
    double sh[8];
    PrefixShared psm;
};

template <int K>
__device__ void prep_cell(const BatchDev& d, double* N, const pbe_batch_cell_params_t* params, int cell,
                          int stage, double c, double dt6, const StageCombine& sc, PrepShared& sm)
{
    const BatchCellDev cd = d.cells[cell];
    const BatchGridDev gd = d.grids[cd.grid];
    const pbe_batch_cell_params_t P = params[cell];
    const bool agg = d.kernel >= 0;
    const int F = d.selection;
    const int off = cd.off, n = cd.n;
    const CellPart part = cell_part(n);
    double* Nc = N + off;
    double* kc = d.k + off;
    double* ac = d.kacc + off;
    double* Yc = d.Y + off;
    const double* x = d.gx + gd.off;
    // j-side coefficients: Nj = cN * N, Hj = cH * x N
    const double cN = (K <= 2) ? P.beta0 : P.beta_br;
    const double cH = (K == 1 || K == 2) ? P.beta0 : P.beta_sh;
    const double dtc = (stage == kStageCombine) ? sc.dt[cell] : 0.0;
    for (int i = part.r0 + threadIdx.x; i < part.r1; i += blockDim.x) {
        double y;
        if (stage == kStageCombine) {
            double s_ = 0.0;
            for (int j = 0; j < sc.nk; ++j) s_ = fma(sc.a[j], sc.k[j][off + i], s_);
            y = fma(dtc, s_, Nc[i]);
            Yc[i] = y;
        } else {
            y = stage_update(stage, Nc, kc, ac, Yc, i, c, dt6);
        }
        if (stage == kStageFinish) continue;
        const double xi = x[i];
        if (agg) {
            const double h = xi * y;
            if (K != 2 && K != 4) d.Nj[off + i] = cN * y;
            if (NeedH<K>::j) d.Hj[off + i] = cH * h;
            if (NeedH<K>::k) d.Hk[off + i] = h;
        }
        if (F >= 0) {
            const double S = d.Sx ? d.Sx[off + i] : sel_value(F, xi, P.S0, P.v_ref, P.alpha, P.v_min);
            d.SN[off + i] = (S != 0.0 && y > kBreakageNMin) ? S * y : 0.0;
        }
    }
    if (stage == kStageFinish) return;
    __syncthreads();                       // this CTA's part of the stage arrays is complete
    const double* Yk = (stage == kStageRhs || stage == kStageNext) ? Nc : Yc;
    double* mom = d.mom + static_cast<size_t>(cell) * kMomStride;
    if (agg) {
        cell_prefix<K>(x, d.ga + gd.off, d.gia + gd.off, Yk, part, n, sm.psm, d.pre + off, d.total, mom);
    }
    cell_sync(part);                       // the cell's stage arrays are complete; all shared reads done
    if (agg) {
        const SlotGrid g = slot_grid(d, gd, n, P);
        SlotPass sp[1];
        slot_passes<1>(d, Yk - off, off, sp);
        const int nt = part.ranks * static_cast<int>(blockDim.x);
        const double clip = block_sum(slot_clip<K, 1>(g, sp, slot_clip_tid(part.rank, part.ranks), nt,
                                                      slot_clip_lanes(n, nt)), sm.sh);
        if (threadIdx.x == 0) mom[10 + part.rank] = clip;
    }
    if (d.nq > 0 && !(d.brk & kBrkTasks)) cell_breakage(d, gd, d.SN + off, d.Bk + off, n, part.r0, part.r1);
}

template <int K>
__global__ void __launch_bounds__(256)
batch_prep_kernel(BatchDev d, double* N, const pbe_batch_cell_params_t* __restrict__ params,
                  int stage, double c, double dt6, StageCombine sc)
{
    const int dep = dep_wait();
    params += dep;
    __shared__ PrepShared sm;
    const int cell = blockIdx.x / cg::this_cluster().num_blocks();
    if (d.skip && d.skip[cell]) return;             // whole cluster
    prep_cell<K>(d, N, params, cell, stage, c, dt6, sc, sm);
}

// ---------------------------------------------------------------------------
// Prep of a Jacobian-vector product at the state A along v (one cluster per
// cell). The aggregation RHS is quadratic: R(N) = T(N, N) with T(a, b) = sum
// over pairs j <= k of c_d beta(j, k) a_j b_k (deposits as the RHS; death b_i
// sum_k beta_ik a_k), so J(N) v = T(N, v) + T(v, N), both in one pass of the
// pair kernel. This prep builds both vectors' j-side arrays and x products,
// their prefix moments (mom[0..4] of A, mom[5..9] of v), the clipped pairs, and
// the breakage input: the breakage RHS is linear in N wherever its guard passes,
// so its Jacobian-vector product deposits S_j v_j as the RHS deposits S_j N_j,
// for the bins whose A_j passes the guard S_j != 0 && A_j > 2.2e-308.
// ---------------------------------------------------------------------------
template <int K>
__global__ void __launch_bounds__(256)
batch_jvp_prep_kernel(BatchDev d, const double* __restrict__ v,
                      const pbe_batch_cell_params_t* __restrict__ params)
{
    const int dep = dep_wait();
    v += dep; params += dep;
    __shared__ double sh[8];
    __shared__ PrefixShared psm;
    const cg::cluster_group cl = cg::this_cluster();
    const int cell = blockIdx.x / cl.num_blocks();
    if (d.skip && d.skip[cell]) return;             // whole cluster
    const BatchCellDev cd = d.cells[cell];
    const BatchGridDev gd = d.grids[cd.grid];
    const pbe_batch_cell_params_t P = params[cell];
    const bool agg = d.kernel >= 0;
    const int F = d.selection;
    const int off = cd.off, n = cd.n;
    const CellPart part = cell_part(n);
    const double* x = d.gx + gd.off;
    const double cN = (K <= 2) ? P.beta0 : P.beta_br;
    const double cH = (K == 1 || K == 2) ? P.beta0 : P.beta_sh;
    for (int i = part.r0 + threadIdx.x; i < part.r1; i += blockDim.x) {
        const double ya = d.A[off + i], yb = v[off + i];
        const double xi = x[i];
        if (agg) {
            const double ha = xi * ya, hb = xi * yb;
            if (K != 2 && K != 4) { d.Nj[off + i] = cN * ya; d.Nj2[off + i] = cN * yb; }
            if (NeedH<K>::j) { d.Hj[off + i] = cH * ha; d.Hj2[off + i] = cH * hb; }
            d.Ha[off + i] = ha;
            d.Hk[off + i] = hb;
        }
        if (F >= 0) {
            const double S = d.Sx ? d.Sx[off + i] : sel_value(F, xi, P.S0, P.v_ref, P.alpha, P.v_min);
            d.SN[off + i] = (S != 0.0 && ya > kBreakageNMin) ? S * yb : 0.0;
        }
    }
    __syncthreads();
    double* mom = d.mom + static_cast<size_t>(cell) * kMomStride;
    if (agg) {
        cell_prefix<K>(x, d.ga + gd.off, d.gia + gd.off, d.A + off, part, n, psm, d.pre + off, d.total, mom);
        cl.sync();                         // the shared totals are read by every CTA
        cell_prefix<K>(x, d.ga + gd.off, d.gia + gd.off, v + off, part, n, psm, d.pre2 + off, d.total, mom + 5);
    }
    cl.sync();                             // the cell's pass arrays are complete
    if (agg) {
        const SlotGrid g = slot_grid(d, gd, n, P);
        SlotPass sp[2];
        slot_passes<2>(d, v, off, sp);
        const int nt = part.ranks * static_cast<int>(blockDim.x);
        const double clip = block_sum(slot_clip<K, 2>(g, sp, slot_clip_tid(part.rank, part.ranks), nt,
                                                      slot_clip_lanes(n, nt)), sh);
        if (threadIdx.x == 0) mom[10 + part.rank] = clip;
    }
    if (d.nq > 0 && !(d.brk & kBrkTasks)) cell_breakage(d, gd, d.SN + off, d.Bk + off, n, part.r0, part.r1);
}

// A warp as a group of its own: no named barrier (a kernel whose barrier numbers are not
// constants takes all 16 of a CTA, and an SM then holds four CTAs).
struct WarpGroup {
    int g, lane;
    static constexpr int T = 32;
    __device__ __forceinline__ void sync() const { __syncwarp(); }
};

// Shared memory of a CTA of the pair kernel (per group g < kMaxGroups).
struct SlotShared {
    double red[kMaxGroups][2][32];        // per-warp R, TH of every slot
    double extra[kMaxGroups][SW];         // per-bin breakage (kBrkTasks)
};

// ---------------------------------------------------------------------------
// One pair task (cell, first bin I) on a group of T threads: the bins
// [I, I + 31), lane l of each warp holding slot I - 1 + l. FP64 instructions per
// slot, Brownian + shear: 4 per direct pair, 22 for the prefix part, 12 for the
// death term and the bin.
// ---------------------------------------------------------------------------
// Group: TileGroup, or WarpGroup for one warp.
template <int K, int NP, class Group>
__device__ void batch_task(const BatchDev& d, const double* __restrict__ Yg,
                           const pbe_batch_cell_params_t* __restrict__ params, double* out,
                           bool accumulate, int4 tk, SlotShared& sm, const Group& G)
{
    const int c = tk.x, I = tk.y;
    if (d.skip && d.skip[c]) return;                // the whole group
    const BatchCellDev cd = d.cells[c];
    const BatchGridDev gd = d.grids[cd.grid];
    const int n = cd.n, off = cd.off;
    const bool agg = d.kernel >= 0;
    const int l = G.lane & 31, w = G.lane >> 5, nw = G.T >> 5;
    const pbe_batch_cell_params_t P = params[c];
    const SlotGrid g = slot_grid(d, gd, n, P);
    SlotPass p[NP];
    slot_passes<NP>(d, Yg, off, p);
    const int s = I - 1 + l;                        // this lane's slot and bin
    const bool slot = s >= 0 && s <= n - 2;
    const int St = slot ? -exponent_of(__ldg(g.x + s)) : 0;
    double R = 0.0, TH = 0.0;
    unsigned exact = 0u;
    if (agg) {
        if (g.geo) slot_lags<K, NP>(g, p, I, w, nw, R, TH);
        else slot_pairs_any<K, NP>(g, p, s, slot, slot ? __ldg(d.gJt + gd.off + s) : 0, w, nw, R, TH);
        // (two pairs of an exact slot in flight: an RHS of one cell of 3840 with every other
        // section empty 210 us, 180 so; not with two passes or 72 registers, where they spill)
        constexpr int kU = NP == 1 && !std::is_same<Group, WarpGroup>::value ? 2 : 1;
        exact = slot_exact_turns<K, NP, kU>(g, p, I, w, nw, R, TH);
    }
    const bool brk = d.nq > 0;
    const bool brk_tasks = (d.brk & kBrkTasks) != 0;
    if (brk && brk_tasks) tile_breakage(d, gd, d.SN + off, n, I, sm.extra[G.g], G);
    if (nw > 1) {
        sm.red[G.g * nw + w][0][l] = R;
        sm.red[G.g * nw + w][1][l] = TH;
    }
    G.sync();
    if (w != 0) return;
    for (int q = 1; q < nw; ++q) {
        R += sm.red[G.g * nw + q][0][l];
        TH += sm.red[G.g * nw + q][1][l];
    }
    double clip = 0.0, death = 0.0;
    if (agg && s >= 0 && s < n) {
        const double as = __ldg(g.a + s), ias = __ldg(g.ia + s), xv = __ldg(g.x + s);
        const double* mom = d.mom + static_cast<size_t>(c) * kMomStride;
        const int cut = slot_cut(g, s);
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            const double b = p[q].Nk[s];
            if (cut > 0 && !((exact >> l) & 1u)) {
                const double* pre = (q == 0 ? d.pre : d.pre2) + off + (cut - 1);
                double M[kMomN], M1[kMomN];
#pragma unroll
                for (int m = 0; m < kMomN; ++m) {
                    M[m] = need_moment<K>(m) ? pre[m * d.total] : 0.0;
                    M1[m] = need_moment<K>(m) ? pre[(kMomN + m) * d.total] : 0.0;
                }
                const double r = b * death_factor<K>(xv, as, ias, M, g.b0, g.bbr, g.bsh);
                if (slot) {
                    const double t = death_factor<K>(xv, as, ias, M1, g.b0, g.bbr, g.bsh);
                    R += r;
                    TH += b * scale_down(t, exponent_of(__ldg(g.x + cut - 1)) + St);
                } else {
                    clip += r;                      // bin n - 1: clipped
                }
            }
            double M[kMomN];
#pragma unroll
            for (int m = 0; m < kMomN; ++m) M[m] = need_moment<K>(m) ? mom[5 * q + m] : 0.0;
            death += b * death_factor<K>(xv, as, ias, M, g.b0, g.bbr, g.bsh);
        }
        if (s == n - 1)
            for (int r = 0; r < d.prep_ranks; ++r) clip += mom[10 + r];
    }
    // the slot's own part of its bin, and its w-part, owed to the bin above
    double own = 0.0, up = 0.0;
    if (slot) {
        const double sd = scalbn(__ldg(g.inv_dx + s), -St);
        own = fma(-TH, sd, R);
        up = TH * sd;
    }
    const double in = __shfl_up_sync(0xffffffffu, up, 1);
    if (l >= 1 && s < n) {
        double val = 0.0;
        if (agg) val = ((own + in) + clip) - death;
        if (brk) val += brk_tasks ? sm.extra[G.g][l - 1] : d.Bk[off + s];
        double* o = out + off + s;
        *o = accumulate ? *o + val : val;
    }
}

#ifndef PBE_BATCH_CTAS
#define PBE_BATCH_CTAS 3
#endif
template <int K, int NP>
__global__ void __launch_bounds__(kMainThreads, PBE_BATCH_CTAS)
batch_main_kernel(BatchDev d, const double* __restrict__ Y,
                  const pbe_batch_cell_params_t* __restrict__ params, double* out, int accumulate,
                  const int4* __restrict__ bundles, const int4* __restrict__ tasks)
{
    const int dep = dep_wait();
    Y += dep; params += dep; bundles += dep; tasks += dep;
    __shared__ SlotShared sm;
    const int4 bu = bundles[blockIdx.x];     // {first task, tasks, group size, 0}
    const int T = bu.z;
    const int g = threadIdx.x / T;
    if (g >= bu.y) return;                   // whole groups
    const TileGroup G{g, static_cast<int>(threadIdx.x) - g * T, T};
    batch_task<K, NP>(d, Y, params, out, accumulate != 0, tasks[bu.x + g], sm, G);
}

// ---------------------------------------------------------------------------
// RK4 of small cells: a CTA per cell, a warp per slot block, up to kCellSteps steps
// in one launch (cells do not see each other). With a prep and a pair kernel a stage,
// 4096 cells of 48 sections took 462 us a step, most of it the arrays' way through
// L2 and the latency of two short kernels at a few warps an SM; 411 us here (256 cells
// of 48: 121 and 84).
// ---------------------------------------------------------------------------
template <int K>
__global__ void __launch_bounds__(32 * kCellWarps, 7)
batch_cells_rk4_kernel(BatchDev d, double* N, const pbe_batch_cell_params_t* __restrict__ params,
                       double dt, int n_steps)
{
    const int dep = dep_wait();
    params += dep;
    __shared__ PrepShared psm;
    __shared__ SlotShared sm;
    const int cell = blockIdx.x, n = d.cells[cell].n, w = threadIdx.x >> 5;
    const WarpGroup G{w, static_cast<int>(threadIdx.x & 31)};
    const double h = 0.5 * dt, dt6 = dt / 6.0;
    for (int step = 0; step < n_steps; ++step) {
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
            const int stage = q > 1 ? kStageThree : q == 1 ? kStageTwo : step == 0 ? kStageRhs : kStageNext;
            prep_cell<K>(d, N, params, cell, stage, q == 3 ? dt : h, dt6, StageCombine{}, psm);
            __syncthreads();
            for (int I = SW * w; I < n; I += SW * static_cast<int>(blockDim.x >> 5)) {
                batch_task<K, 1>(d, q == 0 ? N : d.Y, params, d.k, false, make_int4(cell, I, 0, 0), sm, G);
                __syncwarp();
            }
            __syncthreads();
        }
    }
    prep_cell<K>(d, N, params, cell, kStageFinish, 0.0, dt6, StageCombine{}, psm);
}

template <int K>
cudaError_t main_k(const BatchDev& d, const double* Y, const pbe_batch_cell_params_t* params,
                   double* out, bool accumulate, const int4* bundles, const int4* tasks,
                   int n_bundles, cudaStream_t s)
{
    if (n_bundles <= 0) return cudaSuccess;
    if (d.A)
        launch_dep(batch_main_kernel<K, 2>, dim3(n_bundles), kMainThreads, 0, s, 1, d, Y, params, out,
                   accumulate ? 1 : 0, bundles, tasks);
    else
        launch_dep(batch_main_kernel<K, 1>, dim3(n_bundles), kMainThreads, 0, s, 1, d, Y, params, out,
                   accumulate ? 1 : 0, bundles, tasks);
    return cudaGetLastError();
}

} // namespace

cudaError_t batch_cells_rk4(const BatchDev& d, double* N, const pbe_batch_cell_params_t* params, double dt,
                            int n_steps, int max_n, cudaStream_t s)
{
    auto run = [&](auto kern) {
        // a warp per slot block, as far as the SMs hold all cells' CTAs at once (28 warps of
        // 72 registers each); the prep's scan costs per warp
        int warps = (max_n + SW - 1) / SW;
        while (warps > 1 && static_cast<long long>(warps) * d.n_cells > 28LL * d.num_sms) --warps;
        cudaError_t e = cudaSuccess;
        for (int st = 0; st < n_steps && e == cudaSuccess; st += kCellSteps)   // launches of milliseconds
            e = launch_dep(kern, dim3(d.n_cells), 32 * warps, 0, s, 1, d, N, params, dt,
                           n_steps - st < kCellSteps ? n_steps - st : kCellSteps);
        return launch_result(e);
    };
    switch (d.kernel < 0 ? 0 : d.kernel) {
    case 0: return run(batch_cells_rk4_kernel<0>);
    case 1: return run(batch_cells_rk4_kernel<1>);
    case 2: return run(batch_cells_rk4_kernel<2>);
    case 3: return run(batch_cells_rk4_kernel<3>);
    case 4: return run(batch_cells_rk4_kernel<4>);
    case 5: return run(batch_cells_rk4_kernel<5>);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t batch_grid_tables(const BatchDev& d, const double* t_q, const double* bw_q,
                              int max_grid_n, cudaStream_t s)
{
    (void)max_grid_n;
    if (d.n_grids <= 0) return cudaErrorInvalidValue;
    launch_dep(batch_grid_kernel, dim3(d.n_grids), 256, 0, s, 1, d);
    if (d.nq > 0) launch_dep(batch_frag_kernel, dim3(d.n_grids), 256, 0, s, 1, d, t_q, bw_q);
    return cudaGetLastError();
}

namespace {
cudaError_t prep_any(const BatchDev& d, double* N, const pbe_batch_cell_params_t* params, int stage,
                     double c, double dt6, const StageCombine& sc, cudaStream_t s)
{
    if (d.n_cells <= 0) return cudaErrorInvalidValue;
    switch (d.kernel < 0 ? 0 : d.kernel) {
    case 0: return launch_prep(d, batch_prep_kernel<0>, d.prep_threads, s, d, N, params, stage, c, dt6, sc);
    case 1: return launch_prep(d, batch_prep_kernel<1>, d.prep_threads, s, d, N, params, stage, c, dt6, sc);
    case 2: return launch_prep(d, batch_prep_kernel<2>, d.prep_threads, s, d, N, params, stage, c, dt6, sc);
    case 3: return launch_prep(d, batch_prep_kernel<3>, d.prep_threads, s, d, N, params, stage, c, dt6, sc);
    case 4: return launch_prep(d, batch_prep_kernel<4>, d.prep_threads, s, d, N, params, stage, c, dt6, sc);
    case 5: return launch_prep(d, batch_prep_kernel<5>, d.prep_threads, s, d, N, params, stage, c, dt6, sc);
    default: return cudaErrorInvalidValue;
    }
}

__global__ void __launch_bounds__(256)
rk45_control_kernel(BatchDev d, double* N, const double* __restrict__ Y, StageCombine e,
                    double* k0, Rk45Ctl ctl)
{
    const int dep = dep_wait();
    Y += dep;
    __shared__ double sh[8];
    __shared__ int accept_s;
    const int c = blockIdx.x;
    if (ctl.status[c] != 0) return;                 // whole block
    const BatchCellDev cd = d.cells[c];
    const int off = cd.off, n = cd.n;
    const double dt = ctl.dt[c];
    double s2 = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        double s_ = 0.0;
        for (int j = 0; j < e.nk; ++j) s_ = fma(e.a[j], e.k[j][off + i], s_);
        const double sc = ctl.atol + ctl.rtol * fmax(fabs(N[off + i]), fabs(Y[off + i]));
        const double r = (dt * s_) / sc;
        s2 = fma(r, r, s2);
    }
    s2 = block_sum(s2, sh);
    if (threadIdx.x == 0) {
        const double err = sqrt(s2 / n);
        const bool finite = (err == err) && err <= 1.7e308;
        const bool accept = finite && err <= 1.0;
        double fac;
        if (!finite) fac = 0.2;
        else if (err == 0.0) fac = 5.0;
        else fac = fmin(5.0, fmax(0.2, 0.9 * pow(err, -0.2)));
        if (!accept) fac = fmin(fac, 1.0);
        double t = ctl.t[c];
        if (accept) { t += dt; ctl.t[c] = t; ctl.steps[c] += 1; }
        else ctl.rejects[c] += 1;
        const double rem = ctl.t_end - t;
        double nd = fmin(dt * fac, rem);
        int st = 0;
        if (accept && rem <= 1e-12 * fmax(fabs(ctl.t_end), 1.0)) { st = 1; nd = 0.0; }
        else if (nd <= 1e-14 * fmax(fabs(ctl.t_end), 1.0)) { st = 2; nd = 0.0; }
        ctl.dt[c] = nd;
        if (st != 0) { ctl.status[c] = st; atomicAdd(ctl.done, 1); }
        accept_s = accept ? 1 : 0;
    }
    __syncthreads();
    if (accept_s) {
        const double* k6 = e.k[6];
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            N[off + i] = Y[off + i];
            k0[off + i] = k6[off + i];     // first stage of the next step (FSAL)
        }
    }
}
} // namespace

cudaError_t batch_prep(const BatchDev& d, double* N, const pbe_batch_cell_params_t* params,
                       int stage, double c, double dt6, cudaStream_t s)
{
    const StageCombine none{};
    return prep_any(d, N, params, stage, c, dt6, none, s);
}

cudaError_t batch_sel(const BatchDev& d, const pbe_batch_cell_params_t* params, double* Sx,
                      long long total, cudaStream_t s)
{
    if (d.n_cells <= 0 || d.selection < 0 || total <= 0) return cudaErrorInvalidValue;
    const long long b = (total + 255) / 256, cap = 16LL * (d.num_sms > 0 ? d.num_sms : 1);
    launch_dep(batch_sel_kernel, dim3(static_cast<int>(b < cap ? b : cap)), 256, 0, s, 1, d, params, Sx,
               total);
    return cudaGetLastError();
}

cudaError_t batch_jvp_prep(const BatchDev& d, const double* v, const pbe_batch_cell_params_t* params,
                           cudaStream_t s)
{
    if (d.n_cells <= 0 || !d.A) return cudaErrorInvalidValue;
    switch (d.kernel < 0 ? 0 : d.kernel) {
    case 0: return launch_prep(d, batch_jvp_prep_kernel<0>, d.prep_threads, s, d, v, params);
    case 1: return launch_prep(d, batch_jvp_prep_kernel<1>, d.prep_threads, s, d, v, params);
    case 2: return launch_prep(d, batch_jvp_prep_kernel<2>, d.prep_threads, s, d, v, params);
    case 3: return launch_prep(d, batch_jvp_prep_kernel<3>, d.prep_threads, s, d, v, params);
    case 4: return launch_prep(d, batch_jvp_prep_kernel<4>, d.prep_threads, s, d, v, params);
    case 5: return launch_prep(d, batch_jvp_prep_kernel<5>, d.prep_threads, s, d, v, params);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t batch_prep_combine(const BatchDev& d, double* N, const pbe_batch_cell_params_t* params,
                               const StageCombine& sc, cudaStream_t s)
{
    return prep_any(d, N, params, kStageCombine, 0.0, 0.0, sc, s);
}

cudaError_t batch_rk45_control(const BatchDev& d, double* N, const double* Y,
                               const StageCombine& err, double* k0, const Rk45Ctl& ctl,
                               cudaStream_t s)
{
    launch_dep(rk45_control_kernel, dim3(d.n_cells), 256, 0, s, 1, d, N, Y, err, k0, ctl);
    return cudaGetLastError();
}

cudaError_t batch_main_bundles(const BatchDev& d, const double* Y,
                               const pbe_batch_cell_params_t* params, double* out,
                               bool accumulate, const int4* bundles, const int4* tasks,
                               int n_bundles, cudaStream_t s)
{
    switch (d.kernel < 0 ? 0 : d.kernel) {
    case 0: return main_k<0>(d, Y, params, out, accumulate, bundles, tasks, n_bundles, s);
    case 1: return main_k<1>(d, Y, params, out, accumulate, bundles, tasks, n_bundles, s);
    case 2: return main_k<2>(d, Y, params, out, accumulate, bundles, tasks, n_bundles, s);
    case 3: return main_k<3>(d, Y, params, out, accumulate, bundles, tasks, n_bundles, s);
    case 4: return main_k<4>(d, Y, params, out, accumulate, bundles, tasks, n_bundles, s);
    case 5: return main_k<5>(d, Y, params, out, accumulate, bundles, tasks, n_bundles, s);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t batch_main(const BatchDev& d, const double* Y, const pbe_batch_cell_params_t* params,
                       double* out, bool accumulate, cudaStream_t s)
{
    return batch_main_bundles(d, Y, params, out, accumulate, d.bundles, d.tasks, d.n_bundles, s);
}

cudaError_t cell_stage(double* N, const double* k, double* kacc, double* Y, int n, int stage,
                       double c, double dt6, cudaStream_t s)
{
    if (n <= 0) return cudaErrorInvalidValue;
    launch_dep(cell_stage_kernel, dim3((n + 255) / 256), 256, 0, s, 1, N, k, kacc, Y, n, stage, c, dt6);
    return cudaGetLastError();
}

} // namespace pbe_gb300
