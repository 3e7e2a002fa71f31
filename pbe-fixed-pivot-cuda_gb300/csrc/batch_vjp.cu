// =============================================================================
// batch_vjp.cu -- vector-Jacobian products of the batched RHS and the
// elementwise steps of the batched RK4 adjoint (sm_103a, FP64).
//
// Given lambda = dL/drhs for every cell (packed like N), one VJP is
//  * batch_vjp_prep_kernel, one cluster of CTAs per cell: x N and the lambda slopes
//    D_i = (lambda_{i+1} - lambda_i) / (x_{i+1} - x_i), the moments of N and of
//    lambda N (the -lambda_j - lambda_k part of the aggregation adjoint), the sums
//    over the bins that the lags from D0 on reduce to, and the breakage VJP of the
//    cell (per parent: Q_j = -lambda_j + sum_q bw_q P_jq from the grid's fragment
//    tables, gN_j += S_j Q_j, and the cell's dL/dS0, dL/dv_ref, dL/dalpha);
//  * batch_vjp_row_kernel (cells on geometric grids): a row per lane, the group's
//    warps splitting the lags below D0. A lag is visited twice, with the row as the
//    smaller and as the larger member (4 FP64 instructions each, Brownian + shear);
//    the lags from D0 on separate into four sums over the bins (vjp.cu derives
//    them and the rule for rows that keep them pair by pair);
//  * batch_vjp_main_kernel (other grids), persistent over bundles of row-tile
//    tasks, running the shared row-tile body (vjp_tile.cuh) on groups of T threads;
//  * batch_vjp_gfin_kernel, a warp per cell: the tasks' partials in order -> dL/dbeta.
// Every task adds its rows' dL/dN and stores its parameter partials at a fixed
// slot of its cell; every sum has a fixed order: deterministic.
// The per-lag tables are the forward's (beta-free, 1/2 on lag 0, so the VJP
// scales lag 0 by 2).
// =============================================================================
#include <type_traits>

#include "batch_scan.cuh"
#include "vjp_tile.cuh"

namespace pbe_gb300 {
namespace {

constexpr int VW = kVW;

__device__ __forceinline__ double sel_value_v(int F, double v, double S0, double v_ref,
                                              double alpha, double v_min)
{
    switch (F) {
    case 0: return selection<0>(v, S0, v_ref, alpha, v_min);
    case 1: return selection<1>(v, S0, v_ref, alpha, v_min);
    case 2: return selection<2>(v, S0, v_ref, alpha, v_min);
    default: return selection<3>(v, S0, v_ref, alpha, v_min);
    }
}

// Breakage VJP of the cell's bins [r0, r1), by one CTA: dL/dN and its part of the
// parameter gradients into part[0..2].
__device__ void cell_brk_vjp(const BatchDev& d, const BatchGridDev& gd, const double* x, const double* Nc,
                             const double* lc, double* gN, const pbe_batch_cell_params_t& P, int off,
                             int n, int r0, int r1, double* sh, double* part)
{
    const int F = d.selection, ng = gd.n;
    double p0 = 0.0, p1 = 0.0, p2 = 0.0;
    for (int j = r0 + threadIdx.x; j < r1; j += blockDim.x) {
        const double xj = x[j], Nj = Nc[j];
        const double S = d.Sx ? d.Sx[off + j]
                              : sel_value_v(F, xj, P.S0, P.v_ref, P.alpha, P.v_min);
        if (!((S != 0.0) && (Nj > kBreakageNMin))) continue;
        double Q = -lc[j];
        for (int q = 0; q < d.nq; ++q) {
            const int e = gd.woff + q * ng + j;
            const int lo = max(d.blo[e], 0);              // clipped below x[0]: lambda_0
            const int hi = min(lo + 1, n - 1);            // its weight is 0 at the cell's end
            Q = fma(d.bwlo[e], lc[lo], Q);
            Q = fma(d.bwhi[e], lc[hi], Q);
        }
        gN[off + j] += S * Q;
        const double NQ = Nj * Q;
        p0 = fma(S / P.S0, NQ, p0);
        if (F == 1) p1 = fma(-(S / P.v_ref), NQ, p1);
        if (F == 2) {
            p1 = fma(-(P.alpha * S / P.v_ref), NQ, p1);
            p2 = fma(S * log(xj / P.v_ref), NQ, p2);
        }
    }
    const double s0 = block_sum(p0, sh);
    const double s1 = block_sum(p1, sh);
    const double s2 = block_sum(p2, sh);
    if (threadIdx.x == 0) { part[0] = s0; part[1] = s1; part[2] = s2; }
}

template <int K>
__global__ void __launch_bounds__(256)
batch_vjp_prep_kernel(BatchDev d, BatchVjpDev vd, const double* __restrict__ N,
                      const double* __restrict__ lam, double* __restrict__ gN,
                      const pbe_batch_cell_params_t* __restrict__ params)
{
    const int dep = dep_wait();
    N += dep; lam += dep; gN += dep; params += dep;
    __shared__ double sh[8];
    __shared__ double msh[kPrepMaxWarps][3 * kMomN];
    __shared__ PrefixShared psm;
    const cg::cluster_group cl = cg::this_cluster();
    const int c = blockIdx.x / cl.num_blocks();
    const BatchCellDev cd = d.cells[c];
    const BatchGridDev gd = d.grids[cd.grid];
    const int off = cd.off, n = cd.n;
    const CellPart part = cell_part(n);
    const double* x = d.gx + gd.off;
    const double* a = d.ga + gd.off;
    const double* ia = d.gia + gd.off;
    const double* idx = d.ginv_dx + gd.off;
    const double* Nc = N + off;
    const double* lc = lam + off;
    double* mom = vd.mom + static_cast<size_t>(c) * kVjpMomStride;
    double* mine = mom + 16 + 18 * part.rank;
    if (d.kernel >= 0) {
        // by rows: the moments of |N|, |lambda N| and u |N| |lambda step|, parts of this
        // CTA (the sums over the bins give those of N and lambda N); by tiles: the
        // moments of N and lambda N
        const bool rows = gd.geo != 0 && vd.rows != 0;
        double m[3][kMomN];
#pragma unroll
        for (int g = 0; g < 3; ++g)
#pragma unroll
            for (int q = 0; q < kMomN; ++q) m[g][q] = 0.0;
        for (int i = part.r0 + threadIdx.x; i < part.r1; i += blockDim.x) {
            const double xi = x[i], Ni = Nc[i], li = lc[i];
            double dl = 0.0, Di = 0.0, u = 0.0;
            if (i < n - 1) {
                dl = lc[i + 1] - li;
                Di = dl / (x[i + 1] - xi);
                u = 1.1102230246251565e-16 * (x[i + 1] * idx[i]);
            }
            vd.h[off + i] = xi * Ni;
            vd.D[off + i] = Di;
            const double w[kMomN] = {(K >= 3) ? ia[i] : 0.0, 1.0, (K >= 3) ? a[i] : 0.0,
                                     (K >= 4) ? a[i] * a[i] : 0.0, xi};
            double v[3] = {Ni, li * Ni, 0.0};
            if (rows) {
                v[0] = fabs(v[0]);
                v[1] = fabs(v[1]);
                v[2] = u * fabs(dl * Ni);
            }
#pragma unroll
            for (int g = 0; g < 3; ++g)
#pragma unroll
                for (int q = 0; q < kMomN; ++q)
                    if (need_moment<K>(q)) m[g][q] = fma(w[q], v[g], m[g][q]);
        }
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
        for (int g = 0; g < 3; ++g)
#pragma unroll
            for (int q = 0; q < kMomN; ++q) {
                const double s = need_moment<K>(q) ? warp_sum(m[g][q]) : 0.0;
                if (lane == 0) msh[w][kMomN * g + q] = s;
            }
        __syncthreads();
        if (threadIdx.x < 3 * kMomN) {
            double s = 0.0;
            for (int v = 0; v < static_cast<int>(blockDim.x >> 5); ++v) s += msh[v][threadIdx.x];
            mine[threadIdx.x] = s;
        }
        cl.sync();                         // D and the parts of the whole cell
        // the CTAs' parts together: by tiles in slots 0.., by rows in CTA 0's own
        if (part.rank == 0 && threadIdx.x < (rows ? 3 : 2) * kMomN) {
            double s = 0.0;
            for (int r = 0; r < part.ranks; ++r) s += mom[16 + 18 * r + threadIdx.x];
            mom[(rows ? 16 : 0) + threadIdx.x] = s;
        }
        if (rows) {
            double* pre = vd.pre + off;
            const double* D = vd.D + off;
            cell_scan<K, false>(x, a, ia,
                                [&](int i, double xi, double& y, double& z) { y = Nc[i]; z = y * mantissa_of(xi); },
                                part, n, psm, pre, d.total, mom);
            cl.sync();                         // the shared totals are read by every CTA
            cell_scan<K, true>(x, a, ia,
                               [&](int i, double xi, double& y, double& z) {
                                   y = lc[i] * Nc[i];
                                   z = Nc[i] * scalbn(D[i], exponent_of(xi));
                               },
                               part, n, psm, pre + 2 * kMomN * d.total, d.total, mom + 5);
            cl.sync();
        }
    }
    if (d.nq > 0)
        cell_brk_vjp(d, gd, x, Nc, lc, gN, params[c], off, n, part.r0, part.r1, sh, mine + 15);
}

// ---------------------------------------------------------------------------
// Row blocks of cells on geometric grids.
// ---------------------------------------------------------------------------
struct RowShared {
    double red[kMaxGroups][2][32];        // per-warp sums of every row
    double ex[kMaxGroups][2][32];         // exact rows: their sums from D0 on (per group's first warp)
};

// The two partner sums of row m over the lags d0, d0 + step, .. below d1: A0 (beta0 or Brownian), A1
// (shear, over x_m), as vjp_tile.cuh.
template <int K, bool LAG0>
__device__ __forceinline__ void row_lags(const VjpCellView& v, int m, bool valid, int d0, int d1, int step,
                                         double lamlast, double& A0, double& A1)
{
    const int n = v.n;
    const double xm = valid ? __ldg(v.x + m) : 1.0;
    const EwOperandA ma = ew_operand_a(xm);
    const EwOperandB mb = ew_operand_b(xm);
    for (int d = d0; d < d1; d += step) {
        const int L = __ldg(v.Ld + d);
        const double Bf = ((K == 3 || K == 5) ? __ldg(v.Bf + d) : 0.0) * (LAG0 ? v.lag0_scale : 1.0);
        const double Sf = ((K >= 4) ? __ldg(v.Sf + d) : 0.0) * (LAG0 ? v.lag0_scale : 1.0);
        const double Sl = (K >= 4) ? __ldg(v.Sl + d) : 0.0;
        auto visit = [&](int k, int lo, double num, double S) {
            double P = lamlast;
            if (lo < n - 1) P = fma(num, __ldg(v.D + lo), __ldg(v.lam + lo));
            if constexpr (K == 2) {
                A0 = fma(P, __ldg(v.h + k), A0);
            } else {
                const double Nk = __ldg(v.N + k);
                if constexpr (K == 0) A0 = fma(P, Nk, A0);
                if constexpr (K == 1) { A0 = fma(P, Nk, A0); A1 = fma(P, __ldg(v.h + k), A1); }
                if constexpr (K >= 3) {
                    const double t = P * Nk;
                    if constexpr (K == 3 || K == 5) A0 = fma(t, Bf, A0);
                    if constexpr (K == 4 || K == 5) A1 = fma(t, S, A1);
                }
            }
        };
        const int ku = m + d;                          // m the smaller member
        if (valid && ku < n) {
            const int lo = (L >= kLagClipAll) ? n : m + L;
            double num = 0.0;
            if (lo < n - 1)
                num = sum_minus_scaled_dec(ew_operand_a(__ldg(v.x + ku)), mb, ew_operand_c(__ldg(v.x + lo), 0));
            visit(ku, lo, num, Sf);
        }
        const int kl = m - d;                          // m the larger member
        if (!LAG0 && valid && kl >= 0) {
            const int lo = (L >= kLagClipAll) ? n : m + L - d;
            double num = 0.0;
            if (lo < n - 1) num = sum_minus_scaled_pre(ma, __ldg(v.x + kl), ew_operand_c(__ldg(v.x + lo), 0));
            visit(kl, lo, num, Sl);
        }
    }
}

// The lags from Dm on of row m pair by pair, by one warp; with the kernel factor's
// power of x_m taken in as the sums of row_lags (A1 over x_m). Valid in every lane.
template <int K>
__device__ __forceinline__ void row_exact(const VjpCellView& v, int m, int Dm, double lamlast, double& A0,
                                          double& A1)
{
    const int n = v.n, lane = threadIdx.x & 31;
    const double xm = __ldg(v.x + m), Dk = v.D[m], lm = __ldg(v.lam + m);
    const EwOperandA ma = ew_operand_a(xm);
    const EwOperandB mb = ew_operand_b(xm);
    const EwOperandC mc = ew_operand_c(xm, 0);
    double s0 = 0.0, s1 = 0.0;
    auto add = [&](int k, int d, double P, double S) {
        const double Nk = __ldg(v.N + k);
        if constexpr (K == 0) s0 = fma(P, Nk, s0);
        if constexpr (K == 1) { s0 = fma(P, Nk, s0); s1 = fma(P, v.h[k], s1); }
        if constexpr (K == 2) s0 = fma(P, v.h[k], s0);
        if constexpr (K == 3 || K == 5) s0 = fma(P * Nk, __ldg(v.Bf + d), s0);
        if constexpr (K == 4 || K == 5) s1 = fma(P * Nk, S, s1);
    };
#pragma unroll 4
    for (int j = lane; j <= m - Dm; j += 32) {
        const double P = m < n - 1 ? fma(sum_minus_scaled_pre(ma, __ldg(v.x + j), mc), Dk, lm) : lamlast;
        add(j, m - j, P, K >= 4 ? __ldg(v.Sl + m - j) : 0.0);
    }
#pragma unroll 4
    for (int k = m + Dm + lane; k < n; k += 32) {
        const double xk = __ldg(v.x + k);
        double P = __ldg(v.lam + k);
        if (k < n - 1)
            P = fma(sum_minus_scaled_dec(ew_operand_a(xk), mb, ew_operand_c(xk, 0)), v.D[k], P);
        add(k, k - m, P, K >= 4 ? __ldg(v.Sf + k - m) : 0.0);
    }
    A0 = warp_sum(s0);
    A1 = warp_sum(s1);
}

template <int K>
__global__ void __launch_bounds__(kMainThreads, 3)
batch_vjp_row_kernel(BatchDev d, BatchVjpDev vd, const double* __restrict__ N,
                     const double* __restrict__ lam, double* __restrict__ gN,
                     const pbe_batch_cell_params_t* __restrict__ params)
{
    const int dep = dep_wait();
    N += dep; lam += dep; gN += dep; params += dep;
    __shared__ RowShared sm;
    const int4 bu = vd.rbundles[blockIdx.x];  // {first task, tasks, group size, 0}
    const int T = bu.z;
    const int g = threadIdx.x / T;
    if (g >= bu.y) return;                    // whole groups
    const TileGroup G{g, static_cast<int>(threadIdx.x) - g * T, T};
    const int4 tk = vd.rtasks[bu.x + g];      // {cell, first row, slot, 0}
    const int c = tk.x, I = tk.y;
    const BatchCellDev cd = d.cells[c];
    const BatchGridDev gd = d.grids[cd.grid];
    const int n = cd.n, off = cd.off;
    const int l = G.lane & 31, w = G.lane >> 5, nw = G.T >> 5;
    VjpCellView v;
    v.x = d.gx + gd.off;
    v.N = N + off;
    v.h = vd.h + off;
    v.lam = lam + off;
    v.D = vd.D + off;
    v.a = d.ga + gd.off; v.ia = d.gia + gd.off;
    v.Bf = d.gBd + gd.off; v.Sf = d.gSd + gd.off; v.Sl = d.gSl + gd.off; v.Ld = d.gLd + gd.off;
    v.lag0_scale = 2.0;
    v.n = n;
    v.geo = true;
    const double lamlast = __ldg(v.lam + n - 1);
    const int m = I + l;
    const bool valid = m < n;
    const int Dm = min(gd.D0, n);
    // the lags below D0 (none beyond the last row's partners), interleaved over the
    // warps: long lags have one of their two visits, or none, inside the cell
    const int lags = min(Dm, max(n - I, min(I + 32, n)));
    double A0 = 0.0, A1 = 0.0;
    if (w == 0) row_lags<K, true>(v, m, valid, 0, 1, 1, lamlast, A0, A1);
    row_lags<K, false>(v, m, valid, w > 0 ? w : nw, lags, nw, lamlast, A0, A1);
    if (nw > 1) {
        sm.red[G.g * nw + w][0][l] = A0;
        sm.red[G.g * nw + w][1][l] = A1;
    }
    // rows that take the lags from D0 on pair by pair (vjp.cu), spread over the warps
    const double* mom = vd.mom + static_cast<size_t>(c) * kVjpMomStride;
    const pbe_batch_cell_params_t P = params[c];
    const double xm = valid ? __ldg(v.x + m) : 1.0, am = valid ? __ldg(v.a + m) : 1.0;
    const double iam = valid ? __ldg(v.ia + m) : 1.0, lm = valid ? __ldg(v.lam + m) : 0.0;
    bool ex = false;
    if (valid && (m >= Dm || m + Dm < n)) {
        const double c0 = fabs(P.beta0), c1 = fabs(P.beta_br), c2 = fabs(P.beta_sh);
        double S[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) S[q] = death_factor<K>(xm, am, iam, mom + 16 + 5 * q, c0, c1, c2);
        double err = S[2];
        if (m < n - 1)
            err = fma(1.1102230246251565e-16 * (__ldg(v.x + m + 1) * __ldg(d.ginv_dx + gd.off + m)) *
                      fabs(__ldg(v.lam + m + 1)), S[0], err);
        ex = err > kVjpGuard * fma(fabs(lm), S[0], S[1]);
    }
    const unsigned exact = __ballot_sync(0xffffffffu, ex);
    int turn = 0;
    for (unsigned em = exact; em != 0u; em &= em - 1u) {
        const int le = __ffs(em) - 1;
        if (turn == w) {
            double e0, e1;
            row_exact<K>(v, I + le, Dm, lamlast, e0, e1);
            if (l == 0) { sm.ex[G.g * nw][0][le] = e0; sm.ex[G.g * nw][1][le] = e1; }
        }
        turn = turn + 1 == nw ? 0 : turn + 1;
    }
    G.sync();
    if (w != 0) return;
    for (int q = 1; q < nw; ++q) {
        A0 += sm.red[G.g * nw + q][0][l];
        A1 += sm.red[G.g * nw + q][1][l];
    }
    double gB = 0.0, gS = 0.0;
    if (valid) {
        const double Nm = __ldg(v.N + m);
        double T0 = 0.0, T1 = 0.0;             // the lags from D0 on, beta0 / Brownian and shear parts
        if ((exact >> l) & 1u) {
            A0 += sm.ex[G.g * nw][0][l];
            A1 += sm.ex[G.g * nw][1][l];
        } else {
            const int Em = exponent_of(xm);
            const double* pre = vd.pre + off;
            auto sums = [&](int grp, int i, double* o) {
#pragma unroll
                for (int q = 0; q < kMomN; ++q)
                    o[q] = need_moment<K>(q) ? pre[(grp * kMomN + q) * d.total + i] : 0.0;
            };
            auto part = [&](auto X, const double* o) { return moment_factor<K, decltype(X)::value>(xm, am, iam, o); };
            using B = std::integral_constant<int, 0>;
            using Sh = std::integral_constant<int, 1>;
            double s[kMomN], t[kMomN];
            if (m >= Dm) {                     // the larger member
                sums(0, m - Dm, s);
                sums(1, m - Dm, t);
                const double Dn = scalbn(v.D[m], Em);
                const int sh = exponent_of(__ldg(v.x + m - Dm)) - Em;
                if constexpr (K != 4) T0 += fma(lm, part(B{}, s), scale_down(Dn * part(B{}, t), sh));
                if constexpr (K >= 4) T1 += fma(lm, part(Sh{}, s), scale_down(Dn * part(Sh{}, t), sh));
            }
            if (m + Dm < n) {                  // the smaller member
                sums(2, m + Dm, s);
                sums(3, m + Dm, t);
                const double xmm = mantissa_of(xm);
                const int sh = Em - exponent_of(__ldg(v.x + m + Dm));
                if constexpr (K != 4) T0 += part(B{}, s) + scale_down(xmm * part(B{}, t), sh);
                if constexpr (K >= 4) T1 += part(Sh{}, s) + scale_down(xmm * part(Sh{}, t), sh);
            }
        }
        double AX0 = 0.0, AX1 = 0.0;           // A for beta0 / Brownian, and for shear
        if constexpr (K != 4) {
            double Tv = A0;
            if constexpr (K == 1) Tv = fma(xm, A0, A1);
            if constexpr (K == 2) Tv = xm * A0;
            AX0 = (Tv + T0) - fma(lm, moment_factor<K, 0>(xm, am, iam, mom), moment_factor<K, 0>(xm, am, iam, mom + 5));
        }
        if constexpr (K >= 4)
            AX1 = fma(xm, A1, T1) - fma(lm, moment_factor<K, 1>(xm, am, iam, mom), moment_factor<K, 1>(xm, am, iam, mom + 5));
        double gr;
        if constexpr (K <= 2) gr = P.beta0 * AX0;
        else if constexpr (K == 3) gr = P.beta_br * AX0;
        else if constexpr (K == 4) gr = P.beta_sh * AX1;
        else gr = fma(P.beta_br, AX0, P.beta_sh * AX1);
        gN[off + m] += gr;
        gB = 0.5 * Nm * AX0;
        gS = 0.5 * Nm * AX1;
    }
    const double s0 = warp_sum(gB), s1 = warp_sum(gS);
    if (l == 0) {
        vd.tpart[2 * tk.z + 0] = s0;
        vd.tpart[2 * tk.z + 1] = s1;
    }
}

template <int K>
__device__ void batch_vjp_task(const BatchDev& d, const BatchVjpDev& vd, const double* N,
                               const double* lam, double* gN,
                               const pbe_batch_cell_params_t* __restrict__ params, int4 tk,
                               double* red, VjpShared& sm, const TileGroup& G)
{
    const int c = tk.x, I = tk.y;
    const BatchCellDev cd = d.cells[c];
    const BatchGridDev gd = d.grids[cd.grid];
    const int n = cd.n;
    VjpCellView v;
    v.x = d.gx + gd.off;
    v.N = N + cd.off;
    v.h = vd.h + cd.off;
    v.lam = lam + cd.off;
    v.D = vd.D + cd.off;
    v.a = d.ga + gd.off; v.ia = d.gia + gd.off;
    v.Bf = d.gBd + gd.off; v.Sf = d.gSd + gd.off; v.Sl = d.gSl + gd.off; v.Ld = d.gLd + gd.off;
    v.lag0_scale = 2.0;
    v.n = n;
    v.geo = gd.geo != 0;
    // epilogue values through shared memory (no registers held in the loops)
    if (G.lane < 16) {
        const int l = G.lane;
        double val = 0.0;
        if (l < 10) val = vd.mom[static_cast<size_t>(c) * kVjpMomStride + l];
        else if (l == 10) val = params[c].beta0;
        else if (l == 11) val = params[c].beta_br;
        else if (l == 12) val = params[c].beta_sh;
        sm.cinfo[G.g][l] = val;
    }
    vjp_tile_accumulate<K>(v, I, 0, n, red, sm, G);    // syncs the group first
    const int tmax = min(VW, n - I);
    if (G.lane < VW) {
        double gB = 0.0, gS = 0.0;
        if (G.lane < tmax) {
            const double* ci = sm.cinfo[G.g];
            double g;
            vjp_tile_row<K>(v, I + G.lane, G.lane, sm.fin[G.g], ci, ci + 5, ci[10], ci[11], ci[12],
                            g, gB, gS);
            gN[cd.off + I + G.lane] += g;
        }
        sm.gsh[G.g][G.lane][0] = gB;
        sm.gsh[G.g][G.lane][1] = gS;
    }
    G.sync();
    if (G.lane == 0) {
        double s0 = 0.0, s1 = 0.0;
        for (int t = 0; t < VW; ++t) { s0 += sm.gsh[G.g][t][0]; s1 += sm.gsh[G.g][t][1]; }
        vd.tpart[2 * tk.z + 0] = s0;
        vd.tpart[2 * tk.z + 1] = s1;
    }
}

template <int K>
__global__ void __launch_bounds__(kMainThreads, 2)
batch_vjp_main_kernel(BatchDev d, BatchVjpDev vd, const double* __restrict__ N,
                      const double* __restrict__ lam, double* __restrict__ gN,
                      const pbe_batch_cell_params_t* __restrict__ params)
{
    const int dep = dep_wait();
    N += dep; lam += dep; gN += dep; params += dep;
    extern __shared__ double red[];     // [kVRows][kMainThreads]
    __shared__ VjpShared sm;
    __shared__ int s_b;
    const int tid = threadIdx.x;
    for (;;) {
        if (tid == 0) s_b = atomicAdd(vd.counter, 1);
        __syncthreads();
        const int b = s_b;
        __syncthreads();
        if (b >= vd.n_bundles) break;
        const int4 bu = vd.bundles[b];
        const int T = bu.z;
        const int g = tid / T;
        if (g < bu.y) {
            const TileGroup G{g, tid - g * T, T};
            batch_vjp_task<K>(d, vd, N, lam, gN, params, vd.tasks[bu.x + g], red + g * T, sm, G);
        }
        __syncthreads();
    }
}

// Parameter gradients, a warp per cell: the tasks' partials of dL/dbeta (lanes over
// the tasks, fixed butterfly) and the prep CTAs' breakage parts in order.
template <int K>
__global__ void __launch_bounds__(256)
batch_vjp_gfin_kernel(BatchDev d, BatchVjpDev vd, double* __restrict__ gparams)
{
    const int dep = dep_wait();
    gparams += dep;
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, l = threadIdx.x & 31;
    if (c >= d.n_cells) return;
    if (d.kernel >= 0) {
        double s0 = 0.0, s1 = 0.0;
        for (int t = vd.tile_off[c] + l; t < vd.tile_off[c + 1]; t += 32) {
            s0 += vd.tpart[2 * t];
            s1 += vd.tpart[2 * t + 1];
        }
        s0 = warp_sum(s0);
        s1 = warp_sum(s1);
        if (l == 0) {
            if constexpr (K <= 2) gparams[c * 8 + 0] += s0;
            if constexpr (K == 3 || K == 5) gparams[c * 8 + 1] += s0;
            if constexpr (K == 4 || K == 5) gparams[c * 8 + 2] += s1;
        }
    }
    if (d.nq > 0 && l < 3) {
        const double* p = vd.mom + static_cast<size_t>(c) * kVjpMomStride + 16 + 15 + l;
        double s = 0.0;
        for (int r = 0; r < d.prep_ranks; ++r) s += p[18 * r];
        gparams[c * 8 + 3 + l] += s;
    }
}

template <int K>
cudaError_t vjp_k(const BatchDev& d, const BatchVjpDev& vd, const double* N, const double* lam,
                  double* gN, double* gparams, const pbe_batch_cell_params_t* params,
                  cudaStream_t s)
{
    cudaError_t e = launch_prep(d, batch_vjp_prep_kernel<K>, d.vjp_prep_threads, s, d, vd, N, lam, gN, params);
    if (e != cudaSuccess) return e;
    if (d.kernel >= 0) {
        if (vd.n_rbundles > 0)
            launch_dep(batch_vjp_row_kernel<K>, dim3(vd.n_rbundles), kMainThreads, 0, s, 1, d, vd, N, lam,
                       gN, params);
        if (vd.n_bundles > 0) {
            e = cudaMemsetAsync(vd.counter, 0, sizeof(int), s);
            if (e != cudaSuccess) return e;
            const int grid = vd.n_bundles < 2 * d.num_sms ? vd.n_bundles : 2 * d.num_sms;
            const size_t smem = sizeof(double) * kVRows * kMainThreads;
            launch_dep(batch_vjp_main_kernel<K>, dim3(grid), kMainThreads, smem, s, 1, d, vd, N, lam, gN,
                       params);
        }
    }
    launch_dep(batch_vjp_gfin_kernel<K>, dim3((d.n_cells + 7) / 8), 256, 0, s, 1, d, vd, gparams);
    return cudaGetLastError();
}

template <int K>
cudaError_t vjp_attr_k()
{
    return cudaFuncSetAttribute(batch_vjp_main_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(sizeof(double) * kVRows * kMainThreads));
}

// a = w lam' (+ c mu), mu = 0
__global__ void __launch_bounds__(256)
adj_coeff_kernel(double* a, const double* lp, double* mu, double w, double c, long long n,
                 int first)
{
    const int dep = dep_wait();
    lp += dep;
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    a[i] = first ? w * lp[i] : fma(c, mu[i], w * lp[i]);
    mu[i] = 0.0;
}

__global__ void __launch_bounds__(256) adj_sum_kernel(double* lsum, const double* mu, long long n)
{
    const int dep = dep_wait();
    mu += dep;
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) lsum[i] += mu[i];
}

} // namespace

cudaError_t batch_vjp_setup(int kernel)
{
    switch (kernel < 0 ? 0 : kernel) {
    case 0: return vjp_attr_k<0>();
    case 1: return vjp_attr_k<1>();
    case 2: return vjp_attr_k<2>();
    case 3: return vjp_attr_k<3>();
    case 4: return vjp_attr_k<4>();
    case 5: return vjp_attr_k<5>();
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t batch_vjp(const BatchDev& d, const BatchVjpDev& vd, const double* N, const double* lam,
                      double* gN, double* gparams, const pbe_batch_cell_params_t* params,
                      cudaStream_t s)
{
    switch (d.kernel < 0 ? 0 : d.kernel) {
    case 0: return vjp_k<0>(d, vd, N, lam, gN, gparams, params, s);
    case 1: return vjp_k<1>(d, vd, N, lam, gN, gparams, params, s);
    case 2: return vjp_k<2>(d, vd, N, lam, gN, gparams, params, s);
    case 3: return vjp_k<3>(d, vd, N, lam, gN, gparams, params, s);
    case 4: return vjp_k<4>(d, vd, N, lam, gN, gparams, params, s);
    case 5: return vjp_k<5>(d, vd, N, lam, gN, gparams, params, s);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t batch_adj_coeff(double* a, const double* lp, double* mu, double w, double c,
                            long long n, bool first, cudaStream_t s)
{
    launch_dep(adj_coeff_kernel, dim3(static_cast<int>((n + 255) / 256)), 256, 0, s, 1, a, lp, mu, w, c, n,
               first ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t batch_adj_sum(double* lsum, const double* mu, long long n, cudaStream_t s)
{
    launch_dep(adj_sum_kernel, dim3(static_cast<int>((n + 255) / 256)), 256, 0, s, 1, lsum, mu, n);
    return cudaGetLastError();
}

} // namespace pbe_gb300
