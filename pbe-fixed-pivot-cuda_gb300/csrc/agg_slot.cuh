// =============================================================================
// agg_slot.cuh -- aggregation pair sums with one output slot per lane, for any
// grid: the pair work of the batched kernel (batch_kernels.cu) and, on grids that
// are not geometric, of the single-instance kernel (agg_lane.cuh).
//
// Slot s collects the pairs (j <= k) whose bracket is lo = s: R_s = sum rate,
// TH_s = sum rate (fl(x_j + x_k) - x_s) 2^St_s, St_s = -exponent of x_s
// (reference src/aggregation_kernels.cuh:145-239, regrouped; aggregation.cu has
// the derivation). The pairs of a slot split in two:
//
//  * k = s, j < jcut(s): the sum still lands below x_{s+1}, so the larger member
//    is the slot's own bin. beta is a sum of products of powers of x_j and x_k,
//    so these sums come from prefix moments over j (cell_prefix):
//      R += N_s death_factor(x_s; P),  TH += N_s death_factor(x_s; T),
//    P, T the moments of N and x N over j < jcut(s). On a geometric grid
//    jcut(s) = s - D0 + 1 (lags from D0 on); on any other a table per grid. With
//    q sections an octave D0 is about q log2(1.44 q): 10 lags of n at q = 4, 176
//    at q = 32. Why the sums may be separated, and when not (mom_exact_slot):
//    agg_lane.cuh.
//  * the rest pair by pair (slot_pairs_geo: the lags below D0, runs of lags with
//    one bracket offset sharing their larger member; slot_pairs_any: a monotone
//    walk over the rows j).
//
// NP = 1: the RHS. NP = 2: its Jacobian-vector product, T(N, v) + T(v, N) with
// T(a, b) the pair sum with rate beta a_j b_k, both in one pass over the pairs
// (they share brackets and weights).
// =============================================================================
#pragma once

#include "agg_rates.cuh"
#include "agg_moments.cuh"

namespace pbe_gb300 {

// The grid of a cell (its first n pivots) and the cell's coefficients. The lag
// factors carry the coefficients in single-instance use (Nj = a_j, Hj = x_j a_j
// then), and not in batched use.
struct SlotGrid {
    const double* x;
    const double* a;        // x^(1/3)
    const double* ia;       // x^(-1/3)
    const double* inv_dx;
    const double* Bd;       // lag factors, c_d = 1/2 on lag 0, no beta (geometric grids)
    const double* Sd;
    const int* Ld;          // bracket offset of a lag
    const int* J0;          // first j with fl(x_j + x_s) >= x_{s+1} (other grids)
    int n, D0;
    bool geo;
    double b0, bbr, bsh;
};

// One bilinear pass: j side a, k side b. Nj = beta a_j and Hj = beta x_j a_j carry
// the cell's coefficient (the lag factors do not); Aj = a_j and AHj = x_j a_j for
// the walk on other grids.
struct SlotPass {
    const double* Nj;
    const double* Hj;
    const double* Aj;
    const double* AHj;
    const double* Nk;
    const double* Hk;
};

// Rows j < slot_cut(s) with k = s belong to the prefix sums.
__device__ __forceinline__ int slot_cut(const SlotGrid& g, int s)
{
    if (g.geo) return max(0, s - g.D0 + 1);
    // the clipped slot n - 1 takes every j < n - 1; the diagonal pair is never in
    return s >= g.n - 1 ? s : min(g.J0[s], s);
}

// Lags [d0, d1) of slot s on a geometric grid (uniform d0, d1, smax across the
// warp; Ld nondecreasing). pc: the slot's pivot, decoded.
template <int K, int NP>
__device__ __forceinline__ void slot_pairs_geo(const SlotGrid& g, const SlotPass* p, int s, bool slot,
                                               int smax, int d0, int d1, const EwOperandC& pc,
                                               double& R, double& TH)
{
    EwOperandA pa = ew_operand_a(0.0);               // x_k of the current run
    double Q[NP], QT[NP], F[NP], hk[NP];
#pragma unroll
    for (int q = 0; q < NP; ++q) { Q[q] = QT[q] = F[q] = hk[q] = 0.0; }
    int e_cur = -1;
    for (int d = d0; d < d1; ++d) {
        const int L = g.Ld[d];
        if (L > smax) break;
        const int e = L - d;
        if (e != e_cur) {                              // uniform across the warp
            e_cur = e;
            const int k = s - e;
            const bool kin = slot && k >= 0;
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                if constexpr (K != 1) {
                    R = fma(F[q], Q[q], R);
                    TH = fma(F[q], QT[q], TH);
                    Q[q] = 0.0;
                    QT[q] = 0.0;
                }
                F[q] = kin ? (K == 2 ? p[q].Hk : p[q].Nk)[k] : 0.0;
                if constexpr (K == 1) hk[q] = kin ? p[q].Hk[k] : 0.0;
            }
            pa = ew_operand_a(kin ? __ldg(g.x + k) : 0.0);
        }
        const double B = g.Bd[d], S = g.Sd[d];
        const int j = s - L;
        if (slot && j >= 0) {
            const double th = sum_minus_scaled_pre(pa, __ldg(g.x + j), pc);
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                const double Nj = (K == 2 || K == 4) ? 0.0 : p[q].Nj[j];
                const double hj = NeedH<K>::j ? p[q].Hj[j] : 0.0;
                if constexpr (K != 1) {
                    const double r = q_slot<K>(B, S, Nj, hj);
                    Q[q] += r;
                    QT[q] = fma(r, th, QT[q]);
                } else {
                    const double r = rate_geo<1>(B, S, Nj, hj, F[q], hk[q]);
                    R += r;
                    TH = fma(r, th, TH);
                }
            }
        }
    }
    if constexpr (K != 1) {
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            R = fma(F[q], Q[q], R);
            TH = fma(F[q], QT[q], TH);
        }
    }
}

// beta(x_j, x_k) of one row j as a polynomial in a_k, 1/a_k (no minus signs in it):
//   Brownian  beta_br (a_j/a_k + a_k/a_j + 2),
//   shear     beta_sh (a_j + a_k)^3 = beta_sh (x_j + 3 a_j^2 a_k + 3 a_j a_k^2 + a_k^3).
// Five FP64 instructions a row and up to four a pair, where a pair alone takes eight.
template <int K>
struct RowBeta {
    double c0, c1, c2, c3, ci;
    __device__ __forceinline__ RowBeta(const SlotGrid& g, int j)
    {
        c0 = c1 = c2 = c3 = ci = 0.0;
        if constexpr (K >= 3) {
            const double aj = g.a[j];
            if constexpr (K == 3 || K == 5) { c0 = 2.0 * g.bbr; c1 = g.bbr * g.ia[j]; ci = g.bbr * aj; }
            if constexpr (K == 4 || K == 5) {
                c3 = g.bsh;
                c2 = (3.0 * g.bsh) * aj;
                c1 = fma(c2, aj, c1);
                c0 = fma(g.bsh, __ldg(g.x + j), c0);
            }
        }
    }
    __device__ __forceinline__ double operator()(double ak, double iak) const
    {
        if constexpr (K == 3) return fma(ci, iak, fma(c1, ak, c0));
        const double shear = fma(ak, fma(ak, fma(ak, c3, c2), c1), c0);
        if constexpr (K == 4) return shear;
        return fma(ci, iak, shear);
    }
};

// beta(x_j, x_k) a_j b_k from per-bin values, every pass (row: the row's RowBeta).
template <int K, int NP>
__device__ __forceinline__ double slot_rate_any(const SlotGrid& g, const SlotPass* p, const RowBeta<K>& row, int j,
                                                int k)
{
    double beta = 0.0;
    if constexpr (K >= 3) beta = row(g.a[k], g.ia[k]);
    double r = 0.0;
#pragma unroll
    for (int q = 0; q < NP; ++q) {
        double v;
        if constexpr (K == 0) v = (g.b0 * p[q].Aj[j]) * p[q].Nk[k];
        else if constexpr (K == 1) v = g.b0 * fma(p[q].AHj[j], p[q].Nk[k], p[q].Aj[j] * p[q].Hk[k]);
        else if constexpr (K == 2) v = (g.b0 * p[q].AHj[j]) * p[q].Hk[k];
        else v = (beta * p[q].Aj[j]) * p[q].Nk[k];
        r = q == 0 ? v : r + v;
    }
    return j == k ? 0.5 * r : r;
}

// First j <= s + 1 with 2 x_j >= x_{s+1}, sought from `guess`: from there on a row has
// no larger member with which it stays below x_{s+1}. On a linear grid that is half of
// the rows.
__device__ __forceinline__ int slot_rows_end(const double* __restrict__ x, int s, int guess)
{
    const long long top = dbits(__ldg(x + s + 1));
    auto end = [&](int j) { return dbits(2.0 * __ldg(x + j)) >= top; };
    int lo, hi, step = 1;                              // lo: not yet (or -1); hi: 2 x_hi >= x_{s+1}
    const int g = min(max(guess, 0), s);
    if (end(g)) {
        hi = g;
        while (hi - step > 0 && end(hi - step)) { hi -= step; step <<= 1; }
        lo = hi - step > 0 ? hi - step : -1;
    } else {
        lo = g;
        while (lo + step <= s && !end(lo + step)) { lo += step; step <<= 1; }
        hi = min(s + 1, lo + step);
    }
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (end(mid)) hi = mid; else lo = mid;
    }
    return hi;
}

// Share w of nw of slot s's rows on any grid, but for the pairs of the prefix
// sums: for each row j the larger members k with x_s <= fl(x_j + x_k) < x_{s+1}
// lie in one run below the previous row's, so a lane walks down k as j grows. Rows
// from jt on have none (slot_rows_end, or s + 1).
template <int K, int NP>
__device__ __forceinline__ void slot_pairs_any(const SlotGrid& g, const SlotPass* p, int s, bool slot,
                                               int jt, int w, int nw, double& R, double& TH)
{
    if (!slot) return;
    const double* __restrict__ x = g.x;
    const double xs = __ldg(x + s), xu = __ldg(x + s + 1);
    const long long lo = dbits(xs), hi = dbits(xu);
    const int St20 = -exponent_of(xs) * (1 << 20);
    const int Js = slot_cut(g, s);
    const int j0 = s > 0 ? min(Js, slot_cut(g, s - 1)) : Js;
    const int per = (max(0, jt - j0) + nw - 1) / nw;
    const int ja = j0 + w * per, jb = min(jt, ja + per);
    if (ja >= jb) return;
    // last k <= s with fl(x_ja + x_k) < x_{s+1} (below ja: the rows are done)
    const double xa = __ldg(x + ja);
    int k = s, kb = ja - 1;
    while (kb < k) {
        const int mid = (kb + k + 1) >> 1;
        if (dbits(xa + __ldg(x + mid)) < hi) kb = mid; else k = mid - 1;
    }
    for (int j = ja; j < jb && k >= j; ++j) {
        const double xj = __ldg(x + j);
        double v = xj + __ldg(x + k);
        while (dbits(v) >= hi && --k >= j) v = xj + __ldg(x + k);
        if (k < j) break;
        const RowBeta<K> row(g, j);
        for (int q = k; dbits(v) >= lo;) {
            if (q != s || j >= Js) {                   // (else in the prefix sums)
                const double r = slot_rate_any<K, NP>(g, p, row, j, q);
                R += r;
                TH = fma(r, scale_pow2(v - xs, St20), TH);
            }
            if (--q < j) break;
            v = xj + __ldg(x + q);
        }
    }
}

// Thread tid of nt's share of the prefix part of slot s, pair by pair: for the
// slots of mom_exact_slot. U: pairs in flight.
template <int K, int NP, int U = 1>
__device__ __forceinline__ void slot_exact_part(const SlotGrid& g, const SlotPass* p, int s, int tid,
                                                int nt, double& r, double& t)
{
    const double xs = __ldg(g.x + s);
    const int St = -exponent_of(xs);
    const EwOperandA pa = ew_operand_a(xs);
    const EwOperandC pc = ew_operand_c(xs, St);
    const int cut = slot_cut(g, s);
    r = 0.0;
    t = 0.0;
#pragma unroll U
    for (int j = tid; j < cut; j += nt) {
        double rate, th;
        if (g.geo) {
            const int d = s - j;
            rate = 0.0;
#pragma unroll
            for (int q = 0; q < NP; ++q)
                rate += rate_geo<K>(g.Bd[d], g.Sd[d], p[q].Nj[j],
                                    NeedH<K>::j ? p[q].Hj[j] : 0.0, p[q].Nk[s],
                                    NeedH<K>::k ? p[q].Hk[s] : 0.0);
            th = sum_minus_scaled_pre(pa, __ldg(g.x + j), pc);
        } else {
            rate = slot_rate_any<K, NP>(g, p, RowBeta<K>(g, j), j, s);
            th = scale_pow2((__ldg(g.x + j) + xs) - xs, St * (1 << 20));
        }
        r += rate;
        t = fma(rate, th, t);
    }
}

// The same by one warp, summed by a fixed butterfly. Valid in every lane.
template <int K, int NP, int U>
__device__ __forceinline__ void slot_exact(const SlotGrid& g, const SlotPass* p, int s, double& R,
                                           double& TH)
{
    double r, t;
    slot_exact_part<K, NP, U>(g, p, s, threadIdx.x & 31, 32, r, t);
    R = warp_sum(r);
    TH = warp_sum(t);
}

// Warp w of nw's turns of those among the 32 slots s = I - 1 + lane (I the first bin) that
// keep their exact pair sums (spread over the warps), added to R, TH. Returns the mask of
// those slots; the prefix part of the others is left to the caller.
template <int K, int NP, int U = 1>
__device__ __forceinline__ unsigned slot_exact_turns(const SlotGrid& g, const SlotPass* p, int I, int w, int nw,
                                                     double& R, double& TH)
{
    const int l = threadIdx.x & 31, s = I - 1 + l, n = g.n;
    const bool slot = s >= 0 && s <= n - 2;
    // (mom_exact_slot; not where x_{s+1} is within kMomGuard 2^53 = 2252 of x_0: bin s + 1
    // gets at least x_0 / dx_s of every one of these pairs' rates, and u is within
    // kMomGuard of that. 4096 cells of 48 sections: 503 us, 465 with this)
    bool ex = false;
    const double xu = slot ? __ldg(g.x + s + 1) : 0.0;
    if (slot && slot_cut(g, s) > 0 && xu > (kMomGuard * 9007199254740992.0) * __ldg(g.x)) {
        const double idx = g.inv_dx[s];
#pragma unroll
        for (int q = 0; q < NP; ++q) ex = ex || mom_exact_slot(p[q].Nk[s], p[q].Nk[s + 1], xu, idx);
    }
    const unsigned exact = __ballot_sync(0xffffffffu, ex);
    int turn = 0;
    for (unsigned m = exact; m != 0u; m &= m - 1u) {
        const int le = __ffs(m) - 1;
        if (turn == w) {
            double r, t;
            slot_exact<K, NP, U>(g, p, I - 1 + le, r, t);
            if (l == le) { R += r; TH += t; }
        }
        turn = turn + 1 == nw ? 0 : turn + 1;
    }
    return exact;
}

// Warp w of nw's direct lags of the 32 slots s = I - 1 + lane on a geometric grid:
// equal contiguous shares of the lags below D0 (each warp sees its runs in order).
template <int K, int NP>
__device__ __forceinline__ void slot_lags(const SlotGrid& g, const SlotPass* p, int I, int w, int nw,
                                          double& R, double& TH)
{
    const int s = I - 1 + (threadIdx.x & 31), n = g.n;
    const bool slot = s >= 0 && s <= n - 2;
    const int smax = min(I - 1 + 31, n - 2);
    const double xs = slot ? __ldg(g.x + s) : 1.0;
    const int lags = min(min(n, g.D0), smax + 1);
    const int per = (lags + nw - 1) / nw;
    const int d0 = w * per;
    slot_pairs_geo<K, NP>(g, p, s, slot, smax, d0, min(lags, d0 + per), ew_operand_c(xs, -exponent_of(xs)), R, TH);
}

// Clipped pairs (x_j + x_k >= x[n-1], all deposited on bin n-1,
// src/aggregation_kernels.cuh:191-192) but for those of the prefix sums of slot
// n - 1, share of thread tid of nt: a warp per lag with its lanes over j on a
// geometric grid, lanes over a row's larger members otherwise. Neighbouring warps have shares of about
// equal length and far ones have not, so CTAs that share a cell take warps in turn
// (slot_clip_tid).
__device__ __forceinline__ int slot_clip_tid(int rank, int ranks)
{
    return ((static_cast<int>(threadIdx.x >> 5) * ranks + rank) << 5) + static_cast<int>(threadIdx.x & 31);
}

// A row's larger members over as many lanes as a cell's CTAs have threads for: a pair is a
// chain of some ten dependent FP64 instructions, and n / 2 of them in a row took 31 us at
// 155 linear sections.
__device__ __forceinline__ int slot_clip_lanes(int n, int nt)
{
    int G = 1;
    while (G < 32 && 2 * G * n <= nt) G <<= 1;
    return G;
}

// G: lanes a row (a power of two).
template <int K, int NP>
__device__ double slot_clip(const SlotGrid& g, const SlotPass* p, int tid, int nt, int G)
{
    const int n = g.n;
    double acc = 0.0;
    if (g.geo) {
        const int l = tid & 31;
        for (int d = tid >> 5; d < min(n, g.D0); d += nt >> 5) {
            const int L = g.Ld[d];
            const int jlo = L >= kLagClipAll ? 0 : max(0, n - 1 - L);
            const double B = g.Bd[d], S = g.Sd[d];
            for (int j = jlo + l; j <= n - 1 - d; j += 32)
#pragma unroll
                for (int q = 0; q < NP; ++q)
                    acc += rate_geo<K>(B, S, p[q].Nj[j], NeedH<K>::j ? p[q].Hj[j] : 0.0,
                                       p[q].Nk[j + d],
                                       NeedH<K>::k ? p[q].Hk[j + d] : 0.0);
        }
    } else {
        const long long top = dbits(__ldg(g.x + n - 1));
        for (int j = tid / G; j < n; j += nt / G) {
            const double xj = __ldg(g.x + j);
            int lo = j, hi = n - 1;                    // x_j + x[n-1] >= x[n-1] always holds
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (dbits(xj + __ldg(g.x + mid)) >= top) hi = mid; else lo = mid + 1;
            }
            // k = n - 1 is in the prefix sums, but for the diagonal pair
            const int sub = tid & (G - 1);
            const RowBeta<K> row(g, j);
#pragma unroll 2
            for (int k = lo + sub; k < n - 1; k += G) acc += slot_rate_any<K, NP>(g, p, row, j, k);
            if (j == n - 1 && sub == 0) acc += slot_rate_any<K, NP>(g, p, row, j, j);
        }
    }
    return acc;
}

} // namespace pbe_gb300
