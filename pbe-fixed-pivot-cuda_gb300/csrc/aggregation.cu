// =============================================================================
// aggregation.cu -- fixed-pivot aggregation RHS for GB300 (sm_103a), FP64.
//
// Reference semantics (acuoci/pbe-fixed-pivot-cuda src/aggregation_kernels.cuh:145-239):
// for every pair j <= k, rate = beta_jk N_j N_k (x1/2 if j == k); death -rate
// at j and at k (-2 rate on the diagonal); birth of v = x_j + x_k split onto
// the bracketing pivots lo, lo+1 with w = (v - x_lo)/(x_{lo+1} - x_lo); v >=
// x[n-1] goes wholly to bin n-1 (:191-192).
//
// Formulation used here (same sums, reorganised for an FP64-starved GPU):
//  * Death is separable: sum_k beta_ik N_k is a combination of five moments
//    M_p = sum_k x_k^p N_k (p = -1/3, 0, 1/3, 2/3, 1) for every kernel type,
//    so the death term costs O(n) instead of O(n^2).
//  * Birth is a gather over "slots": slot s collects the pairs whose bracket
//    is lo = s. Per slot two sums are kept, R_s = sum rate and
//    TH_s = sum rate * (v - x_s). Then bin i receives
//    (R_i - TH_i / dx_i) + TH_{i-1} / dx_{i-1}, which is the reference's
//    (1 - w) rate + w rate regrouped.
//  * Pairs that land on their larger member's own slot are separable too, from
//    prefix moments of N and x N (agg_lane.cuh): O(n).
//  * Geometric grids (verified on the device, see agg_prep_kernel): the
//    bracket offset lo - j, the Brownian factor and the shear factor depend on
//    the lag d = k - j only. They come from per-lag tables, so a pair costs
//    1-3 FP64 operations plus two accumulations. The weight numerator
//    fl(x_j + x_k) - x_lo is formed from the actual pivots exactly as the
//    reference forms it, but on the integer pipe (exact_weight.cuh).
//  * Other grids: brackets by a monotone walk over k, beta from per-bin cube
//    roots (agg_slot.cuh).
//  * Pairs clipped at x[n-1] are summed by up to 32 tasks; in gather mode the
//    last of them and of the task owning bin n-1 adds their parts, in order, to
//    rhs[n-1].
//
// Kernels per call: up to kSmallMaxN sections, one cluster kernel in gather mode
// (agg_small_kernel); else prep (per-bin values, lag tables, prefix moments, geometric
// check; its last block finishes moments, flag and counters) -> pair kernel
// (persistent CTAs pulling tasks from an atomic counter, agg_lane.cuh). GATHER
// mode: each output bin is written once, from sums reduced in a fixed order ->
// bitwise reproducible. SCATTER mode: every task flushes its bins with FP64
// atomicAdd.
// =============================================================================
#include <cooperative_groups.h>

#include "agg_lane.cuh"
#include "device_answer.h"
#include "tape_stage.cuh"

namespace pbe_gb300 {
namespace {

// Prefix sums of one prep block (see AggWs::mloc), two warps in lane order, and
// the block totals. The weighted sums run at the exponent of each bin's pivot,
// so they keep the range of x_j / x_i on grids of any span; a shift between
// exponents takes integer instructions only. Fixed order: reproducible.
template <int K>
__device__ __forceinline__ void prep_prefix(const double* m, double xm, int E, int i, int n, int nb,
                                            const AggWs& ws, double* gsum)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    static_assert(kPrepThreads == 64, "two warps of bins");
    double P[kMomN], T[kMomN];
#pragma unroll
    for (int q = 0; q < kMomN; ++q) { P[q] = m[q]; T[q] = m[q] * xm; }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int dE = __shfl_up_sync(0xffffffffu, E, o) - E;
#pragma unroll
        for (int q = 0; q < kMomN; ++q) {
            if (!need_moment<K>(q)) continue;
            const double p = __shfl_up_sync(0xffffffffu, P[q], o);
            const double t = __shfl_up_sync(0xffffffffu, T[q], o);
            if (lane >= o) { P[q] += p; T[q] += scale_down(t, dE); }
        }
    }
    // the first warp's sums enter the second's at its bins' exponents
    __shared__ int e_s;
    if (w == 0 && lane == 31) {
        e_s = E;
#pragma unroll
        for (int q = 0; q < kMomN; ++q) { gsum[q] = P[q]; gsum[kMomN + q] = T[q]; }
    }
    asm volatile("bar.sync 1, %0;" :: "n"(kPrepThreads) : "memory");
    const int b = blockIdx.x;
    const int last = min(n - 1, b * kPrepThreads + kPrepThreads - 1);
#pragma unroll
    for (int q = 0; q < kMomN; ++q) {
        if (!need_moment<K>(q)) continue;
        if (w == 1 && i < n) {
            P[q] += gsum[q];
            T[q] += scale_down(gsum[kMomN + q], e_s - E);
        }
        if (i < n) {
            ws.mloc[static_cast<size_t>(q) * n + i] = P[q];
            ws.mloc[static_cast<size_t>(kMomN + q) * n + i] = T[q];
        }
        if (i == last) {
            ws.mtot[q * nb + b] = P[q];
            ws.mtot[(kMomN + q) * nb + b] = T[q];
        }
    }
}

// Window tables of one prep block (AggWs::wtab) and, FULL, the coefficients of its bins
// as larger members (AggWs::wc). p and s run through the prefix and suffix sums within
// aligned groups of 1, 2, 4 .. bins: joining two groups, the right half's prefixes
// gain the left half's total and the left half's suffixes the right half's, one
// add a lane, step and moment (p of the left half's last lane and s of the right
// half's first are those totals).
template <int K, bool FULL>
__device__ __forceinline__ void prep_windows(const double* __restrict__ x, double xi, double Ni, double ai,
                                             double iai, int i, int n, const AggWs& ws, double (*wtot)[kWinMom],
                                             double b0, double bbr, double bsh)
{
    const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) & 1;   // two whole warps
    const size_t ns = static_cast<size_t>(n);
    const int E = win_exponent(x), E20 = E * (1 << 20);
    xi = scale_pow2(xi, -E20);
    ai = scale_pow2(ai, -E20 / 3);
    iai = scale_pow2(iai, E20 / 3);
    const double m[kMomN] = {iai * Ni, Ni, ai * Ni, (ai * ai) * Ni, xi * Ni};
    double p[kWinMom], s[kWinMom];
#pragma unroll
    for (int q = 0; q < kWinMom; ++q) {
        if (!need_window<K>(q)) continue;
        double v = q < kMomN ? m[q < kMomN ? q : 0] : xi * m[q >= 3 ? q - 3 : 0];
        p[q] = s[q] = v;
#pragma unroll
        for (int h = 1; h < 32; h <<= 1) {
            const bool right = (lane & h) != 0;
            const int src = (lane & ~(2 * h - 1)) + (right ? h - 1 : h);
            const double t = __shfl_sync(0xffffffffu, right ? s[q] : p[q], src);
            if (h >= 4 && i < n) {
                const int l = h == 4 ? 0 : h == 8 ? 1 : 2;
                ws.wtab[(l * kWinMom + q) * ns + i] = right ? p[q] : s[q];
            }
            if (right) p[q] += t; else s[q] += t;
        }
        if (i < n) ws.wtab[(3 * kWinMom + q) * ns + i] = w ? p[q] : s[q];
        if (lane == 31) wtot[w][q] = p[q];
    }
    asm volatile("bar.sync 3, %0;" :: "n"(kPrepThreads) : "memory");
    if (i >= n) return;
#pragma unroll
    for (int q = 0; q < kWinMom; ++q) {
        if (!need_window<K>(q)) continue;
        ws.wtab[(4 * kWinMom + q) * ns + i] = w ? p[q] + wtot[0][q] : p[q];
        ws.wtab[(5 * kWinMom + q) * ns + i] = w ? s[q] : s[q] + wtot[1][q];
    }
    if constexpr (!FULL) return;
    // beta(x_j, x_k) = sum_q c_q(x_k) m_q(x_j), m_q = {1/a, 1, a, a^2, x}, all in the tables'
    // unit: Sum and Shear are of the first degree in x, Product of the second
    double c[kMomN] = {0.0, 0.0, 0.0, 0.0, 0.0};
    if constexpr (K == 0) c[1] = b0;
    if constexpr (K == 1) { b0 = scalbn(b0, E); c[1] = b0 * xi; c[4] = b0; }
    if constexpr (K == 2) c[4] = scalbn(b0, 2 * E) * xi;
    if constexpr (K == 3 || K == 5) { c[0] = bbr * ai; c[1] = 2.0 * bbr; c[2] = bbr * iai; }
    if constexpr (K == 4 || K == 5) {
        bsh = scalbn(bsh, E);
        c[1] = fma(bsh, xi, c[1]);
        c[2] = fma(3.0 * bsh, ai * ai, c[2]);
        c[3] = (3.0 * bsh) * ai;
        c[4] = bsh;
    }
#pragma unroll
    for (int q = 0; q < kMomN; ++q)
        if (need_moment<K>(q)) ws.wc[q * ns + i] = c[q];
}

// Scan of the block totals by the prep's last block: each lane sums a run of
// consecutive blocks, a warp scan adds the runs, each lane writes its blocks'
// offsets. Warp 0: the moments (their last sums are the death term's moments),
// warp 1: the weighted ones.
template <int K>
__device__ __forceinline__ void prep_offsets(const double* __restrict__ x, int n, int nb,
                                             const AggWs& ws, int w, int lane)
{
    const int per = (nb + 31) / 32;
    const int b0 = min(nb, lane * per), b1 = min(nb, b0 + per);
    auto last_exp = [&](int b) { return exponent_of(__ldg(x + min(n - 1, (b + 1) * kPrepThreads - 1))); };
    // exponent the running sum stands at: that of the last bin before / in the run
    const int Eb = b0 > 0 ? last_exp(b0 - 1) : 0;
    int Ee = b1 > 0 ? last_exp(b1 - 1) : 0;
    const double* tot = ws.mtot + static_cast<size_t>(w) * kMomN * nb;
    double* off = ws.moff + static_cast<size_t>(w) * kMomN * nb;
    double S[kMomN];
#pragma unroll
    for (int q = 0; q < kMomN; ++q) S[q] = 0.0;
    int e = Eb;
    // kRun blocks' totals and exponents at a time, loaded together: a load at a time
    // took 0.7 us a block and pass (256 blocks: the whole call 326 us, 323 so)
    constexpr int kRun = 4;
    double t[kRun][kMomN];
    int en[kRun];
    auto load = [&](int b) {
#pragma unroll
        for (int u = 0; u < kRun; ++u) {
            const int c = min(b + u, nb - 1);
            en[u] = w ? last_exp(c) : 0;
#pragma unroll
            for (int q = 0; q < kMomN; ++q) t[u][q] = need_moment<K>(q) ? __ldcg(tot + q * nb + c) : 0.0;
        }
    };
    for (int b = b0; b < b1; b += kRun) {
        load(b);
#pragma unroll
        for (int u = 0; u < kRun; ++u) {
            if (b + u >= b1) break;
#pragma unroll
            for (int q = 0; q < kMomN; ++q)
                if (need_moment<K>(q)) S[q] = (w ? scale_down(S[q], e - en[u]) : S[q]) + t[u][q];
            e = en[u];
        }
    }
    double R[kMomN];
#pragma unroll
    for (int q = 0; q < kMomN; ++q) R[q] = S[q];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int dE = w ? __shfl_up_sync(0xffffffffu, Ee, o) - Ee : 0;
#pragma unroll
        for (int q = 0; q < kMomN; ++q) {
            if (!need_moment<K>(q)) continue;
            const double r = __shfl_up_sync(0xffffffffu, R[q], o);
            if (lane >= o) R[q] += w ? scale_down(r, dE) : r;
        }
    }
    e = Eb;
#pragma unroll
    for (int q = 0; q < kMomN; ++q) {
        if (!need_moment<K>(q)) continue;
        if (w == 0 && lane == 31) ws.mom[q] = R[q];
        const double r = __shfl_up_sync(0xffffffffu, R[q], 1);
        S[q] = lane > 0 ? r : 0.0;
    }
    for (int b = b0; b < b1; b += kRun) {
        load(b);
#pragma unroll
        for (int u = 0; u < kRun; ++u) {
            if (b + u >= b1) break;
#pragma unroll
            for (int q = 0; q < kMomN; ++q) {
                if (!need_moment<K>(q)) continue;
                off[q * nb + b + u] = S[q];
                S[q] = (w ? scale_down(S[q], e - en[u]) : S[q]) + t[u][q];
            }
            e = en[u];
        }
    }
}

// ---------------------------------------------------------------------------
// prep: blocks of 64 bins. Threads 0..63 (a thread per bin): cube roots, the
// moments' terms and their prefix sums. The last 64 threads (the same bins): the
// window tables of fine grids. Threads 64..127 (FULL): the grid's part --
//   Bd[d], Sd[d] for d = i: beta(x_j, x_{j+d}) = Bd + x_j Sd on a geometric grid,
//   times c_d (1/2 for d = 0), with rho = x_d^(1/3) / x_0^(1/3):
//     Constant/Sum/Product: Bd = c_d beta0 (the x dependence stays per pair)
//     Brownian: Bd = c_d beta_br (rho + 1/rho + 2)
//     Shear:    Sd = c_d beta_sh (1 + rho)^3
//   Ld[d]: bracket of x_0 + x_d (kLagClipAll when it reaches x[n-1]); 1/dx; J0;
//   the geometric-grid deviation.
// The kernel is a chain of dependent FP64 instructions (cube root, divisions,
// log2: some 40 clocks each): the parts of a block run theirs side by side.
//
// FULL = false (stage calls of a caller that keeps the workspace, e.g. the RK4
// tape): every grid-only entry -- a, ia, inv_dx, Bd, Sd, Ld, J0, wc, the window runs, the
// geometric flag mom[5..6] and D0 in counter[1] -- is left as an earlier FULL
// call on the same pivots and coefficients wrote it; only the N-dependent
// values (h, moments, window tables) and the tickets are rewritten, with the
// same arithmetic as a FULL call, so the results are bitwise the same.
// Either way the last block resets counter[2] (the prep's block tickets) and
// the pair kernel's last CTA counter[5] (the exact slots' list), so a
// following call on the same workspace needs no memset.
// ---------------------------------------------------------------------------
constexpr int kPrepFullThreads = 3 * kPrepThreads;
constexpr int kPrepStageThreads = 2 * kPrepThreads;

// First j <= i with fl(x_j + x_i) >= x_{i+1} (i when there is none below), from a
// guess on the geometric grid through the end points, then galloping.
__device__ __forceinline__ int first_above(const double* __restrict__ x, int i, double xi, double xu,
                                           float lx0, float inv_span)
{
    const long long top = dbits(xu);
    const float gf = fminf(fmaxf((log2_approx(xu - xi) - lx0) * inv_span, 0.0f), static_cast<float>(i));
    int g = static_cast<int>(gf), lo = -1, hi = i, step = 1;   // below lo + 1: not yet; from hi on: above
    if (dbits(__ldg(x + g) + xi) >= top) {
        hi = g;
        while (hi - step > 0 && dbits(__ldg(x + hi - step) + xi) >= top) { hi -= step; step <<= 1; }
        lo = hi - step > 0 ? hi - step : -1;
    } else {
        lo = g;
        while (lo + step < i && dbits(__ldg(x + lo + step) + xi) < top) { lo += step; step <<= 1; }
        hi = min(i, lo + step);
    }
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (dbits(__ldg(x + mid) + xi) >= top) hi = mid; else lo = mid;
    }
    return hi;
}

// What a stage call adds to its prep: rhs is zeroed, and the CTAs from nb on do the
// breakage's prep of the stage (brk_stage_block).
struct PrepStage {
    double* rhs;
    BrkArgs brk;
    BrkWs bws;
};

template <int K, bool FULL>
__global__ void __launch_bounds__(FULL ? kPrepFullThreads : kPrepStageThreads)
agg_prep_kernel(const double* __restrict__ N, const double* __restrict__ x, int n, AggWs ws,
                double b0, double bbr, double bsh, int nb, PrepStage st)
{
    const int dep = dep_wait();
    N += dep; x += dep; n += dep;
    __shared__ double dev_s[kPrepThreads / 32];
    __shared__ double gsum[2 * kMomN];
    __shared__ double wtot[kPrepThreads / 32][kWinMom];
    __shared__ int neg_s[kPrepThreads / 32];
    __shared__ double a_s[kPrepThreads], ia_s[kPrepThreads];
    __shared__ double ax0_s;
    __shared__ GeoFit fit_s;
    __shared__ int d0_s[kPrepThreads / 32];
    __shared__ int last_s;
    if constexpr (!FULL) {
        if (static_cast<int>(blockIdx.x) >= nb) {
            brk_stage_block(N, x, st.brk.t_q, st.brk.bw_q, n, st.brk.n_quad, st.bws,
                            static_cast<int>(blockIdx.x) - nb, gsum);
            return;
        }
    }
    const int tid = threadIdx.x, wp = tid >> 5, lane = tid & 31;
    const int i = blockIdx.x * kPrepThreads + (tid & (kPrepThreads - 1));
    const double xi = x[min(i, n - 1)];
    if (tid < kPrepThreads) {
        double m[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        double xm = 0.0;     // mantissa and binary exponent of x_i
        int E = 0;
        double ai = 0.0, iai = 0.0, Ni = 0.0;
        if (i < n) {
            Ni = N[i];
            const double hi = xi * Ni;
            if constexpr (FULL) {
                ai = cbrt(xi);
                iai = 1.0 / ai;
                ws.a[i] = ai;
                ws.ia[i] = iai;
            } else {
                ai = ws.a[i];
                iai = ws.ia[i];
            }
            ws.h[i] = hi;
            if (!FULL) st.rhs[i] = 0.0;
            m[0] = iai * Ni; m[1] = Ni; m[2] = ai * Ni; m[3] = (ai * ai) * Ni; m[4] = hi;
            xm = mantissa_of(xi);
            E = exponent_of(xi);
            if (i < slot_blocks(n)) ws.cticket[i] = 0;
            // slots that keep the exact pair sum of their prefix part (the list's
            // order does not matter: each has its own task and its own sums)
            if (i < n - 1) {
                const double xu = x[i + 1];
                const double idx = FULL ? 1.0 / (xu - xi) : ws.inv_dx[i];
                if (FULL) ws.inv_dx[i] = idx;
                if (mom_exact_slot(Ni, N[i + 1], xu, idx)) ws.xlist[atomicAdd(ws.counter + 5, 1)] = i;
            } else if (FULL) {
                ws.inv_dx[i] = 0.0;
            }
        }
        if constexpr (FULL) {
            a_s[tid] = ai;
            ia_s[tid] = iai;
            __syncwarp();
            asm volatile("bar.arrive 2, %0;" :: "n"(kPrepFullThreads) : "memory");
        }
        const unsigned neg = __ballot_sync(0xffffffffu, !(Ni >= 0.0));   // negative, or NaN
        if (lane == 0) neg_s[wp] = neg != 0u;
        prep_prefix<K>(m, xm, E, i, n, nb, ws, gsum);
    } else if (wp >= (FULL ? 4 : 2)) {
        // window tables; FULL: the cube roots of the first two warps
        if constexpr (FULL) asm volatile("bar.sync 2, %0;" :: "n"(kPrepFullThreads) : "memory");
        if (win_grid(x, n)) {
            double Ni = 0.0, ai = 0.0, iai = 0.0;
            if (i < n) {
                Ni = N[i];
                ai = FULL ? a_s[tid & (kPrepThreads - 1)] : ws.a[i];
                iai = FULL ? ia_s[tid & (kPrepThreads - 1)] : ws.ia[i];
            }
            prep_windows<K, FULL>(x, xi, Ni, ai, iai, i, n, ws, wtot, b0, bbr, bsh);
        }
    } else if constexpr (FULL) {
        // the fit's end points on lanes 0 and 1 of the third warp, the cube root of
        // x_0 on the fourth, beside the bins' own logarithms
        const int Ei = ilogb(xi);
        const double fi = log2(scalbn(xi, -Ei));
        if (wp == 2) {
            const double xe = x[lane == 1 ? n - 1 : 0];
            const int Ee = ilogb(xe);
            const double fe = log2(scalbn(xe, -Ee));
            const double f1 = __shfl_sync(0xffffffffu, fe, 1);
            const int E1 = __shfl_sync(0xffffffffu, Ee, 1);
            if (lane == 0) fit_s = geo_fit_from(Ee, fe, E1, f1, n);
        } else {
            const double c0 = cbrt(x[0]);
            if (lane == 0) ax0_s = c0;
        }
        const float lx0 = log2_approx(__ldg(x));
        const float span = log2_approx(__ldg(x + n - 1)) - lx0;
        const float inv_span = (n > 1 && span > 0.0f) ? static_cast<float>(n - 1) / span : 0.0f;
        int d0 = n;      // this thread's lag if its pairs land on their larger member (Ld == d)
        if (i < n) {
            const double v = x[0] + xi;     // x[i] <= v: its bracket is at or above i
            const int L = (dbits(v) >= dbits(x[n - 1])) ? kLagClipAll : bracket_from(x, n, v, i);
            ws.Ld[i] = L;
            if (L == i && i > 0) d0 = i;    // lag 0 carries the pair 1/2: never separated
            // runs of lags with one bracket offset e = L - i: where this one ends,
            // the last run, and the first run that windows sum (win_grid)
            const int e = L - i;
            if (L < kLagClipAll) {
                const double vn = i + 1 < n ? x[0] + x[i + 1] : 0.0;
                const bool over = i + 1 >= n || dbits(vn) >= dbits(x[n - 1]);
                if (over || dbits(vn) < dbits(x[L + 1])) ws.rend[e] = i + 1;
                if (over) ws.counter[9] = e;
            }
            const double start = kWinStart * x[0];
            if (xi >= start && (i == 0 || x[i - 1] < start)) ws.counter[8] = L < kLagClipAll ? e - 1 : 0;
            if (i == n - 1 && xi < start) ws.counter[8] = 0;
            ws.J0[i] = i < n - 1 ? first_above(x, i, xi, x[i + 1], lx0, inv_span) : i;
        }
        __syncwarp();
        asm volatile("bar.sync 2, %0;" :: "n"(kPrepFullThreads) : "memory");   // a_s, fit_s, ax0_s
        double dev = 0.0;
        if (i < n) {
            const double c = (i == 0) ? 0.5 : 1.0;
            double B = 0.0, S = 0.0;
            if constexpr (K <= 2) B = c * b0;
            if constexpr (K >= 3) {
                const double rho = a_s[tid - kPrepThreads] / ax0_s;
                if constexpr (K == 3 || K == 5) B = c * bbr * (rho + 1.0 / rho + 2.0);
                if constexpr (K == 4 || K == 5) { const double t = 1.0 + rho; S = c * bsh * (t * t) * t; }
            }
            ws.Bd[i] = B;
            ws.Sd[i] = S;
            if (n >= 2) {
                dev = geo_dev_from(fit_s, Ei, fi, i);
                if (!(dev == dev)) dev = 1.0;   // NaN -> not geometric
            }
        }
        dev = warp_max(dev);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) d0 = min(d0, __shfl_xor_sync(0xffffffffu, d0, o));
        if (lane == 0) { dev_s[wp - 2] = dev; d0_s[wp - 2] = d0; }
    }
    __syncthreads();                           // the block's totals are written
    if (tid == 0) {
        if (FULL) {
            ws.mom_part[blockIdx.x * 8 + 5] = fmax(dev_s[0], dev_s[1]);
            ws.mom_part[blockIdx.x * 8 + 6] = static_cast<double>(min(d0_s[0], d0_s[1]));
        }
        ws.mom_part[blockIdx.x * 8 + 7] = (neg_s[0] | neg_s[1]) ? 1.0 : 0.0;
        __threadfence();                       // partials visible before the ticket
        last_s = (atomicAdd(ws.counter + 2, 1) == nb - 1);
    }
    __syncthreads();
    if (!last_s) return;
    // The last block to finish reduces every block's partials (read through L2)
    // in a fixed order. No block waits for another. Warps 0 and 1: the scan of the
    // block totals (prefix offsets, and the moments as its last sums); FULL, warp
    // 2: the largest deviation, warp 3: the smallest D0 candidate.
    __threadfence();
    if (wp < 2) {
        prep_offsets<K>(x, n, nb, ws, wp, lane);
        if (wp == 1) {
            double neg = 0.0;
            for (int b = lane; b < nb; b += 32) neg = fmax(neg, __ldcg(ws.mom_part + b * 8 + 7));
            neg = warp_max(neg);
            if (lane == 0) ws.mom[7] = neg;    // some N_i is negative or NaN
        }
    } else if (FULL && wp == 2) {
        double m5 = 0.0;
        for (int b = lane; b < nb; b += 32) m5 = fmax(m5, __ldcg(ws.mom_part + b * 8 + 5));
        m5 = warp_max(m5);
        if (lane == 0) {
            // neighbour ratio <= 64 keeps fl(x_j + x_k) within kMaxExpGap binades of
            // its bracket pivot (precondition of sum_minus_scaled)
            const bool geo = n >= 2 && m5 <= kGeoTol && x[1] <= 64.0 * x[0];
            ws.mom[5] = geo ? 1.0 : 0.0;
            ws.mom[6] = m5;
            const int entry = window_first_entry(__ldcg(ws.counter + 8), __ldcg(ws.counter + 9), n);
            ws.counter[10] = entry >= 0 ? __ldcg(ws.rend + entry) : 0;
        }
    } else if (FULL && wp == 3) {
        int dmin = n;
        for (int b = lane; b < nb; b += 32)
            dmin = min(dmin, static_cast<int>(__ldcg(ws.mom_part + b * 8 + 6)));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dmin = min(dmin, __shfl_xor_sync(0xffffffffu, dmin, o));
        if (lane == 0) ws.counter[1] = dmin;   // lags d >= counter[1] >= 1 have lo(j, j+d) = j + d
    }
    if (tid == 0) {
        ws.counter[0] = 0;          // task counter of the pair kernel
        ws.counter[2] = 0;          // this kernel's block tickets, ready for the next call
        ws.counter[3] = 0;          // contributors to bin n-1 done (clip tasks + top block)
        ws.counter[6] = 0;          // CTAs of the pair kernel done
    }
}

// Gather mode: the clip tasks and the task that owns bin n-1 each take a
// ticket after their contribution is stored; the last of the nclip + 1 adds
// the clip parts, in order, to rhs[n-1]. Called by one thread.
// (Bin n-1 is never a block's first bin: blocks are aligned to the top.)
__device__ __forceinline__ void clip_contributor_done(double* rhs, int n, const AggWs& ws,
                                                      int nclip)
{
    __threadfence();
    if (atomicAdd(ws.counter + 3, 1) != nclip) return;
    __threadfence();
    double s = 0.0;
    for (int c = 0; c < nclip; ++c) s += __ldcg(ws.clip_part + c);
    rhs[n - 1] = __ldcg(rhs + (n - 1)) + s;
}

// ---------------------------------------------------------------------------
// Pair kernel: persistent CTAs pulling tasks (agg_lane.cuh) -- clip tasks first,
// then the exact slots, then the tasks (block t, share p) of every block's direct
// pairs, share by share with the top blocks first (all shares of a geometric grid
// have equal lags but those of the lowest blocks, which come last).
// ---------------------------------------------------------------------------
#ifndef PBE_LANE_CTAS
#define PBE_LANE_CTAS 4
#endif
constexpr int kLaneCtas = PBE_LANE_CTAS;   // CTAs per SM (64 registers; 3: an irregular grid 115 us, not 97, others the same)

template <int K, bool SCATTER>
__global__ void __launch_bounds__(kMainThreads, kLaneCtas)
agg_lane_kernel(const double* __restrict__ N, const double* __restrict__ x,
                double* __restrict__ rhs, AggWs ws, int n, int nclip, double b0, double bbr,
                double bsh, int flip)
{
    const int dep = dep_wait();
    N += dep; x += dep; rhs += dep; n += dep;
    __shared__ LaneSmem sm;

    const int tid = threadIdx.x;
    LaneView v;
    v.g = SlotGrid{x, ws.a, ws.ia, ws.inv_dx, ws.Bd, ws.Sd, ws.Ld, ws.J0,
                   n, ws.counter[1], ws.mom[5] != 0.0, b0, bbr, bsh};
    v.p = SlotPass{N, ws.h, N, ws.h, N, ws.h};
#pragma unroll
    for (int q = 0; q < kMomN; ++q) v.M[q] = ws.mom[q];

    const int nblk = slot_blocks(n);
    // direct pairs of a slot: its lags below D0; on other grids at most its rows
    int Dm = min(v.g.D0, n), eh = 0, el = 1;
    if (!SCATTER && v.g.geo && ws.mom[7] == 0.0 && flip != kRatesMixed && win_grid(x, n)) {
        eh = ws.counter[8];
        el = max(1, ws.counter[9]);
        if (eh >= el) Dm = ws.counter[10];
    }
    // (a window counts as 5 pairs)
    const int parts = lane_parts(v.g.geo ? Dm + 5 * max(0, eh - el + 1) : n, nblk, gridDim.x);
    const int nexact = ws.counter[5];
    const int ntasks = nclip + nexact + nblk * parts;
    const LaneArgs la{ws.lpart, ws.cticket, parts, Dm, eh, el, flip};
    for (int next = blockIdx.x;;) {                      // the first task by the CTA's own index
        int task = next;
        if (task >= ntasks) break;
        if (task < nclip) {
            // a part of the clipped pairs (but for the prefix part of slot n - 1),
            // summed over the CTA in a fixed order
            // (a thread a row: 2049 irregular sections 125 us, 132 with two)
            double sc = warp_sum(slot_clip<K, 1>(v.g, &v.p, task * kMainThreads + tid, nclip * kMainThreads, 1));
            if ((tid & 31) == 0) sm.sum[tid >> 5] = sc;
            __syncthreads();
            if (tid == 0) {
                sc = 0.0;
                for (int w = 0; w < kLaneWarps; ++w) sc += sm.sum[w];
                if constexpr (SCATTER) {
                    if (sc != 0.0) atomicAdd(rhs + (n - 1), sc);
                } else {
                    ws.clip_part[task] = sc;
                    clip_contributor_done(rhs, n, ws, nclip);
                }
            }
            __syncthreads();
        } else if ((task -= nclip) < nexact) {
            exact_slot_task<K, SCATTER>(v, ws, la, rhs, ws.xlist[task], nclip, sm);
        } else {
            task -= nexact;
            lane_task<K, SCATTER>(v, ws, la, rhs, task % nblk, task / nblk, nclip, sm);
        }
        if (tid == 0) sm.task = static_cast<int>(gridDim.x) + atomicAdd(ws.counter, 1);
        __syncthreads();
        next = sm.task;
        __syncthreads();
    }
    // the last CTA leaves the exact slots' list empty for the next prep
    if (tid == 0 && atomicAdd(ws.counter + 6, 1) == static_cast<int>(gridDim.x) - 1) ws.counter[5] = 0;
}

// ---------------------------------------------------------------------------
// Small instances (gather mode, n <= kSmallMaxN): the whole call as one cluster,
// CTA r owning the bins [31 r, 31 r + 31) (a warp's lanes: their slots and the
// one below, so nothing is handed over). At these sizes a call is a chain of
// latencies -- two launches, a memset, tickets with memory fences, the FP64
// chains of the prep -- not work: 24 us of it at n = 64 in the kernels above.
//  1. grid tables and moments of the CTA's bins as agg_prep_kernel (warp 0 the
//     moments and their scan, warp 1 logarithms, brackets and J0, warp 2 the
//     geometric fit and 1/dx, warp 3 the lag factors), totals in shared memory;
//  2. cluster barrier; every CTA adds the others' totals (distributed shared
//     memory): prefix offsets, moments, geometric flag, D0;
//  3. the slots' pairs over the CTA's eight warps, the bins by warp 0.
// KIND as the launcher's: kAggTables stops after 2 and keeps the tables,
// kAggStage takes them from the workspace.
// ---------------------------------------------------------------------------
enum { kAggFull = 0, kAggTables = 1, kAggStage = 2 };
constexpr int kSmallBins = 31;
constexpr int kSmallMaxCtas = 16;
constexpr int kSmallMaxN = kSmallBins * kSmallMaxCtas;
constexpr int kSmallClipRows = 32;     // most rows of clipped pairs that the last CTA sums alone

template <int K, int KIND>
__global__ void __launch_bounds__(kMainThreads)
agg_small_kernel(const double* __restrict__ N, const double* __restrict__ x, double* __restrict__ rhs,
                 AggWs ws, int n, double b0, double bbr, double bsh)
{
    const int dep = dep_wait();
    N += dep; x += dep; rhs += dep; n += dep;
    namespace cg = cooperative_groups;
    const cg::cluster_group cl = cg::this_cluster();
    __shared__ double tot[2 * kMomN];                  // this CTA's totals (read by the cluster)
    __shared__ int te_s, d0_s;                         // exponent of its last bin, its D0 candidate
    __shared__ double dev_s;
    __shared__ double off[kSmallMaxCtas][2 * kMomN];   // sums over the CTAs before r
    __shared__ int oe[kSmallMaxCtas];                  // exponent they stand at
    __shared__ double M_s[kMomN];
    __shared__ double a_s[32];
    __shared__ double ax0_s;
    __shared__ GeoFit fit_s;
    __shared__ int D0_all;
    __shared__ int geo_all;
    __shared__ double red[kLaneWarps][2][32];
    __shared__ double csum[kLaneWarps];
    __shared__ double cpart[kSmallMaxCtas];            // last CTA: the CTAs' parts of the clipped pairs
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int r = static_cast<int>(cl.block_rank()), ranks = static_cast<int>(cl.num_blocks());
    const int I = kSmallBins * r;
    const int i = I + lane;
    const bool on = lane < kSmallBins && i < n;
    const int last = min(I + kSmallBins - 1, n - 1);   // the CTA's last bin
    const double xi = x[on ? i : last];

    // 1. grid tables and moments
    int Ei = 0, d0 = n;
    double fi = 0.0;
    if (w == 0) {
        double ai, iai;
        if constexpr (KIND == kAggStage) {
            ai = ws.a[on ? i : last];
            iai = ws.ia[on ? i : last];
        } else {
            ai = cbrt(xi);
            iai = 1.0 / ai;
            if (on) { ws.a[i] = ai; ws.ia[i] = iai; }
            a_s[lane] = ai;
        }
        if constexpr (KIND != kAggTables) {
            const double Ni = on ? N[i] : 0.0;
            const double hi = xi * Ni, xm = mantissa_of(xi);
            const int E = exponent_of(xi);
            if (on) ws.h[i] = hi;
            double P[kMomN] = {iai * Ni, Ni, ai * Ni, (ai * ai) * Ni, hi}, T[kMomN];
#pragma unroll
            for (int q = 0; q < kMomN; ++q) T[q] = P[q] * xm;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int dE = __shfl_up_sync(0xffffffffu, E, o) - E;
#pragma unroll
                for (int q = 0; q < kMomN; ++q) {
                    if (!need_moment<K>(q)) continue;
                    const double p = __shfl_up_sync(0xffffffffu, P[q], o);
                    const double t = __shfl_up_sync(0xffffffffu, T[q], o);
                    if (lane >= o) { P[q] += p; T[q] += scale_down(t, dE); }
                }
            }
#pragma unroll
            for (int q = 0; q < kMomN; ++q) {
                if (!need_moment<K>(q)) continue;
                if (on) {
                    ws.mloc[q * n + i] = P[q];
                    ws.mloc[(kMomN + q) * n + i] = T[q];
                }
                if (lane == 31) { tot[q] = P[q]; tot[kMomN + q] = T[q]; }
            }
            if (lane == 31) te_s = E;
        }
    }
    if constexpr (KIND != kAggStage) {
        if (w == 1) {
            Ei = ilogb(xi);
            fi = log2(scalbn(xi, -Ei));
            const float lx0 = log2_approx(__ldg(x));
            const float span = log2_approx(__ldg(x + n - 1)) - lx0;
            const float inv_span = (n > 1 && span > 0.0f) ? static_cast<float>(n - 1) / span : 0.0f;
            if (on) {
                const double v = x[0] + xi;
                const int L = (dbits(v) >= dbits(x[n - 1])) ? kLagClipAll : bracket_from(x, n, v, i);
                ws.Ld[i] = L;
                if (L == i && i > 0) d0 = i;           // lag 0 carries the pair 1/2: never separated
                ws.J0[i] = i < n - 1 ? first_above(x, i, xi, x[i + 1], lx0, inv_span) : i;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) d0 = min(d0, __shfl_xor_sync(0xffffffffu, d0, o));
        } else if (w == 2) {
            const double xe = x[lane == 1 ? n - 1 : 0];
            const int Ee = ilogb(xe);
            const double fe = log2(scalbn(xe, -Ee));
            const double f1 = __shfl_sync(0xffffffffu, fe, 1);
            const int E1 = __shfl_sync(0xffffffffu, Ee, 1);
            if (lane == 0) fit_s = geo_fit_from(Ee, fe, E1, f1, n);
            if (on) ws.inv_dx[i] = (i < n - 1) ? 1.0 / (x[i + 1] - xi) : 0.0;
        } else if (w == 3) {
            const double c0 = cbrt(x[0]);
            if (lane == 0) ax0_s = c0;
        }
        __syncthreads();
        if (w == 1) {
            double dev = (on && n >= 2) ? geo_dev_from(fit_s, Ei, fi, i) : 0.0;
            if (!(dev == dev)) dev = 1.0;              // NaN -> not geometric
            dev = warp_max(dev);
            if (lane == 0) { dev_s = dev; d0_s = d0; }
        } else if (w == 3 && on) {
            const double c = (i == 0) ? 0.5 : 1.0;
            double B = 0.0, S = 0.0;
            if constexpr (K <= 2) B = c * b0;
            if constexpr (K >= 3) {
                const double rho = a_s[lane] / ax0_s;
                if constexpr (K == 3 || K == 5) B = c * bbr * (rho + 1.0 / rho + 2.0);
                if constexpr (K == 4 || K == 5) { const double t = 1.0 + rho; S = c * bsh * (t * t) * t; }
            }
            ws.Bd[i] = B;
            ws.Sd[i] = S;
        }
    }
    cl.sync();

    // 2. the other CTAs' totals
    if (w == 0 && lane < 2 * kMomN && KIND != kAggTables) {
        const bool weighted = lane >= kMomN;
        double acc = 0.0;
        int e = 0;
        for (int q = 0; q < ranks; ++q) {
            const int en = *cl.map_shared_rank(&te_s, q);
            off[q][lane] = acc;
            if (lane == 0) oe[q] = e;
            if (weighted && q > 0) acc = scale_down(acc, e - en);
            acc += *cl.map_shared_rank(&tot[lane], q);
            e = en;
        }
        if (!weighted) M_s[lane] = acc;
    }
    if (w == 1) {
        if constexpr (KIND == kAggStage) {
            if (lane == 0) { geo_all = ws.mom[5] != 0.0 ? 1 : 0; D0_all = ws.counter[1]; }
        } else {
            double dev = 0.0;
            int dm = n;
            if (lane < ranks) {
                dev = *cl.map_shared_rank(&dev_s, lane);
                dm = *cl.map_shared_rank(&d0_s, lane);
            }
            dev = warp_max(dev);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) dm = min(dm, __shfl_xor_sync(0xffffffffu, dm, o));
            if (lane == 0) {
                // neighbour ratio <= 64: precondition of sum_minus_scaled
                geo_all = (n >= 2 && dev <= kGeoTol && x[1] <= 64.0 * x[0]) ? 1 : 0;
                D0_all = dm;
                if (KIND == kAggTables && r == 0) {
                    ws.mom[5] = geo_all ? 1.0 : 0.0;
                    ws.counter[1] = dm;
                }
            }
        }
    }
    cl.sync();            // offsets in place; nobody reads another CTA's memory from here on
    if constexpr (KIND == kAggTables) return;

    // 3. pairs and bins
    const SlotGrid g{x, ws.a, ws.ia, ws.inv_dx, ws.Bd, ws.Sd, ws.Ld, ws.J0, n, D0_all, geo_all != 0,
                     b0, bbr, bsh};
    const SlotPass p{N, ws.h, N, ws.h, N, ws.h};
    const int s = I - 1 + lane;                        // this lane's slot and bin
    const bool slot = s >= 0 && s <= n - 2;
    double R = 0.0, TH = 0.0;
    if (g.geo) {
        slot_lags<K, 1>(g, &p, I, w, kLaneWarps, R, TH);
    } else {
        // the rows' end sought from where a geometric grid through the end points would have it
        int jt = 0;
        if (slot) {
            const float lx0 = log2_approx(__ldg(x)), span = log2_approx(__ldg(x + n - 1)) - lx0;
            const float gf = (log2_approx(__ldg(x + s + 1)) - 1.0f - lx0) * (static_cast<float>(n - 1) / span);
            jt = slot_rows_end(x, s, static_cast<int>(fminf(fmaxf(gf, 0.0f), static_cast<float>(s))));
        }
        slot_pairs_any<K, 1>(g, &p, s, slot, jt, w, kLaneWarps, R, TH);
    }
    const unsigned exact = slot_exact_turns<K, 1>(g, &p, I, w, kLaneWarps, R, TH);
    red[w][0][lane] = R;
    red[w][1][lane] = TH;
    // the clipped pairs: of few rows (D0 of a geometric grid, those from J0(n - 2) on of
    // another) by the last CTA, else (fine or linear grids: up to half of all pairs) a
    // share per CTA (all of them in the last one: 480 sections at 128 an octave 99 us, 248
    // linear ones 140)
    const bool alone = ranks == 1 || (g.geo ? g.D0 : n - ws.J0[n - 2]) <= kSmallClipRows;
    if (!alone || r == ranks - 1) {
        const int nt = (alone ? 1 : ranks) * kMainThreads;
        const double c = warp_sum(slot_clip<K, 1>(g, &p, alone ? tid : slot_clip_tid(r, ranks), nt,
                                                  slot_clip_lanes(n, nt)));
        if (lane == 0) csum[w] = c;
    }
    __syncthreads();
    if (!alone) {
        if (tid == 0) {
            double sum = 0.0;
            for (int q = 0; q < kLaneWarps; ++q) sum += csum[q];
            *cl.map_shared_rank(&cpart[r], static_cast<unsigned>(ranks - 1)) = sum;
        }
        cl.sync();                                     // the parts are there; nobody left before
    }
    if (w != 0) return;
    R = 0.0;
    TH = 0.0;
#pragma unroll
    for (int q = 0; q < kLaneWarps; ++q) { R += red[q][0][lane]; TH += red[q][1][lane]; }
    double death = 0.0, clip = 0.0, own = 0.0, up = 0.0;
    if (s >= 0 && s < n) {
        const double xs = x[s], as = g.a[s], ias = g.ia[s], Ns = N[s];
        const int St = -exponent_of(xs);
        death = Ns * death_factor<K>(xs, as, ias, M_s, b0, bbr, bsh);
        const int cut = slot_cut(g, s);
        if (cut > 0 && !((exact >> lane) & 1u)) {
            const int j = cut - 1, b = j / kSmallBins, Ej = exponent_of(x[j]);
            double P[kMomN], T[kMomN];
#pragma unroll
            for (int q = 0; q < kMomN; ++q) {
                P[q] = T[q] = 0.0;
                if (!need_moment<K>(q)) continue;
                P[q] = ws.mloc[q * n + j] + off[b][q];
                T[q] = ws.mloc[(kMomN + q) * n + j] + scale_down(off[b][kMomN + q], oe[b] - Ej);
            }
            const double rr = Ns * death_factor<K>(xs, as, ias, P, b0, bbr, bsh);
            if (slot) {
                R += rr;
                TH += Ns * scale_down(death_factor<K>(xs, as, ias, T, b0, bbr, bsh), Ej + St);
            } else {
                clip = rr;                             // bin n - 1: clipped
            }
        }
        if (slot) {
            const double sd = scalbn(g.inv_dx[s], -St);
            own = fma(-TH, sd, R);
            up = TH * sd;
        } else {
            if (alone) for (int q = 0; q < kLaneWarps; ++q) clip += csum[q];
            else for (int q = 0; q < ranks; ++q) clip += cpart[q];
        }
    }
    const double in = __shfl_up_sync(0xffffffffu, up, 1);
    if (lane >= 1 && s < n)
        rhs[s] = (KIND == kAggStage ? 0.0 : rhs[s]) + (((own + in) + clip) - death);   // a stage call writes rhs
}

// One cluster of the current device can hold 16 CTAs of this kernel (a size beyond the
// portable 8, asked for once per kernel and device).
template <int K, int KIND>
bool small_cluster_ok(int ranks)
{
    if (ranks <= 8) return true;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    static DeviceAnswer answer;
    return answer.get(dev, []() {
        auto kern = agg_small_kernel<K, KIND>;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(kSmallMaxCtas);
        cfg.blockDim = dim3(kMainThreads);
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = kSmallMaxCtas;
        at.val.clusterDim.y = 1;
        at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int num = 0;
        if (cudaOccupancyMaxActiveClusters(&num, kern, &cfg) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        return num > 0 ? 1 : -1;
    });
}

template <int K, int KIND>
cudaError_t launch_small(const AggArgs& a, const AggWs& ws, cudaStream_t s, int ranks)
{
    const bool prof = KIND != kAggTables && g_prof_start && g_prof_stop;
    if (prof) cudaEventRecord(g_prof_start, s);
    const cudaError_t e = launch_dep(agg_small_kernel<K, KIND>, dim3(static_cast<unsigned>(ranks)),
                                     kMainThreads, 0,
                                     s, static_cast<unsigned>(ranks), a.N, a.x, a.rhs, ws, a.n, a.beta0,
                                     a.beta_br, a.beta_sh);
    if (prof) cudaEventRecord(g_prof_stop, s);
    return launch_result(e);
}

// Tasks that sum the clipped pairs (about n + 1.2 q^2 pairs on a grid with q bins
// per octave, up to half of all pairs on others).
int agg_clip_tasks(int n)
{
    const int c = (n + 63) / 64;
    return c < 1 ? 1 : (c > kMaxClipTasks ? kMaxClipTasks : c);
}

// kind: kAggFull = tables + pair kernel (the drop-in calls), kAggTables =
// the FULL prep only, kAggStage = the light prep + pair kernel on a
// workspace whose tables an earlier kAggTables call wrote.
template <int K, bool SC>
cudaError_t launch_k(const AggArgs& a, const AggWs& ws, int num_sms, cudaStream_t s, int kind,
                     const PrepStage* st, bool* brk_done)
{
    const int n = a.n;
    if (!SC && n <= kSmallMaxN) {
        // (n = 64, aggregation + breakage: 43.8 us through the two kernels below, 31.1 through one)
        const int ranks = (n + kSmallBins - 1) / kSmallBins;
        if (small_cluster_ok<K, kAggFull>(ranks) && small_cluster_ok<K, kAggTables>(ranks) &&
            small_cluster_ok<K, kAggStage>(ranks)) {
            if (kind == kAggFull) return launch_small<K, kAggFull>(a, ws, s, ranks);
            if (kind == kAggTables) return launch_small<K, kAggTables>(a, ws, s, ranks);
            return launch_small<K, kAggStage>(a, ws, s, ranks);
        }
    }
    const int nb = agg_prep_blocks(n);
    const int nclip = agg_clip_tasks(n);
    auto kern = agg_lane_kernel<K, SC>;
    // the number of tasks is known on the device only (it follows D0)
    const long long cap = static_cast<long long>(kLaneCtas) * num_sms;
    const long long most = static_cast<long long>(slot_blocks(n)) * kLaneMaxParts + nclip;
    const int grid = static_cast<int>(most < cap ? most : cap);
    cudaError_t e = cudaSuccess;
    if (kind == kAggStage) {
        // counter[2] and [5] were left at 0 by the previous call on this workspace
        // (a stage's rhs is zeroed and its breakage prep done by further CTAs of the same launch)
        const int bb = st->brk.n_quad > 0 ? brk_prep_blocks(n, st->brk.n_quad) : 0;
        launch_dep(agg_prep_kernel<K, false>, dim3(nb + bb), kPrepStageThreads, 0, s, 1, a.N, a.x, n, ws, a.beta0,
                   a.beta_br, a.beta_sh, nb, *st);
        *brk_done = bb > 0;
    } else {
        // the prep's block tickets; and what pivots that are no numbers leave unwritten
        e = cudaMemsetAsync(ws.counter, 0, kAggCounters * sizeof(int), s);
        if (e != cudaSuccess) return e;
        launch_dep(agg_prep_kernel<K, true>, dim3(nb), kPrepFullThreads, 0, s, 1, a.N, a.x, n, ws, a.beta0,
                   a.beta_br, a.beta_sh, nb, PrepStage{});
        if (kind == kAggTables) {
            e = cudaGetLastError();
            // this call's exact slots are no one's: the next prep starts its own list
            return e != cudaSuccess ? e : cudaMemsetAsync(ws.counter + 5, 0, sizeof(int), s);
        }
    }
    const bool prof = g_prof_start && g_prof_stop;
    if (prof) cudaEventRecord(g_prof_start, s);
    launch_dep(kern, dim3(grid), kMainThreads, 0, s, 1, a.N, a.x, a.rhs, ws, n, nclip, a.beta0, a.beta_br,
               a.beta_sh, rates_flip(a.kernel, a.beta0, a.beta_br, a.beta_sh));
    if (prof) cudaEventRecord(g_prof_stop, s);
    return cudaGetLastError();
}

template <bool SC>
cudaError_t dispatch(const AggArgs& a, const AggWs& ws, int num_sms, cudaStream_t s, int kind,
                     const PrepStage* st = nullptr, bool* brk_done = nullptr)
{
    switch (a.kernel) {
    case 0: return launch_k<0, SC>(a, ws, num_sms, s, kind, st, brk_done);
    case 1: return launch_k<1, SC>(a, ws, num_sms, s, kind, st, brk_done);
    case 2: return launch_k<2, SC>(a, ws, num_sms, s, kind, st, brk_done);
    case 3: return launch_k<3, SC>(a, ws, num_sms, s, kind, st, brk_done);
    case 4: return launch_k<4, SC>(a, ws, num_sms, s, kind, st, brk_done);
    case 5: return launch_k<5, SC>(a, ws, num_sms, s, kind, st, brk_done);
    default: return cudaErrorInvalidValue;
    }
}

} // namespace

cudaEvent_t g_prof_start = nullptr;
cudaEvent_t g_prof_stop = nullptr;

cudaError_t agg_launch(const AggArgs& a, bool scatter, void* ws_base, int num_sms, cudaStream_t s)
{
    AggWs ws;
    agg_ws_layout(a.n, static_cast<char*>(ws_base), &ws);
    return scatter ? dispatch<true>(a, ws, num_sms, s, kAggFull)
                   : dispatch<false>(a, ws, num_sms, s, kAggFull);
}

cudaError_t agg_tables_launch(const AggArgs& a, void* ws_base, int num_sms, cudaStream_t s)
{
    AggWs ws;
    agg_ws_layout(a.n, static_cast<char*>(ws_base), &ws);
    return dispatch<false>(a, ws, num_sms, s, kAggTables);
}

cudaError_t agg_stage_launch(const AggArgs& a, void* ws_base, int num_sms, cudaStream_t s,
                             const BrkArgs* brk, void* brk_ws, bool* brk_done)
{
    AggWs ws;
    agg_ws_layout(a.n, static_cast<char*>(ws_base), &ws);
    PrepStage st{};
    st.rhs = a.rhs;
    if (brk) {
        st.brk = *brk;
        brk_ws_layout(a.n, brk->n_quad, static_cast<char*>(brk_ws), &st.bws);
    }
    *brk_done = false;
    return dispatch<false>(a, ws, num_sms, s, kAggStage, &st, brk_done);
}

} // namespace pbe_gb300
