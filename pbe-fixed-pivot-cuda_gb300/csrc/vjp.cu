// =============================================================================
// vjp.cu -- vector-Jacobian products (adjoints) of the aggregation and
// breakage RHS, FP64, sm_103a. No counterpart in the reference.
//
// Given lambda = dL/drhs, the calls ADD dL/dN into gN and dL/d(parameters)
// into a small device array, like the forward calls add into rhs.
//
// Aggregation. For pair p = (j <= k): rate_p = c_p beta_jk N_j N_k (c = 1/2 on
// the diagonal), L = sum_p rate_p G_p with G_p = P_p - lambda_j - lambda_k,
// P_p = lambda_lo + w (lambda_hi - lambda_lo) (lambda_{n-1} for pairs clipped
// at x[n-1]). Then
//   dL/dN_m  = sum_k G(m,k) beta(m,k) N_k           (all partners k, k = m once)
//   dL/dbeta_X = 1/2 sum_m N_m A_X[m],  A_X[m] = sum_k G(m,k) f_X(m,k) N_k
// where beta = sum_X beta_X f_X. The -lambda_m - lambda_k part of G reduces to
// moments of N and of lambda*N (as the forward death term); the P part is a
// row gather: row m meets each partner k once as the smaller member
// ("upper", lo = m + Ld[k-m]) and once as the larger ("lower",
// lo = k + Ld[m-k]). P uses the reference's weight numerator fl(x_j + x_k) -
// x_lo (integer pipe) times (lambda_{lo+1} - lambda_lo)/(x_{lo+1} - x_lo).
// One CTA owns each row tile and reduces it in a fixed order -> deterministic.
//
// Breakage. rhs_i = -S_i N_i + sum_j S_j N_j sum_q bw_q eta_i(x_j t_q) over
// the guarded parents. With Q_j = -lambda_j + sum_q bw_q P_jq:
//   dL/dN_j = S_j Q_j, dL/dS0 = sum_j (S_j/S0) N_j Q_j, dL/dv_ref, dL/dalpha
// (PowerLaw: dS/dalpha = S ln(x/v_ref)), dL/dv_min = 0 (threshold step).
// =============================================================================
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "pbe_internal.cuh"
#include "vjp_tile.cuh"

namespace pbe_gb300 {
namespace {

constexpr int VW = kVW;                 // rows per task

// dL/dN needs, per kernel type K, up to two row sums (see vjp_main_kernel):
//   K=0: R0 = sum P N_k                       f = 1
//   K=1: R0 = sum P N_k, R1 = sum P h_k       f N_k = x_m N_k + h_k
//   K=2: R0 = sum P h_k                       f N_k = x_m h_k
//   K=3: R0 = sum P N_k Bf                    Brownian factor per lag
//   K=4: R1 = sum_upper P N_k Sf + sum_lower P N_k Sl (shear f = x_min Sf;
//        on a geometric grid x_min = x_k = x_m x_0/x_d for a lower partner, so
//        f = x_m Sl with Sl = Sf x_0/x_d and both visits sum into R1, times x_m)
//   K=5: R0, R1 as K=3 and K=4
// The generic (non-geometric) path accumulates sum P N_k f directly: R0 for
// K=0..3 (f = f_0 or Bf), R1 for the shear part.

// -------------------------------------------------------------------------
// prep: per-bin values, lag factors (no beta, no diagonal 1/2), moments of N
// and lambda*N, geometric deviation, and the sums over the bins that the lags
// from D0 on reduce to (VjpWs::mloc). Block partials as VjpWs::mom, the maximum
// deviation in slot 10 and the smallest D0 candidate in slot 11.
// Modes: kVjpFull everything; kVjpTables the grid-only part (cube roots, lag
// tables, bracket offsets, deviation) for callers that keep the workspace for
// one set of pivots (the RK4 tape); kVjpStage the N- and lambda-dependent
// part (x N, D, moments) on such a workspace, with kVjpFull's arithmetic.
// Four pairs of warps share the 64 bins of a block, since the kernel is a chain of
// dependent FP64 instructions: each pair does one of the four scans and its share of
// the block's 25 moment sums, and before that (not kVjpStage) a part of the tables --
// pair 0 the cube roots, pair 1 the brackets, pair 2 the bins' logarithms, pair 3 the
// geometric fit and the cube root of x_0. (One pair for everything: n = 16384 31 us,
// 23 with four; a stage at n = 3840 19.4 and 10.6.)
// -------------------------------------------------------------------------
enum { kVjpFull = 0, kVjpTables = 1, kVjpStage = 2 };

// Running sums of v over the prep block's bins, from the first up (SUF = false)
// or from the last down (true); SCALED: each bin's value is relative to 2^E
// (prefix: the sum at bin i stands at 2^E_i, a term of a lower bin is scaled
// down; suffix: at 2^-E_i, a term of a higher bin is scaled down). By one of the block's
// pairs of warps, which meet at barrier 1 + pair; sv, se: the pair's.
template <bool SUF, bool SCALED>
__device__ __forceinline__ void block_scan(double* v, int E, int pair, double* sv, int* se)
{
    const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) & 1;
    static_assert(kPrepThreads == 64, "two warps");
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int Es = SUF ? __shfl_down_sync(0xffffffffu, E, o) : __shfl_up_sync(0xffffffffu, E, o);
        const int sh = SUF ? E - Es : Es - E;
#pragma unroll
        for (int q = 0; q < kMomN; ++q) {
            const double u = SUF ? __shfl_down_sync(0xffffffffu, v[q], o)
                                 : __shfl_up_sync(0xffffffffu, v[q], o);
            if (SUF ? lane + o < 32 : lane >= o) v[q] += SCALED ? scale_down(u, sh) : u;
        }
    }
    if (SUF ? (w == 1 && lane == 0) : (w == 0 && lane == 31)) {
        *se = E;
#pragma unroll
        for (int q = 0; q < kMomN; ++q) sv[q] = v[q];
    }
    asm volatile("bar.sync %0, %1;" :: "r"(1 + pair), "n"(kPrepThreads) : "memory");
    if (SUF ? w == 0 : w == 1) {
        const int sh = SUF ? E - *se : *se - E;
#pragma unroll
        for (int q = 0; q < kMomN; ++q) v[q] += SCALED ? scale_down(sv[q], sh) : sv[q];
    }
}

constexpr int kVPrepThreads = 4 * kPrepThreads;

template <int MODE>
__global__ void __launch_bounds__(kVPrepThreads)
vjp_prep_kernel(const double* __restrict__ N, const double* __restrict__ x,
                const double* __restrict__ lam, int n, VjpWs ws)
{
    const int dep = dep_wait();
    N += dep; x += dep; lam += dep; n += dep;
    __shared__ double sh[kPrepThreads / 32][kVjpMom];
    __shared__ double sv[4][kMomN];
    __shared__ int se[4];
    __shared__ double a_s[kPrepThreads], ia_s[kPrepThreads];
    __shared__ double ax0_s;
    __shared__ GeoFit fit_s;
    const int pair = threadIdx.x / kPrepThreads, t = threadIdx.x % kPrepThreads;
    const int i = blockIdx.x * kPrepThreads + t;
    const int lane = threadIdx.x & 31, wp = t >> 5;
    const int nb = gridDim.x, b = blockIdx.x;
    const double xi = x[min(i, n - 1)];          // bins beyond the last add zeros
    int Ei = 0;
    double fi = 0.0, ai = 0.0, iai = 0.0;
    if constexpr (MODE != kVjpStage) {
        if (pair == 0) {
            ai = cbrt(xi);
            iai = 1.0 / ai;
            a_s[t] = ai;
            ia_s[t] = iai;
            if (i < n) { ws.a[i] = ai; ws.ia[i] = iai; }
        } else if (pair == 1) {
            int d0 = n;
            if (i < n) {
                const double v = x[0] + xi;
                const int L = (dbits(v) >= dbits(x[n - 1])) ? kLagClipAll : bracket_from(x, n, v, i);
                ws.Ld[i] = L;
                if (L == i && i > 0) d0 = i;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) d0 = min(d0, __shfl_xor_sync(0xffffffffu, d0, o));
            if (lane == 0) sh[wp][11] = static_cast<double>(d0);
        } else if (pair == 2) {
            Ei = ilogb(xi);
            fi = log2(scalbn(xi, -Ei));
        } else if (wp == 0) {
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
        __syncthreads();
        ai = a_s[t];
        iai = ia_s[t];
        if (pair == 1 && i < n) {
            const double rho = ai / ax0_s;
            ws.Bf[i] = rho + 1.0 / rho + 2.0;
            const double u = 1.0 + rho;
            ws.Sf[i] = (u * u) * u;
            ws.Sl[i] = (u * u) * u * (x[0] / xi);
        } else if (pair == 2) {
            double dev = (i < n && n >= 2) ? geo_dev_from(fit_s, Ei, fi, i) : 0.0;
            if (!(dev == dev)) dev = 1.0;        // NaN -> not geometric
            dev = warp_max(dev);
            if (lane == 0) sh[wp][10] = dev;
        }
    } else {
        if (i < n) { ai = ws.a[i]; iai = ws.ia[i]; }
    }
    if constexpr (MODE != kVjpTables) {
        double w[kMomN] = {0.0, 0.0, 0.0, 0.0, 0.0};
        double Ni = 0.0, li = 0.0, Di = 0.0, dl = 0.0, u = 0.0;
        if (i < n) {
            Ni = N[i];
            li = lam[i];
            if (pair >= 2 && i < n - 1) {
                const double xu = x[i + 1], dx = xu - xi;
                dl = lam[i + 1] - li;
                if (pair == 3) Di = dl / dx; else u = 1.1102230246251565e-16 * (xu / dx);
            }
            if (pair == 0) ws.h[i] = xi * Ni;
            if (pair == 3) ws.D[i] = Di;
            w[0] = iai; w[1] = 1.0; w[2] = ai; w[3] = ai * ai; w[4] = xi;
        }
        // the block's share of the moments: slots 0.. (N), 5.. (lambda N), 12.. (|N|),
        // 17.. (|lambda N|), 22.. (u |N| |lambda step|)
        auto moments = [&](int slot, double c) {
#pragma unroll
            for (int q = 0; q < kMomN; ++q) {
                const double m = warp_sum(w[q] * c);
                if (lane == 0) sh[wp][slot + q] = m;
            }
        };
        const int E = exponent_of(xi);
        // the sums over the bins: group k = the pair
        double v[kMomN];
        auto fill = [&](double c) {
#pragma unroll
            for (int q = 0; q < kMomN; ++q) v[q] = w[q] * c;
        };
        if (pair == 0) {
            moments(0, Ni);
            fill(Ni);
            block_scan<false, false>(v, E, pair, sv[pair], &se[pair]);
        } else if (pair == 1) {
            moments(5, li * Ni);
            moments(17, fabs(li * Ni));
            const double xm = mantissa_of(xi);
#pragma unroll
            for (int q = 0; q < kMomN; ++q) v[q] = (w[q] * Ni) * xm;
            block_scan<false, true>(v, E, pair, sv[pair], &se[pair]);
        } else if (pair == 2) {
            moments(22, u * fabs(dl * Ni));
            fill(li * Ni);
            block_scan<true, false>(v, E, pair, sv[pair], &se[pair]);
        } else {
            moments(12, fabs(Ni));
            fill(Ni * scalbn(Di, E));
            block_scan<true, true>(v, E, pair, sv[pair], &se[pair]);
        }
        const int first = b * kPrepThreads, last = min(n - 1, first + kPrepThreads - 1);
        const int edge = pair >= 2 ? first : last;
#pragma unroll
        for (int q = 0; q < kMomN; ++q) {
            if (i < n) ws.mloc[static_cast<size_t>(pair * kMomN + q) * n + i] = v[q];
            if (i == edge) ws.mtot[(pair * kMomN + q) * nb + b] = v[q];
        }
    }
    __syncthreads();
    if (threadIdx.x < kVjpMom) {
        const int q = threadIdx.x;
        const double s0 = sh[0][q], s1 = sh[1][q];
        const bool grid_only = q == 10 || q == 11;
        if (q < 27 && (MODE == kVjpFull || (MODE == kVjpTables) == grid_only))
            ws.mom_part[b * kVjpMom + q] = q == 10 ? fmax(s0, s1) : q == 11 ? fmin(s0, s1) : s0 + s1;
    }
}

// One block: the reductions over the prep blocks' partials, spread over the
// warps: warps 0..3 scan the block totals of the four groups of sums into
// offsets (each lane a run of consecutive blocks, a warp scan over the runs);
// warps 4..14 the moments (kVjpFull, kVjpStage), the geometric flag and D0
// (kVjpFull, kVjpTables), lanes striding over the blocks, fixed butterflies.
// Resets the task counters (kVjpFull, kVjpStage). Then warp 15 tries 32 rows spread over
// the grid for the rule of the exact rows (vjp_row_exact) and decides for the lags of
// all (vjp_direct_lags into counter[2]): rows of one kind lie together, so a row among them
// that keeps its exact sum stands for many.
constexpr int kVFinThreads = 512;

// Row m of a geometric grid takes its lags from D0 on pair by pair (vjp_lane_rows_kernel
// derives the rule).
struct RowOfRule {
    double x, a, ia, l, ul;      // the row's pivot, its powers 1/3 and -1/3, |lambda_m|, u_m |lambda_{m+1}|
    __device__ __forceinline__ RowOfRule(const double* __restrict__ xp, const double* __restrict__ lam,
                                         const VjpWs& ws, int n, int m)
        : x(xp[m]), a(ws.a[m]), ia(ws.ia[m]), l(fabs(lam[m])), ul(0.0)
    {
        if (m < n - 1) {
            const double xu = xp[m + 1];
            ul = 1.1102230246251565e-16 * (xu / (xu - x)) * fabs(lam[m + 1]);
        }
    }
};
// mom: slots 12.. of VjpWs::mom.
template <int K>
__device__ __forceinline__ bool vjp_row_exact(const RowOfRule& r, const double* mom, double b0, double bbr,
                                              double bsh)
{
    const double c0 = fabs(b0), c1 = fabs(bbr), c2 = fabs(bsh);
    const double A = death_factor<K>(r.x, r.a, r.ia, mom, c0, c1, c2);
    const double AL = death_factor<K>(r.x, r.a, r.ia, mom + 5, c0, c1, c2);
    const double err = fma(r.ul, A, death_factor<K>(r.x, r.a, r.ia, mom + 10, c0, c1, c2));
    return err > kVjpGuard * fma(r.l, A, AL);
}

// Lags summed pair by pair: those below D0; all of them where `rows` of the 32 rows tried
// are exact and exact rows would take longer. An exact row takes its block 8 to 12 n
// clocks, one after the other (taken as 16 a row tried, at most the block's 32); all lags
// instead of those below D0 take the chip 0.01 (n - D0)^2 clocks. (lambda 1 above the
// largest particles and 0 below, where nearly every row is exact: by exact rows 64
// sections took 387 us, 960 443 and 16384 2.67 ms.)
__device__ __forceinline__ int vjp_direct_lags(int n, int D0, int rows)
{
    const double d = static_cast<double>(n - D0);
    return 1200.0 * min(32, 16 * rows) * n > d * d ? n : min(n, D0);
}

template <int MODE>
__global__ void __launch_bounds__(kVFinThreads)
vjp_fin_kernel(const double* __restrict__ x, const double* __restrict__ lam, int n, VjpWs ws, int kernel,
               double b0, double bbr, double bsh)
{
    const int dep = dep_wait();
    x += dep; lam += dep; n += dep;
    const int nb = (n + kPrepThreads - 1) / kPrepThreads;
    const int wq = threadIdx.x >> 5, lq = threadIdx.x & 31;
    if (wq < 4) {
        if (MODE == kVjpTables) return;
        const bool suf = wq >= 2, scaled = (wq & 1) != 0;
        const int per = (nb + 31) / 32;
        const int k0 = min(nb, lq * per), k1 = min(nb, k0 + per);
        // k-th block in the scan's direction, and the exponent its total stands at
        auto blk = [&](int k) { return suf ? nb - 1 - k : k; };
        auto tag = [&](int k) {
            const int b = blk(k);
            return exponent_of(__ldg(x + (suf ? b * kPrepThreads : min(n - 1, (b + 1) * kPrepThreads - 1))));
        };
        auto shift = [&](double v, int from, int to) {
            return scaled ? scale_down(v, suf ? to - from : from - to) : v;
        };
        const double* tot = ws.mtot + static_cast<size_t>(wq) * kMomN * nb;
        double* off = ws.moff + static_cast<size_t>(wq) * kMomN * nb;
        const int e0 = k0 > 0 ? tag(k0 - 1) : tag(0), e1 = k1 > 0 ? tag(k1 - 1) : e0;
        double S[kMomN], R[kMomN];
#pragma unroll
        for (int q = 0; q < kMomN; ++q) S[q] = 0.0;
        int e = e0;
        // kRun blocks' totals and exponents at a time, loaded together (as the forward's
        // prep_offsets: a load at a time is a chain of 0.7 us each)
        constexpr int kRun = 4;
        double t[kRun][kMomN];
        int en[kRun];
        auto load = [&](int k) {
#pragma unroll
            for (int u = 0; u < kRun; ++u) {
                const int c = min(k + u, nb - 1);
                en[u] = tag(c);
#pragma unroll
                for (int q = 0; q < kMomN; ++q) t[u][q] = tot[q * nb + blk(c)];
            }
        };
        for (int k = k0; k < k1; k += kRun) {
            load(k);
#pragma unroll
            for (int u = 0; u < kRun; ++u) {
                if (k + u >= k1) break;
#pragma unroll
                for (int q = 0; q < kMomN; ++q) S[q] = shift(S[q], e, en[u]) + t[u][q];
                e = en[u];
            }
        }
#pragma unroll
        for (int q = 0; q < kMomN; ++q) R[q] = S[q];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int es = __shfl_up_sync(0xffffffffu, e1, o);
#pragma unroll
            for (int q = 0; q < kMomN; ++q) {
                const double r = __shfl_up_sync(0xffffffffu, R[q], o);
                if (lq >= o) R[q] += shift(r, es, e1);
            }
        }
#pragma unroll
        for (int q = 0; q < kMomN; ++q) {
            const double r = __shfl_up_sync(0xffffffffu, R[q], 1);
            S[q] = lq > 0 ? r : 0.0;
        }
        e = e0;
        for (int k = k0; k < k1; k += kRun) {
            load(k);
#pragma unroll
            for (int u = 0; u < kRun; ++u) {
                if (k + u >= k1) break;
#pragma unroll
                for (int q = 0; q < kMomN; ++q) {
                    off[q * nb + blk(k + u)] = S[q];
                    S[q] = shift(S[q], e, en[u]) + t[u][q];
                }
                e = en[u];
            }
        }
        return;
    }
    __shared__ double mom_s[27];
    if (wq == kVFinThreads / 32 - 1) {
        if (MODE == kVjpTables) return;
        const int m = static_cast<int>((2LL * lq + 1) * n / 64);
        const RowOfRule row(x, lam, ws, n, m);
        asm volatile("bar.sync 1, %0;" :: "n"(kVFinThreads - 128) : "memory");   // warps 4..15
        const int D0 = static_cast<int>(MODE == kVjpFull ? mom_s[11] : ws.mom[11]);
        const bool geo = (MODE == kVjpFull ? mom_s[10] : ws.mom[10]) != 0.0;
        const double* M = mom_s + 12;
        bool ex = false;
        if (geo && (m >= D0 || m + D0 < n)) {
            switch (kernel) {
            case 0: ex = vjp_row_exact<0>(row, M, b0, bbr, bsh); break;
            case 1: ex = vjp_row_exact<1>(row, M, b0, bbr, bsh); break;
            case 2: ex = vjp_row_exact<2>(row, M, b0, bbr, bsh); break;
            case 3: ex = vjp_row_exact<3>(row, M, b0, bbr, bsh); break;
            case 4: ex = vjp_row_exact<4>(row, M, b0, bbr, bsh); break;
            default: ex = vjp_row_exact<5>(row, M, b0, bbr, bsh); break;
            }
        }
        const unsigned rows = __ballot_sync(0xffffffffu, ex);
        if (lq == 0) {
            ws.counter[0] = 0;
            ws.counter[1] = 0;
            ws.counter[2] = vjp_direct_lags(n, D0, __popc(rows));
        }
        return;
    }
    for (int r = wq - 4; r < 27; r += kVFinThreads / 32 - 5) {
        double t = 0.0;
        if (r == 10 || r == 11) {
            if (MODE == kVjpStage) continue;
            if (r == 11) t = static_cast<double>(n);
            for (int b = lq; b < nb; b += 32) {
                const double v = ws.mom_part[b * kVjpMom + r];
                t = r == 10 ? fmax(t, v) : fmin(t, v);
            }
            t = r == 10 ? warp_max(t) : -warp_max(-t);
            // the largest deviation decides the geometric flag
            const bool ratio_ok = n >= 2 && x[1] <= 64.0 * x[0];
            if (r == 10) t = (n >= 2 && t <= kGeoTol && ratio_ok) ? 1.0 : 0.0;
        } else {
            if (MODE == kVjpTables) continue;
#pragma unroll 8
            for (int b = lq; b < nb; b += 32) t += ws.mom_part[b * kVjpMom + r];
            t = warp_sum(t);
        }
        if (lq == 0) { ws.mom[r] = t; mom_s[r] = t; }
    }
    if (MODE != kVjpTables)
        asm volatile("bar.sync 1, %0;" :: "n"(kVFinThreads - 128) : "memory");
}

// Pair sums: task = (row tile, partner chunk); the whole CTA is one group.
// Each task stores its rows' two sums per chunk; vjp_rows_kernel adds the
// chunks in order and finishes the rows.
// lane_on: the lane-block kernel takes geometric grids (this one returns).
template <int K>
__global__ void __launch_bounds__(kMainThreads, 2)
vjp_main_kernel(const double* __restrict__ N, const double* __restrict__ x,
                const double* __restrict__ lam, VjpWs ws, int n, int ntile, int nch, int lane_on)
{
    const int dep = dep_wait();
    N += dep; x += dep; lam += dep; n += dep;
    extern __shared__ double red[];               // [kVRows][kMainThreads]
    __shared__ VjpShared sm;
    __shared__ int s_task;

    if (lane_on && ws.mom[10] != 0.0) return;
    const int tid = threadIdx.x;
    VjpCellView v;
    v.x = x; v.N = N; v.h = ws.h; v.lam = lam; v.D = ws.D; v.a = ws.a; v.ia = ws.ia;
    v.Bf = ws.Bf; v.Sf = ws.Sf; v.Sl = ws.Sl; v.Ld = ws.Ld; v.lag0_scale = 1.0;
    v.n = n;
    v.geo = ws.mom[10] != 0.0;
    const TileGroup G{0, tid, kMainThreads};
    const int span = (n + nch - 1) / nch;

    for (;;) {
        if (tid == 0) s_task = atomicAdd(ws.counter, 1);
        __syncthreads();
        const int task = s_task;
        __syncthreads();
        if (task >= ntile * nch) break;
        const int tile = task / nch, chunk = task - tile * nch;
        const int r0 = min(n, chunk * span), r1 = min(n, r0 + span);
        vjp_tile_accumulate<K>(v, tile * VW, r0, r1, red, sm, G);
        if (tid < kVRows) ws.vpart[(static_cast<size_t>(tile) * nch + chunk) * kVRows + tid] = sm.fin[0][tid];
        __syncthreads();
    }
}

// The rows of one row tile by a warp: sums the tile's chunks in order, adds each
// row's dL/dN_m and stores the tile's parameter partials (fixed order). fin: kVRows
// doubles of shared memory.
template <int K>
__device__ __forceinline__ void tile_rows(const double* __restrict__ N, const double* __restrict__ x,
                                          const double* __restrict__ lam, double* __restrict__ gN,
                                          const VjpWs& ws, int n, int tile, int nch, bool geo, double b0,
                                          double bbr, double bsh, double* fin)
{
    const int lane = threadIdx.x & 31;
    for (int r = lane; r < kVRows; r += 32) {
        double s = 0.0;
        for (int c = 0; c < nch; ++c) s += ws.vpart[(static_cast<size_t>(tile) * nch + c) * kVRows + r];
        fin[r] = s;
    }
    __syncwarp();
    VjpCellView v;
    v.x = x; v.N = N; v.h = ws.h; v.lam = lam; v.D = ws.D; v.a = ws.a; v.ia = ws.ia;
    v.Bf = ws.Bf; v.Sf = ws.Sf; v.Sl = ws.Sl; v.Ld = ws.Ld; v.lag0_scale = 1.0;
    v.n = n;
    v.geo = geo;
    const int I = tile * VW;
    double gB = 0.0, gS = 0.0;
    if (lane < VW && I + lane < n) {
        double g;
        vjp_tile_row<K>(v, I + lane, lane, fin, ws.mom, ws.mom + 5, b0, bbr, bsh, g, gB, gS);
        gN[I + lane] += g;
    }
    double s0 = 0.0, s1 = 0.0;
    for (int t = 0; t < VW; ++t) {
        s0 += __shfl_sync(0xffffffffu, gB, t);
        s1 += __shfl_sync(0xffffffffu, gS, t);
    }
    if (lane == 0) {
        // slots: 0 beta0, 1 beta_br, 2 beta_sh
        ws.gpart[tile * 4 + 0] = (K <= 2) ? s0 : 0.0;
        ws.gpart[tile * 4 + 1] = (K == 3 || K == 5) ? s0 : 0.0;
        ws.gpart[tile * 4 + 2] = (K == 4 || K == 5) ? s1 : 0.0;
    }
}

template <int K>
__global__ void __launch_bounds__(256)
vjp_rows_kernel(const double* __restrict__ N, const double* __restrict__ x,
                const double* __restrict__ lam, double* __restrict__ gN, VjpWs ws, int n,
                int ntile, int nch, double b0, double bbr, double bsh)
{
    const int dep = dep_wait();
    N += dep; x += dep; lam += dep; gN += dep; n += dep;
    __shared__ double fin[8][kVRows];
    const int w = threadIdx.x >> 5, tile = blockIdx.x * 8 + w;
    if (tile < ntile)                             // whole warps
        tile_rows<K>(N, x, lam, gN, ws, n, tile, nch, ws.mom[10] != 0.0, b0, bbr, bsh, fin[w]);
}

// Parameter sums, one block: slots 0..2 of the aggregation's gp (warps 0..2; none if
// null) from its tasks' partials -- ntile of them, or nlane > 0 on a geometric grid, where
// the lane rows kernel wrote them -- and slots 0..3 of the breakage's bgp (warps 4..7;
// none if null) from nb blocks', each by a warp in a fixed order.
__global__ void __launch_bounds__(256) vjp_gfin_kernel(int ntile, int nlane, VjpWs ws, double* gp, int nb, double* bgp)
{
    dep_wait();
    const int w = threadIdx.x >> 5, q = w & 3, l = threadIdx.x & 31;
    double* out = w < 4 ? gp : bgp;
    if (!out || w == 3) return;
    const double* part = w < 4 ? ws.gpart : ws.bpart;
    const int cnt = w >= 4 ? nb : (nlane > 0 && ws.mom[10] != 0.0) ? nlane : ntile;
    double s = 0.0;
    for (int b = l; b < cnt; b += 32) s += part[b * 4 + q];
    s = warp_sum(s);
    if (l == 0) out[q] += s;
}

// -------------------------------------------------------------------------
// Lane blocks (geometric grids). Lane l of a warp owns row j = 32 b + l and
// walks the lags d of its share: the pair (j, k = j + d) lands at
// lo = j + Ld[d], P = lambda_lo + (fl(x_j + x_k) - x_lo) D_lo (lambda_{n-1} when
// clipped). The row of the smaller member sums in registers (U0, U1: the
// tile path's sums of the upper visits); the row of the larger member,
// k = j + d, is the row lane l + 1 held one lag earlier, so its sum W (the
// whole lower-visit term, parameters included) moves one lane down per lag;
// lane 0's finished W leaves the warp each lag into a shared window, and
// every lane's W at the end of the share. Brownian + shear: 7 FP64
// instructions per pair (P; P Bf, P Sf; two sums of the smaller member; two
// FMAs into W) against 8 for the two visits of the tile path.
// Only the lags below D0: from there on every pair lands on its larger member's
// own slot, lo = k, and the sums separate (vjp_lane_rows_kernel; vjp_direct_lags
// tells when all lags are summed here after all).
// Tasks (row block, lag chunk) run chunk by chunk; all but the lowest-lag rows'
// have equal length. Determinism: the windows of the CTA's warps are added in
// warp order; the rows kernel adds the tasks' sums in a fixed order.
// -------------------------------------------------------------------------
#ifndef PBE_VJP_LANE_CTAS
#define PBE_VJP_LANE_CTAS 3
#endif
constexpr int kVLaneCtas = PBE_VJP_LANE_CTAS;
constexpr int kLaneWarps = kMainThreads / 32;   // warps sharing a task's lags
#ifdef PBE_VJP_UNROLL
constexpr int kVjpUnroll = PBE_VJP_UNROLL;
#endif
constexpr int kVLaneMaxChunks = 64;        // vjp_lane_chunks(n, C) bound

template <int K>
__global__ void __launch_bounds__(kMainThreads, kVLaneCtas)
vjp_lane_kernel(const double* __restrict__ N, const double* __restrict__ x,
                const double* __restrict__ lam, VjpWs ws, int n, int C,
                double b0, double bbr, double bsh)
{
    const int dep = dep_wait();
    N += dep; x += dep; lam += dep; n += dep;
    extern __shared__ double esm[];               // [kLaneWarps][per_max + 32] W windows
    __shared__ double red[kLaneWarps][2][kLaneBins];
    __shared__ int s_task;

    if (ws.mom[10] == 0.0) return;                // not geometric: the tile kernel runs
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const double* __restrict__ h = ws.h;
    const double* __restrict__ D = ws.D;
    const int* __restrict__ Ld = ws.Ld;
    const double lamlast = lam[n - 1];
    const int ew = (C + kLaneWarps - 1) / kLaneWarps + 32;
    double* eb = esm + w * ew;
    const int Dm = ws.counter[2];

    for (;;) {
        if (tid == 0) s_task = atomicAdd(ws.counter + 1, 1);
        __syncthreads();
        const int task = s_task;
        __syncthreads();
        // task `task` of the chunk-major order: chunk c of row block b (lags
        // 1 + c C and up, below D0); tix is also where the rows kernel finds its sums
        int b = task, c = 0;
        while (1 + c * C < Dm) {
            const int cnt = vjp_lane_chunk_blocks(n, c, C);
            if (cnt == 0 || b < cnt) break;
            b -= cnt;
            ++c;
        }
        if (1 + c * C >= Dm || vjp_lane_chunk_blocks(n, c, C) == 0) break;
        const int tix = task;
        const int J = kLaneBins * b;
        const int dA = 1 + c * C;
        const int dB = min(min(dA + C, n - J), Dm);   // lags [dA, dB), dB - 1 <= n - 1 - J
        const int len = dB - dA;
        const int per = (len + kLaneWarps - 1) / kLaneWarps;
        const int dw0 = dA + w * per;
        const int dw1 = min(dB, dw0 + per);

        const int j = J + lane;
        const bool jv = j < n;
        const double xj = jv ? __ldg(x + j) : 0.0;
        const double Nj = jv ? __ldg(N + j) : 0.0;
        const double hj = jv ? h[j] : 0.0;
        // lane constants of the lower-visit term
        double cN = 0.0, cH = 0.0;
        if constexpr (K == 0) cN = b0 * Nj;
        if constexpr (K == 1) { cN = b0 * Nj; cH = b0 * hj; }
        if constexpr (K == 2) cH = b0 * hj;
        if constexpr (K == 3) cN = bbr * Nj;
        if constexpr (K == 4) cH = bsh * hj;
        if constexpr (K == 5) { cN = bbr * Nj; cH = bsh * hj; }
        const int jtop = n - 1 - j;               // lo >= n - 1 <=> Ld[d] >= jtop
        const EwOperandB pb = ew_operand_b(jv ? xj : 1.0);   // the row's pivot, decoded once

        double U0 = 0.0, U1 = 0.0, W = 0.0;
#ifdef PBE_VJP_UNROLL
#pragma unroll kVjpUnroll
#endif
        for (int d = dw0; d < dw1; ++d) {
            // lane 0's row (j + d - 1) is complete: out; every row moves one lane down
            const double Wd = __shfl_down_sync(0xffffffffu, W, 1);
            if (lane == 0) eb[d - dw0] = W;
            W = (lane == 31) ? 0.0 : Wd;
            const int L = __ldg(Ld + d);
            double Bf = 0.0, Sf = 0.0;
            if constexpr (K == 3 || K == 5) Bf = __ldg(ws.Bf + d);
            if constexpr (K == 4 || K == 5) Sf = __ldg(ws.Sf + d);
            const int k = j + d;
            if (k < n) {
                const double xk = __ldg(x + k);
                double P = lamlast;
                if (L < jtop) {
                    const int lo = j + L;
                    P = fma(sum_minus_scaled_dec(ew_operand_a(xk), pb, ew_operand_c(__ldg(x + lo), 0)),
                            D[lo], lam[lo]);
                }
                if constexpr (K == 0) {
                    U0 = fma(P, __ldg(N + k), U0);
                    W = fma(P, cN, W);
                } else if constexpr (K == 1) {
                    U0 = fma(P, __ldg(N + k), U0);
                    U1 = fma(P, h[k], U1);
                    W = fma(P, fma(cN, xk, cH), W);
                } else if constexpr (K == 2) {
                    U0 = fma(P, h[k], U0);
                    W = fma(P * xk, cH, W);
                } else {
                    const double Nk = __ldg(N + k);
                    if constexpr (K == 3 || K == 5) {
                        const double u0 = P * Bf;
                        U0 = fma(u0, Nk, U0);
                        W = fma(u0, cN, W);
                    }
                    if constexpr (K == 4 || K == 5) {
                        const double u1 = P * Sf;
                        U1 = fma(u1, Nk, U1);
                        W = fma(u1, cH, W);
                    }
                }
            }
        }
        if (dw1 > dw0) eb[dw1 - dw0 + lane] = W;  // rows j + dw1 - 1
        red[w][0][lane] = U0;
        red[w][1][lane] = U1;
        __syncthreads();
        if (w == 0) {
            double s0 = 0.0, s1 = 0.0;
#pragma unroll
            for (int q = 0; q < kLaneWarps; ++q) {
                s0 += red[q][0][lane];
                s1 += red[q][1][lane];
            }
            ws.lup[static_cast<size_t>(tix) * 2 * kLaneBins + lane] = s0;
            ws.lup[static_cast<size_t>(tix) * 2 * kLaneBins + kLaneBins + lane] = s1;
        }
        // the task's window: entry i is row J + dA - 1 + i, i < len + 32; warp q's
        // window starts at i = q per and holds its share's length + 32 entries
        double* seg = ws.llo + static_cast<size_t>(tix) * (C + 32);
        for (int i = tid; i < C + 32; i += kMainThreads) {   // zeros beyond len + 32
            double sum = 0.0;
            for (int q = 0; q < kLaneWarps; ++q) {
                const int q0 = q * per, q1 = min(len, q0 + per);
                if (q1 <= q0) break;
                const int o = i - q0;
                if (o >= 0 && o < q1 - q0 + 32) sum += esm[q * ew + o];
            }
            seg[i] = sum;
        }
        __syncthreads();
    }
}

// Sums over the bins (VjpWs::mloc) at bin i: group k's five values; for the
// scaled groups at i's exponent.
template <bool SUF, bool SCALED>
__device__ __forceinline__ void bin_sums(const VjpWs& ws, const double* __restrict__ x, int n, int k,
                                         int i, double* v)
{
    const int nb = agg_prep_blocks(n), b = i / kPrepThreads;
    int sh = 0;
    if (SCALED) {
        const int ib = SUF ? (b + 1) * kPrepThreads : b * kPrepThreads - 1;   // the neighbour block's edge
        const int eb = ib >= 0 && ib < n ? exponent_of(__ldg(x + ib)) : 0, ei = exponent_of(__ldg(x + i));
        sh = SUF ? ei - eb : eb - ei;
        if (ib < 0 || ib >= n) sh = 0;
    }
#pragma unroll
    for (int q = 0; q < kMomN; ++q) {
        const double o = ws.moff[(k * kMomN + q) * nb + b];
        v[q] = ws.mloc[static_cast<size_t>(k * kMomN + q) * n + i] + (SCALED ? scale_down(o, sh) : o);
    }
}

// Rows of the lane path: one CTA per row block b (rows 32 b + lane). Warp g
// adds the larger-member sums of the row blocks b' = g, g + 16, ... <= b (the
// chunk holding lag d = m - 32 b' and, for the first 32 lags of a chunk, the
// tail of the chunk before); warp 0 adds the 16 warps' in order, the block's own
// smaller-member sums chunk by chunk, the diagonal pair, the lags from D0 on,
// the death moments, and stores dL/dN_m and the block's parameter partials.
//
// Lags from D0 on: lo = k and fl(x_j + x_k) - x_k is x_j up to the sum's
// rounding, so P = lambda_k + x_j D_k and, with beta a sum of products of powers
// of x_j and x_k, row m's sums are
//   as the larger member   lambda_m beta[P(m - D0)] + D_m beta[T(m - D0)]
//   as the smaller member  beta[SL(m + D0)] + x_m beta[SD(m + D0)]
// (beta[M]: the death polynomial at x_m; P, T the moments of N and x N over the
// bins up to an index, SL, SD those of lambda N and D N from an index up).
// Leaving out the rounding changes P by at most u_k |lambda_{k+1} - lambda_k|,
// u_k = 2^-53 x_{k+1}/dx_k. Bounded over all partners with the moments of
// |N|, |lambda N| and u |N| |lambda step|, it may move a row by at most
// kVjpGuard of the row's sum of |terms|; rows where it could (a lambda that is
// nonzero on few bins) take their lags from D0 on pair by pair (vjp_row_exact).
#ifndef PBE_VROWS_WARPS
#define PBE_VROWS_WARPS 16
#endif
constexpr int kVRowsWarps = PBE_VROWS_WARPS;

template <int K>
__global__ void __launch_bounds__(kVRowsWarps * 32)
vjp_lane_rows_kernel(const double* __restrict__ N, const double* __restrict__ x,
                     const double* __restrict__ lam, double* __restrict__ gN, VjpWs ws, int n,
                     int C, int ntile, int nch, double b0, double bbr, double bsh)
{
    const int dep = dep_wait();
    N += dep; x += dep; lam += dep; gN += dep; n += dep;
    __shared__ double fin[kVRowsWarps][kVRows];
    __shared__ double lw[kVRowsWarps][kLaneBins];
    __shared__ int base[kVLaneMaxChunks + 1];
    __shared__ double xs3[3][kLaneBins];           // exact rows: larger-member sum, smaller-member sums
    __shared__ double red[kVRowsWarps];
    __shared__ unsigned exact_s;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (ws.mom[10] == 0.0) {                       // not geometric: the row tiles' sums
        for (int tile = blockIdx.x * kVRowsWarps + w; tile < ntile; tile += gridDim.x * kVRowsWarps)
            tile_rows<K>(N, x, lam, gN, ws, n, tile, nch, false, b0, bbr, bsh, fin[w]);
        return;
    }
    const int b = gridDim.x - 1 - blockIdx.x;      // top row blocks (the most lower blocks) first
    const int m = kLaneBins * b + lane;
    const int Dm = ws.counter[2];                  // lags below Dm were summed pair by pair
    int nchunks = 0;                               // chunks that hold such lags
    while (nchunks < kVLaneMaxChunks && 1 + nchunks * C < Dm && vjp_lane_chunk_blocks(n, nchunks, C) > 0) ++nchunks;
    if (threadIdx.x == 0) {
        int sacc = 0;
        for (int c = 0; c < nchunks; ++c) {
            base[c] = sacc;
            sacc += vjp_lane_chunk_blocks(n, c, C);
        }
    }
    // rows that take the other lags so too
    if (w == 0) {
        bool ex = false;
        if (m < n && (m >= Dm || m + Dm < n))
            ex = vjp_row_exact<K>(RowOfRule(x, lam, ws, n, m), ws.mom + 12, b0, bbr, bsh);
        const unsigned em = __ballot_sync(0xffffffffu, ex);
        if (lane == 0) exact_s = em;
    }
    __syncthreads();
    const unsigned exact = exact_s;
    const size_t S = static_cast<size_t>(C) + 32;
    double acc = 0.0;
    if (m < n && nchunks > 0) {
        // the loads of several row blocks in flight: addresses do not depend on acc.
        // Lower blocks whose window reaches row m: lags d < Dm + 32
        const float invC = 1.0f / static_cast<float>(C);
        const int bp0 = max(0, (kLaneBins * b - Dm) / kLaneBins - 1);
#pragma unroll 4
        for (int bp = bp0 + w; bp <= b; bp += kVRowsWarps) {
            const int d = m - kLaneBins * bp;
            // c1 = d / C: the float quotient, corrected by one either way
            int c1 = __float2int_rz(static_cast<float>(d) * invC);
            c1 -= (c1 * C > d) ? 1 : 0;
            c1 += ((c1 + 1) * C <= d) ? 1 : 0;
            const int idx = d - c1 * C;
            double v = 0.0;
            if (d >= 1) {
                if (c1 >= 1 && idx < 32 && c1 - 1 < nchunks)
                    v = __ldcg(ws.llo + (base[c1 - 1] + bp) * S + C + idx);
                // chunk c1 exists for block bp when its first lag 1 + c1 C <= n - 1 - 32 bp
                if (c1 < nchunks && 1 + c1 * C <= n - 1 - kLaneBins * bp)
                    v += __ldcg(ws.llo + (base[c1] + bp) * S + idx);
            }
            acc += v;
        }
    }
    lw[w][lane] = acc;
    __syncthreads();

    // exact rows, one after the other: the CTA over the partners, fixed order
    for (unsigned em = exact; em != 0u; em &= em - 1u) {
        const int le = __ffs(em) - 1, r = kLaneBins * b + le;
        const double xr = x[r], Dr = ws.D[r], lr = lam[r];
        const EwOperandA ar = ew_operand_a(xr);
        const EwOperandB br = ew_operand_b(xr);
        const EwOperandC cr = ew_operand_c(xr, 0);
        double W = 0.0, U0 = 0.0, U1 = 0.0;
        for (int j = threadIdx.x; j <= r - Dm; j += kVRowsWarps * 32) {     // r the larger member
            const int d = r - j;
            const double P = r < n - 1 ? fma(sum_minus_scaled_pre(ar, x[j], cr), Dr, lr) : lr;
            if constexpr (K == 0) W = fma(P, b0 * N[j], W);
            if constexpr (K == 1) W = fma(P, b0 * fma(N[j], xr, ws.h[j]), W);
            if constexpr (K == 2) W = fma(P * xr, b0 * ws.h[j], W);
            if constexpr (K == 3 || K == 5) W = fma(P * ws.Bf[d], bbr * N[j], W);
            if constexpr (K == 4 || K == 5) W = fma(P * ws.Sf[d], bsh * ws.h[j], W);
        }
        for (int k = r + Dm + threadIdx.x; k < n; k += kVRowsWarps * 32) {  // r the smaller member
            const int d = k - r;
            const double xk = x[k], Nk = N[k];
            double P = lam[k];
            if (k < n - 1)
                P = fma(sum_minus_scaled_dec(ew_operand_a(xk), br, ew_operand_c(xk, 0)), ws.D[k], P);
            if constexpr (K == 0) U0 = fma(P, Nk, U0);
            if constexpr (K == 1) U0 = fma(P, fma(xr, Nk, ws.h[k]), U0);
            if constexpr (K == 2) U0 = fma(P, xr * ws.h[k], U0);
            if constexpr (K == 3 || K == 5) U0 = fma(P * ws.Bf[d], Nk, U0);
            if constexpr (K == 4 || K == 5) U1 = fma(P * ws.Sf[d], xr * Nk, U1);
        }
        const double t[3] = {block_sum(W, red), block_sum(U0, red), block_sum(U1, red)};
        if (threadIdx.x < 3) xs3[threadIdx.x][le] = t[threadIdx.x];
        __syncthreads();
    }
    if (w != 0) return;

    double gB = 0.0, gS = 0.0;
    if (m < n) {
        double Wm = 0.0;
#pragma unroll
        for (int q = 0; q < kVRowsWarps; ++q) Wm += lw[q][lane];
        const int dmax = min(n - 1 - kLaneBins * b, Dm - 1);
        const int nchb = dmax >= 1 ? (dmax + C - 1) / C : 0;
        double U0 = 0.0, U1 = 0.0;
        for (int c = 0; c < nchb; ++c) {
            const double* up = ws.lup + static_cast<size_t>(base[c] + b) * 2 * kLaneBins;
            U0 += __ldcg(up + lane);
            U1 += __ldcg(up + kLaneBins + lane);
        }
        // diagonal pair (m, m), counted once
        const double xm = x[m], Nm = N[m], hm = ws.h[m], lm = lam[m];
        const int L0 = ws.Ld[0];
        double P = lam[n - 1];
        if (L0 < n - 1 - m) {
            const int lo = m + L0;
            P = fma(sum_minus_scaled(xm, xm, x[lo], 0), ws.D[lo], lam[lo]);
        }
        double d0 = 0.0, d1 = 0.0;
        if constexpr (K == 0) d0 = P * Nm;
        if constexpr (K == 1) { d0 = P * Nm; d1 = P * hm; }
        if constexpr (K == 2) d0 = P * hm;
        if constexpr (K == 3 || K == 5) d0 = (P * Nm) * ws.Bf[0];
        if constexpr (K == 4 || K == 5) d1 = (P * Nm) * ws.Sf[0];
        U0 += d0;
        U1 += d1;
        // Tv: the smaller-member sums (diagonal included) weighted as the kernel
        // factor f(m, k) N_k; Td: the diagonal's share
        double Tv0 = U0, Td0 = d0, Tv1 = 0.0, Td1 = 0.0;
        if constexpr (K == 1) { Tv0 = fma(xm, U0, U1); Td0 = fma(xm, d0, d1); }
        if constexpr (K == 2) { Tv0 = xm * U0; Td0 = xm * d0; }
        if constexpr (K == 4 || K == 5) { Tv1 = xm * U1; Td1 = xm * d1; }
        const double am = ws.a[m], iam = ws.ia[m];
        // the lags from D0 on
        if ((exact >> lane) & 1u) {
            Wm += xs3[0][lane];
            Tv0 += xs3[1][lane];
            Tv1 += xs3[2][lane];
        } else {
            const int Em = exponent_of(xm);
            if (m >= Dm) {
                double p[kMomN], t[kMomN];
                bin_sums<false, false>(ws, x, n, 0, m - Dm, p);
                Wm = fma(lm, death_factor<K>(xm, am, iam, p, b0, bbr, bsh), Wm);
                if (m < n - 1) {
                    bin_sums<false, true>(ws, x, n, 1, m - Dm, t);
                    const double ft = death_factor<K>(xm, am, iam, t, b0, bbr, bsh);
                    Wm += scale_down(scalbn(ws.D[m], Em) * ft, exponent_of(x[m - Dm]) - Em);
                }
            }
            if (m + Dm < n) {
                double sl[kMomN], sd[kMomN];
                bin_sums<true, false>(ws, x, n, 2, m + Dm, sl);
                bin_sums<true, true>(ws, x, n, 3, m + Dm, sd);
                const int sh = Em - exponent_of(x[m + Dm]);
                const double xmm = mantissa_of(xm);
                if constexpr (K != 4)
                    Tv0 += moment_factor<K, 0>(xm, am, iam, sl) +
                           scale_down(xmm * moment_factor<K, 0>(xm, am, iam, sd), sh);
                if constexpr (K == 4 || K == 5)
                    Tv1 += moment_factor<K, 1>(xm, am, iam, sl) +
                           scale_down(xmm * moment_factor<K, 1>(xm, am, iam, sd), sh);
            }
        }
        const double* M = ws.mom;
        const double* Lm = ws.mom + 5;
        double g = Wm;
        if constexpr (K != 4) {
            const double dth0 = fma(lm, moment_factor<K, 0>(xm, am, iam, M), moment_factor<K, 0>(xm, am, iam, Lm));
            const double coef = (K <= 2) ? b0 : bbr;
            g = fma(coef, Tv0 - dth0, g);
            gB = Nm * Tv0 - 0.5 * Nm * (Td0 + dth0);
        }
        if constexpr (K == 4 || K == 5) {
            const double dth1 = fma(lm, moment_factor<K, 1>(xm, am, iam, M), moment_factor<K, 1>(xm, am, iam, Lm));
            g = fma(bsh, Tv1 - dth1, g);
            gS = Nm * Tv1 - 0.5 * Nm * (Td1 + dth1);
        }
        gN[m] += g;
    }
    const double s0 = warp_sum(gB);
    const double s1 = warp_sum(gS);
    if (lane == 0) {
        // slots: 0 beta0, 1 beta_br, 2 beta_sh
        ws.gpart[b * 4 + 0] = (K <= 2) ? s0 : 0.0;
        ws.gpart[b * 4 + 1] = (K == 3 || K == 5) ? s0 : 0.0;
        ws.gpart[b * 4 + 2] = (K == 4 || K == 5) ? s1 : 0.0;
    }
}

// -------------------------------------------------------------------------
// breakage VJP: nqp lanes per parent j (nqp = n_quad rounded up to a power of
// two, <= 32), each lane the fragments q = l % nqp, + nqp, ... (their bracket
// searches run side by side), summed over the lanes by a fixed butterfly;
// block partials of the parameter sums.
// -------------------------------------------------------------------------
template <int F>
__global__ void __launch_bounds__(256)
brk_vjp_kernel(const double* __restrict__ N, const double* __restrict__ x,
               const double* __restrict__ t_q, const double* __restrict__ bw_q,
               const double* __restrict__ lam, double* __restrict__ gN, double* part, int n,
               int nq, int nqp, double S0, double v_ref, double alpha, double v_min,
               const double* __restrict__ Ssel, const int* __restrict__ lo_tab)
{
    const int dep = dep_wait();
    N += dep; x += dep; t_q += dep; bw_q += dep; lam += dep; gN += dep; Ssel += dep; lo_tab += dep; n += dep;
    __shared__ double sh[8];
    const int l = threadIdx.x % nqp;
    const int j = (blockIdx.x * blockDim.x + threadIdx.x) / nqp;
    double p0 = 0.0, p1 = 0.0, p2 = 0.0;
    double S = 0.0, Nj = 0.0, xj = 1.0;
    bool on = false;
    double acc = 0.0;
    const float lx0 = log2_approx(__ldg(x));
    const float span = log2_approx(__ldg(x + n - 1)) - lx0;
    const float inv_span = (n > 1 && span > 0.0f) ? static_cast<float>(n - 1) / span : 0.0f;
    if (j < n) {
        xj = x[j];
        Nj = N[j];
        S = Ssel ? Ssel[j] : selection<F>(xj, S0, v_ref, alpha, v_min);
        on = (S != 0.0) && (Nj > kBreakageNMin);
        if (on) {
            for (int q = l; q < nq; q += nqp) {
                const double v = xj * t_q[q];
                const int lo = lo_tab ? lo_tab[static_cast<size_t>(q) * n + j]
                                      : frag_bracket_guess(x, n, v, lx0, inv_span);
                double P;
                if (lo < 0) P = lam[0];
                else if (lo >= n - 1) P = lam[n - 1];
                else {
                    const double xl = x[lo], xh = x[lo + 1];
                    const double eta = (v - xl) / (xh - xl);
                    P = fma(1.0 - eta, lam[lo], eta * lam[lo + 1]);
                }
                acc = fma(bw_q[q], P, acc);
            }
        }
    }
    for (int o = nqp >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (on && l == 0) {
        const double Q = acc - lam[j];
        gN[j] += S * Q;
        const double NQ = Nj * Q;
        p0 = (S / S0) * NQ;
        if constexpr (F == 1) p1 = -(S / v_ref) * NQ;
        if constexpr (F == 2) {
            p1 = -(alpha * S / v_ref) * NQ;
            p2 = S * log(xj / v_ref) * NQ;
        }
    }
    const double s0 = block_sum(p0, sh);
    const double s1 = block_sum(p1, sh);
    const double s2 = block_sum(p2, sh);
    if (threadIdx.x == 0) {
        part[blockIdx.x * 4 + 0] = s0;
        part[blockIdx.x * 4 + 1] = s1;
        part[blockIdx.x * 4 + 2] = s2;
        part[blockIdx.x * 4 + 3] = 0.0;
    }
}

// Partner chunks per row tile: the row tiles cost the same, so with ntile
// tasks on 2 num_sms CTA slots the last wave can run half empty; pick the
// chunk count (<= kVjpMaxChunks, chunks of >= 512 partners) whose waves come
// closest to whole numbers, the smaller count on near ties.
int vjp_chunks(int ntile, int num_sms, int n)
{
    const double slots = 2.0 * num_sms;
    int best = 1;
    double best_eff = 0.0;
    for (int c = 1; c <= kVjpMaxChunks; ++c) {
        if (c > 1 && n / c < 512) break;
        const double w = ntile * c / slots;
        const double eff = w / std::ceil(w);
        if (eff > best_eff + 0.02) { best_eff = eff; best = c; }
    }
    return best;
}

// Aggregation VJP pair sums on geometric grids: lane blocks (default) or the
// row tiles of every grid. PBE_GB300_VJP_PATH=tile selects the tiles.
int vjp_lane_mode()
{
    static const int mode = []() {
        const char* e = std::getenv("PBE_GB300_VJP_PATH");
        return (e && std::strcmp(e, "tile") == 0) ? 0 : 1;
    }();
    return mode;
}

// Whether the lane-block kernels run (they leave grids that are not geometric to the tiles).
bool vjp_lane_on(int n)
{
    const int C = vjp_lane_chunk(n);
    return vjp_lane_mode() && vjp_lane_tasks(n, C) > 0 && vjp_lane_chunks(n, C) <= kVLaneMaxChunks;
}

template <int K>
cudaError_t agg_vjp_k(const AggVjpArgs& a, const VjpWs& ws, int num_sms, cudaStream_t s, int kind, bool defer)
{
    const int n = a.n;
    const int nb = (n + kPrepThreads - 1) / kPrepThreads;
    const int ntile = (n + VW - 1) / VW;
    const int nch = vjp_chunks(ntile, num_sms, n);
    const int ntasks = ntile * nch;
    const int grid = ntasks < 2 * num_sms ? ntasks : 2 * num_sms;
    const size_t smem = sizeof(double) * kVRows * kMainThreads;
    cudaError_t e = cudaFuncSetAttribute(vjp_main_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    const int C = vjp_lane_chunk(n);
    const long long ltasks = vjp_lane_tasks(n, C);
    const int lane_on = vjp_lane_on(n) ? 1 : 0;
    if (kind == kVjpTables) {
        launch_dep(vjp_prep_kernel<kVjpTables>, dim3(nb), kVPrepThreads, 0, s, 1, a.N, a.x, a.lam, n, ws);
        launch_dep(vjp_fin_kernel<kVjpTables>, dim3(1), kVFinThreads, 0, s, 1, a.x, a.lam, n, ws, a.kernel, a.beta0,
                   a.beta_br, a.beta_sh);
        return cudaGetLastError();
    }
    if (kind == kVjpStage) {
        launch_dep(vjp_prep_kernel<kVjpStage>, dim3(nb), kVPrepThreads, 0, s, 1, a.N, a.x, a.lam, n, ws);
        launch_dep(vjp_fin_kernel<kVjpStage>, dim3(1), kVFinThreads, 0, s, 1, a.x, a.lam, n, ws, a.kernel, a.beta0,
                   a.beta_br, a.beta_sh);
    } else {
        launch_dep(vjp_prep_kernel<kVjpFull>, dim3(nb), kVPrepThreads, 0, s, 1, a.N, a.x, a.lam, n, ws);
        launch_dep(vjp_fin_kernel<kVjpFull>, dim3(1), kVFinThreads, 0, s, 1, a.x, a.lam, n, ws, a.kernel, a.beta0,
                   a.beta_br, a.beta_sh);
    }
    const int nrb = (n + kLaneBins - 1) / kLaneBins;
    if (lane_on) {
        const size_t lsmem = sizeof(double) * kLaneWarps * ((C + kLaneWarps - 1) / kLaneWarps + 32);
        const int lgrid = static_cast<int>(ltasks < kVLaneCtas * num_sms ? ltasks : kVLaneCtas * num_sms);
        launch_dep(vjp_lane_kernel<K>, dim3(lgrid), kMainThreads, lsmem, s, 1, a.N, a.x, a.lam, ws, n, C,
                   a.beta0, a.beta_br, a.beta_sh);
    }
    launch_dep(vjp_main_kernel<K>, dim3(grid), kMainThreads, smem, s, 1, a.N, a.x, a.lam, ws, n, ntile, nch,
               lane_on);
    if (lane_on)
        launch_dep(vjp_lane_rows_kernel<K>, dim3(nrb), kVRowsWarps * 32, 0, s, 1, a.N, a.x, a.lam, a.gN, ws,
                   n, C, ntile, nch, a.beta0, a.beta_br, a.beta_sh);
    else
        launch_dep(vjp_rows_kernel<K>, dim3((ntile + 7) / 8), 256, 0, s, 1, a.N, a.x, a.lam, a.gN, ws, n, ntile,
                   nch, a.beta0, a.beta_br, a.beta_sh);
    if (!defer)
        launch_dep(vjp_gfin_kernel, dim3(1), 256, 0, s, 1, ntile, lane_on ? nrb : 0, ws, a.gp, 0,
                   static_cast<double*>(nullptr));
    return cudaGetLastError();
}

template <int F>
cudaError_t brk_vjp_f(const BrkVjpArgs& a, const VjpWs& ws, cudaStream_t s, const double* Ssel,
                      const int* lo_tab, const AggVjpArgs* after)
{
    int nqp = 1;
    while (nqp < a.n_quad && nqp < 32) nqp <<= 1;
    const int nb = static_cast<int>((static_cast<long long>(a.n) * nqp + 255) / 256);
    launch_dep(brk_vjp_kernel<F>, dim3(nb), 256, 0, s, 1, a.N, a.x, a.t_q, a.bw_q, a.lam, a.gN, ws.bpart,
               a.n, a.n_quad, nqp, a.S0, a.v_ref, a.alpha, a.v_min, Ssel, lo_tab);
    const int ntile = (a.n + VW - 1) / VW, nlane = vjp_lane_on(a.n) ? (a.n + kLaneBins - 1) / kLaneBins : 0;
    launch_dep(vjp_gfin_kernel, dim3(1), 256, 0, s, 1, ntile, nlane, ws, after ? after->gp : nullptr, nb, a.gp);
    return cudaGetLastError();
}

} // namespace

namespace {
cudaError_t agg_vjp_dispatch(const AggVjpArgs& a, void* ws_base, int num_sms, cudaStream_t s, int kind,
                             bool defer = false)
{
    VjpWs ws;
    vjp_ws_layout(a.n, static_cast<char*>(ws_base), &ws);
    switch (a.kernel) {
    case 0: return agg_vjp_k<0>(a, ws, num_sms, s, kind, defer);
    case 1: return agg_vjp_k<1>(a, ws, num_sms, s, kind, defer);
    case 2: return agg_vjp_k<2>(a, ws, num_sms, s, kind, defer);
    case 3: return agg_vjp_k<3>(a, ws, num_sms, s, kind, defer);
    case 4: return agg_vjp_k<4>(a, ws, num_sms, s, kind, defer);
    case 5: return agg_vjp_k<5>(a, ws, num_sms, s, kind, defer);
    default: return cudaErrorInvalidValue;
    }
}
} // namespace

cudaError_t agg_vjp_launch(const AggVjpArgs& a, void* ws_base, int num_sms, cudaStream_t s)
{
    return agg_vjp_dispatch(a, ws_base, num_sms, s, kVjpFull);
}
cudaError_t agg_vjp_tables_launch(const AggVjpArgs& a, void* ws_base, int num_sms, cudaStream_t s)
{
    return agg_vjp_dispatch(a, ws_base, num_sms, s, kVjpTables);
}
cudaError_t agg_vjp_stage_launch(const AggVjpArgs& a, void* ws_base, int num_sms, cudaStream_t s, bool defer)
{
    return agg_vjp_dispatch(a, ws_base, num_sms, s, kVjpStage, defer);
}

cudaError_t brk_vjp_launch(const BrkVjpArgs& a, void* ws_base, cudaStream_t s, const double* Ssel,
                           const int* lo_tab, const AggVjpArgs* after)
{
    VjpWs ws;
    vjp_ws_layout(a.n, static_cast<char*>(ws_base), &ws);
    switch (a.selection) {
    case 0: return brk_vjp_f<0>(a, ws, s, Ssel, lo_tab, after);
    case 1: return brk_vjp_f<1>(a, ws, s, Ssel, lo_tab, after);
    case 2: return brk_vjp_f<2>(a, ws, s, Ssel, lo_tab, after);
    case 3: return brk_vjp_f<3>(a, ws, s, Ssel, lo_tab, after);
    default: return cudaErrorInvalidValue;
    }
}

} // namespace pbe_gb300
