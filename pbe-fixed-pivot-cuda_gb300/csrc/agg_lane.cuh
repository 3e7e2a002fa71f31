// =============================================================================
// agg_lane.cuh -- the tasks of the single-instance aggregation kernel: one output
// slot per lane, the pairs split over the CTA's warps.
//
// Slot s collects the pairs (j <= k) whose bracket is lo = s, R_s = sum rate,
// TH_s = sum rate (fl(x_j + x_k) - x_s) 2^St_s, St_s = -exponent of x_s
// (reference src/aggregation_kernels.cuh:145-239, regrouped).
//
// Geometric grids: lo(j, j + d) = j + Ld[d], so slot s meets lag d in the pair
// j = s - Ld[d], k = s - e(d) with e(d) = Ld[d] - d >= 0. e is the same for
// every slot, and it stays constant over runs of consecutive lags (Ld grows by
// one per lag once the pivot ratio makes x_0 + x_d fall in the bin above x_d;
// e = 0, the lags whose pairs land on their larger member, is one long run).
// Within a run, k is fixed per slot, so for every kernel but Sum
//   rate = F_k q(d, j),   F = N (x N for Product), q = B_d N_j + S_d x_j N_j,
// and a lane sums q and q th over the run and multiplies by F_k once:
// 3 FP64 instructions per pair for one-term kernels, 4 for Brownian + shear.
// Sum keeps its per-pair rate. Other grids: a monotone walk (agg_slot.cuh).
//
// From lag D0 on e = 0: every pair lands on its larger member's own slot. There
// the sums over j separate. beta is a sum of products of powers of x_j and x_k,
// and fl(x_j + x_k) - x_k is x_j up to the sum's rounding, so
//   R_s  = N_s sum_j beta(x_j, x_s) N_j      = N_s death_factor(x_s; P),
//   TH_s = N_s sum_j beta(x_j, x_s) x_j N_j  = N_s death_factor(x_s; T)
// with the prefix moments P_q, T_q of N and x N over the bins j <= s - D0 (the
// prep's scan): O(n) work instead of half of all pairs at n = 16384 and q = 512
// bins per octave, and nearly all of them on coarse grids. The prefix sums add
// terms of one kind without cancellation. Dropping the rounding of
// fl(x_j + x_k) moves w by at most u = 2^-53 x_{s+1}/dx_s, so bin s + 1 by
// u R_s; that bin's own death term is at least N_{s+1}/N_s times R_s, and where
// u N_s > kMomGuard N_{s+1} (a population that ends or falls steeply within one
// bin, where a tiny w's rounding would show) the slot keeps its exact pair sum,
// a task of its own (exact_slot_task).
//
// Lags below D0 on fine grids (win_grid; gather mode; N without negative entries, and
// coefficients of one sign):
// the runs from lag Dm on are long enough to separate too. In run e, lags [d1, d2),
// slot s has k = s - e and the window j in [k - d2 + 1, k - d1], so
//   R += N_k sum_q c_q(x_k) M_q,  TH += N_k (sum_q c_q M_{q+3} + (x_k - x_s) sum_q c_q M_q),
// M_m = sum over the window of x_j^(m/3) N_j, from two table values (and whole
// blocks of 64 between them): windows of any length and place without a
// subtraction, so sums of one sign keep their relative precision. At n = 16384 and 512
// sections an octave 1330 lags stay pairs and 112 runs cover the other 3549. The rounding of
// fl(x_j + x_k), left out as above, moves bins s and s + 1 by at most u R_win; the
// finishing warp compares that with what these bins are known to receive and lose
// (kMomGuard), and slots beyond it sum those lags pair by pair.
//
// On other grids the same holds for the rows j < J0(s), the first j with
// fl(x_j + x_s) >= x_{s+1}.
//
// Work split: blocks of 31 output bins aligned to the top of the grid (slot_blocks);
// a task is one block and one of `parts` equal shares of the lags below D0
// (of each slot's rows on other grids); the CTA's eight warps take equal
// contiguous shares of the task's lags (each warp sees its runs in order) and
// their sums are added in warp order. With several parts each task stores its
// 5 x 32 sums; the block's last task (ticket) adds them in order and writes the
// bins -- deterministic, nobody waits. Beside its pairs a task is a chain of
// latencies of a microsecond each (n = 3840: 24 of 41 us once, 19 of 37 now), so
// the prefix part and the death term come from a warp of share 0 while the others
// sum pairs, and the slot below a block's first bin is summed twice instead of
// handed over.
//
// The j-side operands are read through L1: a share's window (32 + its lags entries
// of N, x N and x) staged in shared memory by bulk copies measured the same with
// these shorter shares (n = 3840: 37.5 and 37.5 us, n = 16384: 291.5 and 291.5).
// =============================================================================
#pragma once

#include "agg_slot.cuh"

namespace pbe_gb300 {

constexpr int kLaneWarps = kMainThreads / 32;       // warps sharing a task's lags
// Shares of a block's pairs (`lags`: pairs of a slot). Long shares: enough tasks
// to give every CTA four, so that the last ones end together. A task costs a few
// microseconds beside its pairs (fetch, sums, ticket), so where that would leave a share
// less than 192 pairs a slot, as many shares as fit the CTAs in one round (608 CTAs, the
// whole call: n = 3840 8 shares in two rounds 70 us, 4 in one 65; n = 8191 98 and 88). At
// least 32 pairs a share (4 per warp).
__host__ __device__ constexpr int lane_parts(int lags, int nblk, int ctas)
{
    int p = (4 * ctas + nblk - 1) / nblk;
    if (p > kLaneMaxParts || lags < 192 * p) p = ctas / nblk;
    const int most = (lags + 31) / 32;
    if (p > most) p = most;
    if (p > kLaneMaxParts) p = kLaneMaxParts;
    return p < 1 ? 1 : p;
}

// Shared memory of a CTA.
struct LaneSmem {
    double red[kLaneWarps][4][32];   // per-warp R, TH of the pairs and of the windows
    double D[32];                    // the bins' death terms
    double sum[2 * kLaneWarps];      // CTA-wide sums
    unsigned mask;
    int task;
};

// The shares of the blocks and what they sum.
struct LaneArgs {
    double* part;        // [lane_partial_doubles(n)]
    int* ticket;         // [slot_blocks(n)] tasks of the block done (reset by the prep)
    int parts;           // tasks per block
    int Dm;              // lags summed pair by pair (geometric grids)
    int eh, el;          // runs eh .. el (descending) summed by windows; eh < el: none
    int flip;            // rates_flip
};

// The call as its tasks see it: the grid with the lag tables, the one pass
// (N on both sides), the moments of N.
struct LaneView {
    SlotGrid g;
    SlotPass p;
    double M[kMomN];
};


// Prefix moments up to bin i of the prep's scan: P_q = sum m_q, T_q = sum m_q x at
// the binary exponent of x_i.
template <int K>
__device__ __forceinline__ void prefix_moments(const AggWs& ws, const double* __restrict__ x, int n,
                                               int i, double* P, double* T)
{
    const int nb = agg_prep_blocks(n), b = i / kPrepThreads;
    const int dE = b > 0 ? exponent_of(__ldg(x + b * kPrepThreads - 1)) - exponent_of(__ldg(x + i)) : 0;
#pragma unroll
    for (int q = 0; q < kMomN; ++q) {
        P[q] = __ldg(ws.mloc + static_cast<size_t>(q) * n + i) + __ldg(ws.moff + q * nb + b);
        T[q] = __ldg(ws.mloc + static_cast<size_t>(kMomN + q) * n + i)
             + scale_down(__ldg(ws.moff + (kMomN + q) * nb + b), dE);
    }
}

// Slots of block t (one per lane) whose prefix part is summed pair by pair.
__device__ __forceinline__ unsigned exact_mask(const LaneView& v, int t)
{
    const int n = v.g.n, s = n - kSlotBins * (t + 1) - 1 + (threadIdx.x & 31);
    const bool e = s >= 0 && s <= n - 2 && slot_cut(v.g, s) > 0 &&
                   mom_exact_slot(__ldg(v.p.Nk + s), __ldg(v.p.Nk + s + 1), __ldg(v.g.x + s + 1),
                                  v.g.inv_dx[s]);
    return __ballot_sync(0xffffffffu, e);
}

// The sums of a lane: its slot's pairs and prefix part, its windows, its bin's
// death term (less what is clipped from the prefix part of slot n - 1).
struct SlotSums {
    double R, TH, Rw, Tw, D;
};

// One warp, after its contribution to block t is stored: the block's ticket.
// True for the last of its `parts` share tasks and one task per exact slot;
// that one gets the block's sums, added in a fixed order.
__device__ __forceinline__ bool block_ticket(const AggWs& ws, const LaneArgs& la, int n, int t,
                                             unsigned exact, SlotSums& u)
{
    const int lane = threadIdx.x & 31;
    const int want = la.parts + __popc(exact);
    __threadfence();                                   // every lane's stores before the ticket
    __syncwarp();
    int last = 0;
    if (lane == 0) last = (atomicAdd(la.ticket + t, 1) == want - 1);
    if (!__shfl_sync(0xffffffffu, last, 0)) return false;
    __threadfence();
    u = SlotSums{0.0, 0.0, 0.0, 0.0, 0.0};
    const double* bp = la.part + static_cast<size_t>(t) * la.parts * kLanePart + lane;
    for (int q = 0; q < la.parts; ++q, bp += kLanePart) {
        u.R += __ldcg(bp);
        u.TH += __ldcg(bp + 32);
        u.Rw += __ldcg(bp + 64);
        u.Tw += __ldcg(bp + 96);
        if (q == 0) u.D = __ldcg(bp + 128);
    }
    if ((exact >> lane) & 1u) {
        const int s = n - kSlotBins * (t + 1) - 1 + lane;
        u.R += __ldcg(ws.xsum + 2 * s);
        u.TH += __ldcg(ws.xsum + 2 * s + 1);
    }
    return true;
}

// One warp: the prefix part of block t's slots (but the exact ones) and the death
// term of its bins.
template <int K>
__device__ __forceinline__ void lane_base(const LaneView& v, const AggWs& ws, int t, unsigned exact,
                                          double& R, double& TH, double& D)
{
    const int n = v.g.n, lane = threadIdx.x & 31;
    const int s = n - kSlotBins * (t + 1) - 1 + lane;
    R = TH = D = 0.0;
    if (s < 0 || s >= n) return;
    const double as = v.g.a[s], ias = v.g.ia[s], xv = __ldg(v.g.x + s), Ns = __ldg(v.p.Nk + s);
    const int cut = slot_cut(v.g, s);
    if (cut > 0 && !((exact >> lane) & 1u)) {
        double P[kMomN], T[kMomN];
        prefix_moments<K>(ws, v.g.x, n, cut - 1, P, T);
        const double r = Ns * death_factor<K>(xv, as, ias, P, v.g.b0, v.g.bbr, v.g.bsh);
        if (s <= n - 2) {
            // (shifted before N_s comes in: 1e-302 times a shift would leave the normal range)
            const double f = death_factor<K>(xv, as, ias, T, v.g.b0, v.g.bbr, v.g.bsh);
            R = r;
            TH = Ns * scale_down(f, exponent_of(__ldg(v.g.x + cut - 1)) - exponent_of(xv));
        } else {
            D = -r;                                    // clipped: all of it stays in bin n - 1
        }
    }
    D += Ns * death_factor<K>(xv, as, ias, v.M, v.g.b0, v.g.bbr, v.g.bsh);
}

// The runs eh .. el of slot s by windows: Rw += rates, Tw += rates (v - x_s) 2^St_s.
// Every lane of the warp takes part.
template <int K>
__device__ __forceinline__ void lane_windows(const LaneView& v, const AggWs& ws, int s, bool slot, int eh,
                                             int el, double& Rw, double& Tw)
{
    const int n = v.g.n;
    const size_t ns = static_cast<size_t>(n);
    const double xs = slot ? __ldg(v.g.x + s) : 1.0;
    const int E = win_exponent(v.g.x), E20 = E * (1 << 20);
    const int dE = E - exponent_of(xs);              // from the tables' unit to the slot's, at most 0
    for (int e = eh; e >= el; --e) {
        const int d1 = __ldg(ws.rend + e + 1), d2 = __ldg(ws.rend + e);
        const int k = s - e, b = k - d1;
        if (!slot || b < 0) continue;
        const int a = max(0, k - d2 + 1);
        const int A = a >> 6, B = b >> 6;
        const double* pb = ws.wtab + b;                // the part from the middle (or a block's start) to b
        const double* pa = ws.wtab + a;                // the part from a to the middle (or a block's end)
        bool two = true;
        if (A != B) {
            pb += 4 * kWinMom * ns;
            pa += 5 * kWinMom * ns;
        } else if ((a & 63) == 0) {
            pb += 4 * kWinMom * ns;
            two = false;
        } else {                                       // b - a >= 4: they differ in bit 2 or above
            const size_t l = static_cast<size_t>(31 - __clz(a ^ b) - 2) * kWinMom * ns;
            pb += l;
            pa += l;
        }
        double M[kWinMom];
#pragma unroll
        for (int m = 0; m < kWinMom; ++m) {
            M[m] = 0.0;
            if (need_window<K>(m)) M[m] = __ldg(pb + m * ns) + (two ? __ldg(pa + m * ns) : 0.0);
        }
        for (int q = A + 1; q < B; ++q)                // whole blocks of 64 between
#pragma unroll
            for (int m = 0; m < kWinMom; ++m)
                if (need_window<K>(m)) M[m] += __ldg(ws.wtab + (4 * kWinMom + m) * ns + q * 64 + 63);
        double r = 0.0, t = 0.0;
#pragma unroll
        for (int q = 0; q < kMomN; ++q) {
            if (!need_moment<K>(q)) continue;
            const double c = __ldg(ws.wc + q * ns + k);
            r = fma(c, M[q], r);
            t = fma(c, M[q + 3], t);
        }
        // N_k comes last, and t is at the slot's exponent by then: with N_k = 1e-300 in c,
        // or times x, the terms of a population's foot would underflow
        t = fma(scale_pow2(__ldg(v.g.x + k) - xs, -E20), r, t);
        const double Nk = __ldg(v.p.Nk + k);
        Rw = fma(Nk, r, Rw);
        Tw = fma(Nk, scale_down(t, dE), Tw);
    }
}

// The lags [Dm, D0) of slot s pair by pair, by the CTA (threads over the lags),
// summed in a fixed order; red: 2 kLaneWarps doubles of shared memory. Valid in
// every thread; CTA synchronised.
template <int K>
__device__ __forceinline__ void exact_runs(const LaneView& v, int s, int Dm, double* red, double& R,
                                           double& TH)
{
    const double xs = __ldg(v.g.x + s);
    const EwOperandC pc = ew_operand_c(xs, -exponent_of(xs));
    double r = 0.0, t = 0.0;
    for (int d = Dm + static_cast<int>(threadIdx.x); d < min(v.g.D0, v.g.n); d += kMainThreads) {
        const int L = v.g.Ld[d];
        const int j = s - L, k = j + d;
        if (j < 0) break;                              // Ld is nondecreasing
        const double rate = rate_geo<K>(v.g.Bd[d], v.g.Sd[d], __ldg(v.p.Nj + j),
                                        NeedH<K>::j ? v.p.Hj[j] : 0.0, __ldg(v.p.Nk + k),
                                        NeedH<K>::k ? v.p.Hk[k] : 0.0);
        r += rate;
        t = fma(rate, sum_minus_scaled_pre(ew_operand_a(__ldg(v.g.x + k)), __ldg(v.g.x + j), pc), t);
    }
    r = warp_sum(r);
    t = warp_sum(t);
    if ((threadIdx.x & 31) == 0) { red[2 * (threadIdx.x >> 5)] = r; red[2 * (threadIdx.x >> 5) + 1] = t; }
    __syncthreads();
    R = TH = 0.0;
    for (int q = 0; q < kLaneWarps; ++q) { R += red[2 * q]; TH += red[2 * q + 1]; }
    __syncthreads();
}

// The bins of block t from its lanes' sums in warp 0, by the CTA; `finish` and u
// are warp 0's. Scatter mode calls it for every share's own sums.
template <int K, bool SCATTER>
__device__ void lane_finish(const LaneView& v, const AggWs& ws, const LaneArgs& la, double* rhs, int t,
                            int nclip, bool finish, SlotSums u, LaneSmem& sm)
{
    const int n = v.g.n, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int s = n - kSlotBins * (t + 1) - 1 + lane;  // this lane's slot and bin
    const bool slot = s >= 0 && s <= n - 2;
    double sd = 0.0, own = 0.0, up = 0.0;              // the slot's own part of bin s, its w-part of bin s + 1
    if (w == 0 && finish && slot) {
        const int St = -exponent_of(__ldg(v.g.x + s));
        sd = scalbn(v.g.inv_dx[s], -St);
        own = fma(-(u.TH + u.Tw), sd, u.R + u.Rw);
        up = (u.TH + u.Tw) * sd;
    }
    if (!SCATTER && la.eh >= la.el) {
        // windows: slots where the rounding they leave out may show in bin s or s + 1
        if (w == 0) {
            bool ex = false;
            const double below = __shfl_up_sync(0xffffffffu, up, 1);
            const double dn = __shfl_down_sync(0xffffffffu, u.D, 1);
            const double on = __shfl_down_sync(0xffffffffu, own, 1);
            if (finish && slot && u.Rw != 0.0) {
                const double xu = __ldg(v.g.x + s + 1);
                const int fl = la.flip;
                const double err = (xu * v.g.inv_dx[s]) * flip_sign(u.Rw, fl);   // 2^53 times the error
                constexpr double kGuard = kMomGuard * 9007199254740992.0;
                double dup = fmax(flip_sign(dn, fl), 0.0);
                if (lane == 31)
                    dup = flip_sign(__ldg(v.p.Nk + s + 1) * death_factor<K>(xu, v.g.a[s + 1], v.g.ia[s + 1],
                                                                            v.M, v.g.b0, v.g.bbr, v.g.bsh), fl);
                const double here = fmax(flip_sign(own, fl), 0.0) + flip_sign((lane > 0 ? below : 0.0) + u.D, fl);
                const double next = flip_sign(up, fl) + (lane < 31 ? fmax(flip_sign(on, fl), 0.0) : 0.0) + dup;
                // (slot I - 1 matters to bin I alone here)
                ex = !((lane == 0 || err <= kGuard * here) && err <= kGuard * next);
            }
            const unsigned m = __ballot_sync(0xffffffffu, ex);
            if (lane == 0) sm.mask = m;
        }
        __syncthreads();
        for (unsigned m = sm.mask; m != 0u; m &= m - 1u) {
            const int le = __ffs(m) - 1;
            double r, th;
            exact_runs<K>(v, n - kSlotBins * (t + 1) - 1 + le, la.Dm, sm.sum, r, th);
            if (w == 0 && lane == le) {
                own = fma(-(u.TH + th), sd, u.R + r);
                up = (u.TH + th) * sd;
            }
        }
    }
    if (w != 0 || !finish) return;
    const double in = __shfl_up_sync(0xffffffffu, up, 1);
    if constexpr (SCATTER) {
        // (slot I - 1: its w-part enters bin I as `in`; slot I + 30's leaves by lane 0 above)
        const double val = (own + in) - u.D;
        if (lane >= 1 && s >= 0 && val != 0.0) atomicAdd(rhs + s, val);
    } else if (lane >= 1 && s >= 0) {
        rhs[s] = rhs[s] + ((own + in) - u.D);
        if (s == n - 1) {
            __threadfence();
            if (atomicAdd(ws.counter + 3, 1) == nclip) {
                __threadfence();
                double sc = 0.0;
                for (int q = 0; q < nclip; ++q) sc += __ldcg(ws.clip_part + q);
                rhs[n - 1] = __ldcg(rhs + (n - 1)) + sc;
            }
        }
    }
}

// The prefix part of one exact slot, pair by pair: the CTA over j, summed in
// a fixed order. Such slots cluster at the foot of a population, so each is a
// task of its own (summed by its block's last task, 90 of them on a run of 3840
// bins made the whole call 1.5 x slower). red: 2 kLaneWarps doubles.
template <int K, bool SCATTER>
__device__ void exact_slot_task(const LaneView& v, const AggWs& ws, const LaneArgs& la,
                                double* rhs, int s, int nclip, LaneSmem& sm)
{
    const int n = v.g.n, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int cut = slot_cut(v.g, s);
    if (cut <= 0 || s > n - 2) return;                 // no such pairs (the whole CTA)
    double r, th;
    slot_exact_part<K, 1>(v.g, &v.p, s, tid, kMainThreads, r, th);
    r = warp_sum(r);
    th = warp_sum(th);
    if (lane == 0) { sm.sum[2 * w] = r; sm.sum[2 * w + 1] = th; }
    __syncthreads();
    r = 0.0;
    th = 0.0;
    for (int q = 0; q < kLaneWarps; ++q) { r += sm.sum[2 * q]; th += sm.sum[2 * q + 1]; }
    __syncthreads();
    if constexpr (SCATTER) {
        if (tid == 0) {
            const double co = th * scalbn(v.g.inv_dx[s], exponent_of(__ldg(v.g.x + s)));
            atomicAdd(rhs + s, r - co);
            if (co != 0.0) atomicAdd(rhs + s + 1, co);
        }
    } else {
        if (tid == 0) {
            ws.xsum[2 * s] = r;
            ws.xsum[2 * s + 1] = th;
        }
        // the slot's own block, and the one above when the slot is the one below its bins
        const int up = n - 1 - s, t1 = up / kSlotBins;
        for (int t = t1; t >= 0 && (t == t1 || (t == t1 - 1 && up % kSlotBins == 0)); --t) {
            SlotSums u{0.0, 0.0, 0.0, 0.0, 0.0};
            bool finish = false;
            if (w == 0) finish = block_ticket(ws, la, n, t, exact_mask(v, t), u);
            lane_finish<K, false>(v, ws, la, rhs, t, nclip, finish, u, sm);
            __syncthreads();
        }
    }
}

// One lane task: block t, share c of its direct pairs. All kMainThreads threads
// of the CTA take part; returns with the CTA synchronised. Gather mode stores /
// finishes the block's bins; scatter mode flushes this task's share with atomics.
template <int K, bool SCATTER>
__device__ void lane_task(const LaneView& v, const AggWs& ws, const LaneArgs& la, double* rhs,
                          int t, int c, int nclip, LaneSmem& sm)
{
    const int n = v.g.n;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int I = n - kSlotBins * (t + 1);
    const int smax = min(I + kSlotBins - 1, n - 2);
    const int s = I - 1 + lane;
    const bool slot = s >= 0 && s <= smax;
    double R = 0.0, TH = 0.0, Rw = 0.0, Tw = 0.0, D = 0.0;
    const unsigned em = w <= 1 ? exact_mask(v, t) : 0u;
    if (w == 1 && c == 0) lane_base<K>(v, ws, t, em, R, TH, D);
    double r = 0.0, th = 0.0;
    if (v.g.geo) {
        if (!SCATTER && la.eh >= la.el) {
            // this warp's share of the runs summed by windows
            const int ne = la.eh - la.el + 1, sh = la.parts * kLaneWarps, q = c * kLaneWarps + w;
            lane_windows<K>(v, ws, s, slot, la.eh - ne * q / sh, la.eh - ne * (q + 1) / sh + 1, Rw, Tw);
        }
        // and its contiguous share of the task's lags [dA, dB), dB cut where Ld passes
        // the block's top slot (Ld is nondecreasing; clipped lags hold kLagClipAll)
        const int C = (la.Dm + la.parts - 1) / la.parts;
        const int dA = min(c * C, la.Dm);
        const int dB = min(min(dA + C, la.Dm), smax + 1);
        const int per = (dB - dA + kLaneWarps - 1) / kLaneWarps;
        const int dw0 = dA + w * per;
        const double xs = slot ? __ldg(v.g.x + s) : 1.0;
        slot_pairs_geo<K, 1>(v.g, &v.p, s, slot, smax, dw0, min(dB, dw0 + per),
                             ew_operand_c(xs, -exponent_of(xs)), r, th);
    } else {
        slot_pairs_any<K, 1>(v.g, &v.p, s, slot, s + 1, c * kLaneWarps + w, la.parts * kLaneWarps, r, th);
    }
    sm.red[w][0][lane] = R + r;
    sm.red[w][1][lane] = TH + th;
    sm.red[w][2][lane] = Rw;
    sm.red[w][3][lane] = Tw;
    if (w == 1) sm.D[lane] = D;
    __syncthreads();

    SlotSums u{0.0, 0.0, 0.0, 0.0, 0.0};
    bool finish = false;
    if (w == 0) {
#pragma unroll
        for (int q = 0; q < kLaneWarps; ++q) {
            u.R += sm.red[q][0][lane];
            u.TH += sm.red[q][1][lane];
            u.Rw += sm.red[q][2][lane];
            u.Tw += sm.red[q][3][lane];
        }
        u.D = sm.D[lane];
        finish = true;
        if (!SCATTER && (la.parts > 1 || em != 0u)) {
            double* bp = la.part + (static_cast<size_t>(t) * la.parts + c) * kLanePart + lane;
            bp[0] = u.R;
            bp[32] = u.TH;
            bp[64] = u.Rw;
            bp[96] = u.Tw;
            if (c == 0) bp[128] = u.D;
            finish = block_ticket(ws, la, n, t, em, u);
        }
    }
    lane_finish<K, SCATTER>(v, ws, la, rhs, t, nclip, finish, u, sm);
    __syncthreads();
}

} // namespace pbe_gb300
