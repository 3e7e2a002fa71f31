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
// Lags below D0 on fine grids (win_grid; gather mode; N without negative entries):
// the runs from lag Dm on are long enough to separate too. In run e, lags [d1, d2),
// slot s has k = s - e and the window j in [k - d2 + 1, k - d1], so
//   R += sum_q c_q(x_k) N_k M_q,  TH += sum_q c_q N_k M_{q+3} + (x_k - x_s) R_run,
// M_m = sum over the window of x_j^(m/3) N_j, from two table values (and whole
// blocks of 64 between them): windows of any length and place without a
// subtraction, so sums of one sign keep their relative precision. At 512 sections
// an octave 1324 lags stay pairs and 137 runs cover the other 3560. The rounding of
// fl(x_j + x_k), left out as above, moves bins s and s + 1 by at most u R_win; the
// finishing warp compares that with what these bins are known to receive and lose
// (kMomGuard), and slots beyond it sum those lags pair by pair.
//
// On other grids the same holds for the rows j < J0(s), the first j with
// fl(x_j + x_s) >= x_{s+1}.
//
// Work split: blocks of 32 output bins aligned to the top of the grid (block
// t owns bins [n - 32 (t + 1), n - 32 t), so bin n - 1 is never a block's first
// bin); a task is one block and one of `parts` equal shares of the lags below D0
// (of each slot's rows on other grids); the CTA's eight warps take equal
// contiguous shares of the task's lags (each warp sees its runs in order) and
// their sums are added in warp order. With several parts each task stores its
// 4 x 32 sums; the block's last task (ticket) adds them in order and writes the
// bins -- deterministic, nobody waits.
//
// Operand staging (geometric grids): the j-side operands of a task (N_j,
// x_j N_j, x_j for j in one contiguous window of at most kLaneWinMax entries)
// are copied into shared memory with bulk TMA copies (cp.async.bulk, mbarrier
// completion).
// =============================================================================
#pragma once

#include <cstdint>

#include "agg_slot.cuh"

namespace pbe_gb300 {

constexpr int kLaneWarps = kMainThreads / 32;       // warps sharing a task's lags
constexpr int kLaneWinMax = 1792;                   // staged window, entries per array (even)
// Bounded waits on the staging barrier: iterations of mbarrier.try_wait.
constexpr long long kLaneWaitLimit = 1LL << 26;

// Shares of a block's pairs (`lags`: pairs of a slot). Long shares: enough tasks
// to give every CTA four, so that the last ones end together. A task costs a few
// microseconds beside its pairs (fetch, staging, sums, ticket), so where that would
// leave a share less than 192 pairs a slot, as many shares as fit the CTAs in one
// round (n = 3840, 456 CTAs: 8 shares in two rounds 57 us, 3 shares in one 42). At
// least 32 pairs a share (4 per warp). A share longer than the staged window reads
// its operands from the arrays.
__host__ __device__ constexpr int lane_parts(int lags, int nblk, int ctas)
{
    int p = (4 * ctas + nblk - 1) / nblk;
    if (p > kLaneMaxParts || lags < 192 * p) p = ctas / nblk;
    const int most = (lags + 31) / 32;
    if (p > most) p = most;
    if (p > kLaneMaxParts) p = kLaneMaxParts;
    return p < 1 ? 1 : p;
}

// ---- bulk TMA copy + mbarrier helpers (shared::cta addresses) -----------------
__device__ __forceinline__ unsigned smem_addr(const void* p)
{
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_addr(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                 :: "r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// global -> shared bulk copy; dst, src 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, uint64_t* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(smem_addr(bar)) : "memory");
}
// Waits for the barrier's phase `parity` to complete; false after kLaneWaitLimit tries.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity)
{
    const unsigned a = smem_addr(bar);
    for (long long it = 0; it < kLaneWaitLimit; ++it) {
        unsigned done;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done) : "r"(a), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}
__device__ __forceinline__ void fence_proxy_async_smem()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Shared memory of a lane task (carved from the kernel's dynamic buffer).
struct LaneSmem {
    double* red;     // [kLaneWarps][4][32] per-warp R, TH of the pairs and of the windows
    double* wN;      // [kLaneWinMax] staged N_j   (K needs N on the j side)
    double* wH;      // [kLaneWinMax] staged x_j N_j
    double* wX;      // [kLaneWinMax] staged x_j
};

// Staged copies of N and x (scratch, 256-byte aligned, at least n + 2 entries)
// and the chunk partials / tickets of the lane path.
struct LaneArgs {
    const double* Ncp;   // N copy
    const double* xcp;   // x copy
    double* part;        // [lane_partial_doubles(n)]
    int* ticket;         // [lane_blocks(n)] tasks of the block done (reset by the prep)
    int* err;            // set to 1 when a staging wait gave up
    int parts;           // tasks per block
    int Dm;              // lags summed pair by pair (geometric grids)
    int eh, el;          // runs eh .. el (descending) summed by windows; eh < el: none
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
    const int s = v.g.n - kLaneBins * (t + 1) + (threadIdx.x & 31);
    const bool e = s >= 0 && s <= lane_block_smax(v.g.n, t) && slot_cut(v.g, s) > 0 &&
                   mom_exact_slot(__ldg(v.p.Nk + s), __ldg(v.p.Nk + s + 1), __ldg(v.g.x + s + 1),
                                  __ldg(v.g.inv_dx + s));
    return __ballot_sync(0xffffffffu, e);
}

// The sums of a slot: pairs (and prefix part), windows.
struct SlotSums {
    double R, TH, Rw, Tw;
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
    u = SlotSums{0.0, 0.0, 0.0, 0.0};
    const double* bp = la.part + static_cast<size_t>(t) * la.parts * 128 + lane;
    for (int q = 0; q < la.parts; ++q, bp += 128) {
        u.R += __ldcg(bp);
        u.TH += __ldcg(bp + 32);
        u.Rw += __ldcg(bp + 64);
        u.Tw += __ldcg(bp + 96);
    }
    if ((exact >> lane) & 1u) {
        const int s = n - kLaneBins * (t + 1) + lane;
        u.R += __ldcg(ws.xsum + 2 * s);
        u.TH += __ldcg(ws.xsum + 2 * s + 1);
    }
    return true;
}

// The runs eh .. el of slot s by windows: Rw += rates, Tw += rates (v - x_s), not
// scaled. Every lane of the warp takes part.
template <int K>
__device__ __forceinline__ void lane_windows(const LaneView& v, const AggWs& ws, int s, bool slot, int eh,
                                             int el, double& Rw, double& Tw)
{
    const int n = v.g.n;
    const size_t ns = static_cast<size_t>(n);
    const double xs = slot ? __ldg(v.g.x + s) : 0.0;
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
        double r = 0.0;
#pragma unroll
        for (int q = 0; q < kMomN; ++q) {
            if (!need_moment<K>(q)) continue;
            const double c = __ldg(ws.wc + q * ns + k);
            r = fma(c, M[q], r);
            Tw = fma(c, M[q + 3], Tw);
        }
        Rw += r;
        Tw = fma(__ldg(v.g.x + k) - xs, r, Tw);
    }
}

// The lags [Dm, D0) of slot s pair by pair, by one warp (lanes over the lags,
// fixed butterfly). Valid in every lane.
template <int K>
__device__ __forceinline__ void exact_runs(const LaneView& v, int s, int Dm, double& R, double& TH)
{
    const int lane = threadIdx.x & 31;
    const double xs = __ldg(v.g.x + s);
    const EwOperandC pc = ew_operand_c(xs, -exponent_of(xs));
    double r = 0.0, t = 0.0;
    for (int d = Dm + lane; d < min(v.g.D0, v.g.n); d += 32) {
        const int L = __ldg(v.g.Ld + d);
        const int j = s - L, k = j + d;
        if (j < 0) break;                              // Ld is nondecreasing
        const double rate = rate_geo<K>(__ldg(v.g.Bd + d), __ldg(v.g.Sd + d), __ldg(v.p.Nj + j),
                                        NeedH<K>::j ? __ldg(v.p.Hj + j) : 0.0, __ldg(v.p.Nk + k),
                                        NeedH<K>::k ? __ldg(v.p.Hk + k) : 0.0);
        r += rate;
        t = fma(rate, sum_minus_scaled_pre(ew_operand_a(__ldg(v.g.x + k)), __ldg(v.g.x + j), pc), t);
    }
    R = warp_sum(r);
    TH = warp_sum(t);
}

// The bins of block t from its slots' sums (a slot per lane of warp 0), by the
// CTA; `finish` and u are warp 0's. With `first` the prefix part (not of the exact
// slots) and the death term are added; scatter mode calls it for every share's own
// sums. s_ex: shared memory, [2][32] and a mask behind it.
template <int K, bool SCATTER>
__device__ void lane_finish(const LaneView& v, const AggWs& ws, const LaneArgs& la, double* rhs, int t,
                            int nclip, unsigned exact, bool finish, bool first, bool poisoned,
                            SlotSums u, double (*s_ex)[32], unsigned* s_mask)
{
    const int n = v.g.n, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int I = n - kLaneBins * (t + 1);
    const int smax = lane_block_smax(n, t);
    const int s = I + lane, i = s;
    const bool slot = s >= 0 && s <= smax;
    double clip0 = 0.0;                                // the prefix part of the clipped slot n - 1
    double death = 0.0, sd = 0.0, own = 0.0, up = 0.0;
    int St = 0;
    if (w == 0 && finish) {
        const double xs = slot ? __ldg(v.g.x + s) : 0.0;
        St = slot ? -exponent_of(xs) : 0;
        if (first && s >= 0 && s <= n - 1) {
            const double as = __ldg(v.g.a + s), ias = __ldg(v.g.ia + s), xv = __ldg(v.g.x + s);
            const double Ns = __ldg(v.p.Nk + s);
            death = Ns * death_factor<K>(xv, as, ias, v.M, v.g.b0, v.g.bbr, v.g.bsh);
            const int cut = slot_cut(v.g, s);
            if (cut > 0 && !((exact >> lane) & 1u)) {
                double P[kMomN], T[kMomN];
                prefix_moments<K>(ws, v.g.x, n, cut - 1, P, T);
                const double r = Ns * death_factor<K>(xv, as, ias, P, v.g.b0, v.g.bbr, v.g.bsh);
                const double th = Ns * death_factor<K>(xv, as, ias, T, v.g.b0, v.g.bbr, v.g.bsh);
                if (slot) {
                    u.R += r;
                    u.TH += scale_down(th, exponent_of(__ldg(v.g.x + cut - 1)) + St);
                } else {
                    clip0 = r;
                }
            }
        }
        u.Tw = scalbn(u.Tw, St);
        // own part of bin i (slot i) and the w-part of slot i, owed to bin i + 1
        if (slot) {
            const double idx = __ldg(v.g.inv_dx + i);
            sd = scalbn(idx, -St);
            own = fma(-(u.TH + u.Tw), sd, u.R + u.Rw);
            up = (u.TH + u.Tw) * sd;
        }
    }
    if (!SCATTER && la.eh >= la.el) {
        // windows: slots where the rounding they leave out may show in bin s or s + 1
        if (w == 0) {
            bool ex = false;
            const double below = __shfl_up_sync(0xffffffffu, up, 1);
            const double dn = __shfl_down_sync(0xffffffffu, death, 1);
            const double on = __shfl_down_sync(0xffffffffu, own, 1);
            if (finish && slot && u.Rw != 0.0) {
                const double xu = __ldg(v.g.x + s + 1);
                const double err = (1.1102230246251565e-16 * (xu * __ldg(v.g.inv_dx + s))) * u.Rw;
                double dup = dn;
                if (lane == 31)
                    dup = __ldg(v.p.Nk + s + 1) * death_factor<K>(xu, __ldg(v.g.a + s + 1), __ldg(v.g.ia + s + 1),
                                                                  v.M, v.g.b0, v.g.bbr, v.g.bsh);
                const double here = fmax(own, 0.0) + (lane > 0 ? below : 0.0) + death;
                const double next = up + (lane < 31 ? fmax(on, 0.0) : 0.0) + dup;
                ex = !(err <= kMomGuard * here && err <= kMomGuard * next);
            }
            const unsigned m = __ballot_sync(0xffffffffu, ex);
            if (lane == 0) *s_mask = m;
        }
        __syncthreads();
        const unsigned mask = *s_mask;
        if (mask != 0u) {
            int turn = 0;
            for (unsigned m = mask; m != 0u; m &= m - 1u, turn = (turn + 1) & (kLaneWarps - 1)) {
                if (turn != w) continue;
                const int le = __ffs(m) - 1;
                double r, th;
                exact_runs<K>(v, I + le, la.Dm, r, th);
                if (lane == 0) { s_ex[0][le] = r; s_ex[1][le] = th; }
            }
            __syncthreads();
            if (w == 0 && ((mask >> lane) & 1u)) {
                own = fma(-(u.TH + s_ex[1][lane]), sd, u.R + s_ex[0][lane]);
                up = (u.TH + s_ex[1][lane]) * sd;
            }
        }
    }
    if (w != 0 || !finish) return;
    const double in = __shfl_up_sync(0xffffffffu, up, 1);
    if (i >= 0) {
        double val = own;
        if (lane >= 1) val += in;
        val += clip0;
        val -= death;
        if constexpr (SCATTER) {
            if (val != 0.0) atomicAdd(rhs + i, val);
        } else {
            if (poisoned) val = __longlong_as_double(0x7ff8000000000000LL);
            if (lane == 0 && I >= 1) {
                ws.tfirst[t] = val;
                __threadfence();
                if (atomicAdd(ws.tticket + t, 1) == 1) {
                    __threadfence();
                    rhs[I] = __ldcg(rhs + I) + (__ldcg(ws.tfirst + t) + __ldcg(ws.tcarry + t));
                }
            } else {
                rhs[i] = rhs[i] + val;
                if (i == n - 1) {
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
    }
    if constexpr (SCATTER) {
        if (lane == 31 && slot && up != 0.0) atomicAdd(rhs + i + 1, up);
    } else if (lane == 31 && t >= 1) {
        // carry into bin I + 32, the first bin of block t - 1
        ws.tcarry[t - 1] = up;
        __threadfence();
        if (atomicAdd(ws.tticket + (t - 1), 1) == 1) {
            __threadfence();
            const int J = I + kLaneBins;
            rhs[J] = __ldcg(rhs + J) + (__ldcg(ws.tfirst + t - 1) + __ldcg(ws.tcarry + t - 1));
        }
    }
}

// The prefix part of one exact slot, pair by pair: the CTA over j, summed in
// a fixed order. Such slots cluster at the foot of a population, so each is a
// task of its own (summed by its block's last task, 90 of them on a run of 3840
// bins made the whole call 1.5 x slower). `red`: 2 kLaneWarps doubles.
template <int K, bool SCATTER>
__device__ void exact_slot_task(const LaneView& v, const AggWs& ws, const LaneArgs& la,
                                double* rhs, int s, int nclip, double* red, bool poisoned,
                                double (*s_ex)[32], unsigned* s_mask)
{
    const int n = v.g.n, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int t = (n - 1 - s) / kLaneBins;
    const int cut = slot_cut(v.g, s);
    if (cut <= 0 || s > lane_block_smax(n, t)) return;   // no such pairs (the whole CTA)
    const double xe = __ldg(v.g.x + s);
    const int St = -exponent_of(xe);
    double r, th;
    slot_exact_part<K, 1>(v.g, &v.p, s, tid, kMainThreads, r, th);
    r = warp_sum(r);
    th = warp_sum(th);
    if (lane == 0) { red[2 * w] = r; red[2 * w + 1] = th; }
    __syncthreads();
    SlotSums u{0.0, 0.0, 0.0, 0.0};
    unsigned em = 0u;
    bool finish = false;
    if (w == 0) {
        r = 0.0;
        th = 0.0;
        for (int q = 0; q < kLaneWarps; ++q) { r += red[2 * q]; th += red[2 * q + 1]; }
        if constexpr (SCATTER) {
            if (lane == 0) {
                const double co = th * scalbn(__ldg(v.g.inv_dx + s), -St);
                atomicAdd(rhs + s, r - co);
                if (co != 0.0) atomicAdd(rhs + s + 1, co);
            }
        } else {
            if (lane == 0) {
                ws.xsum[2 * s] = r;
                ws.xsum[2 * s + 1] = th;
            }
            em = exact_mask(v, t);
            finish = block_ticket(ws, la, n, t, em, u);
        }
    }
    if constexpr (!SCATTER)
        lane_finish<K, false>(v, ws, la, rhs, t, nclip, em, finish, true, poisoned, u, s_ex, s_mask);
    __syncthreads();
}

// The lags [dw0, dw1) of a warp's slots on a geometric grid, with the operands of
// the task staged (pN, pH, pX indexed by j).
template <int K>
__device__ __forceinline__ void lane_pairs(const LaneView& v, int s, bool slot, int dw0, int dw1,
                                           const double* pN, const double* pH, const double* pX,
                                           double& R, double& TH)
{
    const double xs = slot ? __ldg(v.g.x + s) : 0.0;
    const EwOperandC pc = ew_operand_c(xs, slot ? -exponent_of(xs) : 0);   // the slot pivot, decoded once
    EwOperandA pa = ew_operand_a(0.0);                // x_k of the current run
    double Q = 0.0, QT = 0.0, F = 0.0, hk = 0.0;
    int e_cur = -1;
    for (int d = dw0; d < dw1; ++d) {
        const int L = __ldg(v.g.Ld + d);
        const int e = L - d;
        if (e != e_cur) {                              // uniform across the warp
            if constexpr (K != 1) {
                R = fma(F, Q, R);
                TH = fma(F, QT, TH);
                Q = 0.0;
                QT = 0.0;
            }
            e_cur = e;
            const int k = s - e;
            const bool kin = slot && k >= 0;
            F = kin ? __ldg((K == 2 ? v.p.Hk : v.p.Nk) + k) : 0.0;
            pa = ew_operand_a(kin ? __ldg(v.g.x + k) : 0.0);
            if constexpr (K == 1) hk = kin ? __ldg(v.p.Hk + k) : 0.0;
        }
        const double B = __ldg(v.g.Bd + d), S = __ldg(v.g.Sd + d);
        const int j = s - L;
        if (slot && j >= 0) {
            const double Nj = pN[j];
            const double hj = NeedH<K>::j ? pH[j] : 0.0;
            const double th = sum_minus_scaled_pre(pa, pX[j], pc);
            if constexpr (K != 1) {
                const double q = q_slot<K>(B, S, Nj, hj);
                Q += q;
                QT = fma(q, th, QT);
            } else {
                const double rate = rate_geo<1>(B, S, Nj, hj, F, hk);
                R += rate;
                TH = fma(rate, th, TH);
            }
        }
    }
    if constexpr (K != 1) {
        R = fma(F, Q, R);
        TH = fma(F, QT, TH);
    }
}

// One lane task: block t, share c of its direct pairs. All kMainThreads threads
// of the CTA take part; returns with the CTA synchronised. `phase` is the staging
// barrier's parity (flipped per staged task). Gather mode stores / finishes
// the block's bins; scatter mode flushes this task's share with atomics.
template <int K, bool SCATTER>
__device__ void lane_task(const LaneView& v, const AggWs& ws, const LaneArgs& la, double* rhs,
                          int t, int c, int nclip, const LaneSmem& sm, uint64_t* bar,
                          unsigned& phase, int* s_flag, double (*s_ex)[32], unsigned* s_mask)
{
    const int n = v.g.n;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int I = n - kLaneBins * (t + 1);
    const int smax = lane_block_smax(n, t);
    const int smin = I > 0 ? I : 0;
    const int s = I + lane;
    const bool slot = (s >= smin && s <= smax);
    double R = 0.0, TH = 0.0, Rw = 0.0, Tw = 0.0;
    if (v.g.geo) {
        const int Dm = la.Dm;                          // lags summed pair by pair
        const int C = (Dm + la.parts - 1) / la.parts;
        // lags of this task: [dA, dB), dB cut where Ld passes the block's top slot
        // (Ld is nondecreasing; clipped lags hold kLagClipAll)
        const int dA = min(c * C, Dm);
        int dB = min(min(dA + C, Dm), smax + 1);
        // most shares end below the cut: one load settles it, else bisect
        if (dB > dA && __ldg(v.g.Ld + dB - 1) > smax) {
            int lo = dA, hi = dB;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (__ldg(v.g.Ld + mid) > smax) hi = mid; else lo = mid + 1;
            }
            dB = lo;
        }

        // j-side operand pointers: the staged window or the arrays themselves
        const double* pN = v.p.Nj;
        const double* pH = v.p.Hj;
        const double* pX = v.g.x;
        if (dB > dA) {
            int jw0 = smin - __ldg(v.g.Ld + dB - 1);
            jw0 = jw0 > 0 ? (jw0 & ~1) : 0;
            int jw1 = smax - __ldg(v.g.Ld + dA) + 1;       // exclusive, <= n - 1
            jw1 = (jw1 + 1) & ~1;                           // <= n: copies are padded
            const int cnt = jw1 - jw0;
            if (cnt > 0 && cnt <= kLaneWinMax) {
                const unsigned bytes = static_cast<unsigned>(cnt) * 8u;
                if (tid == 0) {
                    fence_proxy_async_smem();              // earlier generic reads of the window
                    mbar_expect_tx(bar, (NeedH<K>::j ? 3u : 2u) * bytes);
                    bulk_g2s(sm.wN, la.Ncp + jw0, bytes, bar);
                    if constexpr (NeedH<K>::j) bulk_g2s(sm.wH, v.p.Hj + jw0, bytes, bar);
                    bulk_g2s(sm.wX, la.xcp + jw0, bytes, bar);
                }
                if (!mbar_wait(bar, phase)) {
                    // the copy never completed: flag it, poison the block's bins, leave
                    if (tid == 0) *la.err = 1;
                    *s_flag = 1;
                }
                phase ^= 1u;
                pN = sm.wN - jw0;
                pH = sm.wH - jw0;
                pX = sm.wX - jw0;
            }
        }
        // this warp's contiguous share of the lags
        const int per = (dB - dA + kLaneWarps - 1) / kLaneWarps;
        const int dw0 = dA + w * per;
        if (!*s_flag) lane_pairs<K>(v, s, slot, dw0, min(dB, dw0 + per), pN, pH, pX, R, TH);
        if (!SCATTER && la.eh >= la.el) {
            // and of the runs summed by windows
            const int ne = la.eh - la.el + 1, sh = la.parts * kLaneWarps, q = c * kLaneWarps + w;
            lane_windows<K>(v, ws, s, slot, la.eh - ne * q / sh, la.eh - ne * (q + 1) / sh + 1, Rw, Tw);
        }
    } else {
        slot_pairs_any<K, 1>(v.g, &v.p, s, slot, c * kLaneWarps + w, la.parts * kLaneWarps, R, TH);
    }
    constexpr int NS = SCATTER ? 2 : 4;
    double* red = sm.red + w * NS * 32 + lane;
    red[0] = R;
    red[32] = TH;
    if constexpr (!SCATTER) {
        red[64] = Rw;
        red[96] = Tw;
    }
    __syncthreads();
    const bool poisoned = *s_flag != 0;

    SlotSums u{0.0, 0.0, 0.0, 0.0};
    unsigned em = 0u;
    bool finish = false;
    if (w == 0) {
#pragma unroll
        for (int q = 0; q < kLaneWarps; ++q) {
            const double* rq = sm.red + q * NS * 32 + lane;
            u.R += rq[0];
            u.TH += rq[32];
            if constexpr (!SCATTER) {
                u.Rw += rq[64];
                u.Tw += rq[96];
            }
        }
        em = exact_mask(v, t);
        finish = true;
        if (!SCATTER && (la.parts > 1 || em != 0u)) {
            double* bp = la.part + (static_cast<size_t>(t) * la.parts + c) * 128 + lane;
            bp[0] = u.R;
            bp[32] = u.TH;
            bp[64] = u.Rw;
            bp[96] = u.Tw;
            finish = block_ticket(ws, la, n, t, em, u);
        }
    }
    lane_finish<K, SCATTER>(v, ws, la, rhs, t, nclip, em, finish, !SCATTER || c == 0, poisoned, u, s_ex, s_mask);
    __syncthreads();
}

} // namespace pbe_gb300
