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
// On other grids the same holds for the rows j < J0(s), the first j with
// fl(x_j + x_s) >= x_{s+1}.
//
// Work split: blocks of 32 output bins aligned to the top of the grid (block
// t owns bins [n - 32 (t + 1), n - 32 t), so bin n - 1 is never a block's first
// bin); a task is one block and one of `parts` equal shares of the lags below D0
// (of each slot's rows on other grids); the CTA's eight warps take equal
// contiguous shares of the task's lags (each warp sees its runs in order) and
// their sums are added in warp order. With several parts each task stores its
// 2 x 32 sums; the block's last task (ticket) adds them in order and writes the
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

// Shares of a block's direct lags: enough tasks to give every CTA several (the
// last ones then end together), at least 32 lags each (4 per warp). A share
// longer than the staged window reads its operands from the arrays.
__host__ __device__ constexpr int lane_parts(int lags, int nblk, int ctas)
{
    int p = (4 * ctas + nblk - 1) / nblk;
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
    double* red;     // [kLaneWarps][2][32] per-warp R, TH
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

// One warp, after its contribution to block t is stored: the block's ticket.
// True for the last of its `parts` share tasks and one task per exact slot;
// that one gets the block's sums, added in a fixed order.
__device__ __forceinline__ bool block_ticket(const AggWs& ws, const LaneArgs& la, int n, int t,
                                             unsigned exact, double& Rt, double& THt)
{
    const int lane = threadIdx.x & 31;
    const int want = la.parts + __popc(exact);
    __threadfence();                                   // every lane's stores before the ticket
    __syncwarp();
    int last = 0;
    if (lane == 0) last = (atomicAdd(la.ticket + t, 1) == want - 1);
    if (!__shfl_sync(0xffffffffu, last, 0)) return false;
    __threadfence();
    Rt = 0.0;
    THt = 0.0;
    const double* bp = la.part + static_cast<size_t>(t) * la.parts * 64;
    for (int q = 0; q < la.parts; ++q) {
        Rt += __ldcg(bp + q * 64 + lane);
        THt += __ldcg(bp + q * 64 + 32 + lane);
    }
    if ((exact >> lane) & 1u) {
        const int s = n - kLaneBins * (t + 1) + lane;
        Rt += __ldcg(ws.xsum + 2 * s);
        THt += __ldcg(ws.xsum + 2 * s + 1);
    }
    return true;
}

// One warp: the bins of block t from its slots' sums (a slot per lane). With
// `first` the prefix part (not of the exact slots) and the death term are added;
// scatter mode calls it for every share's own sums.
template <int K, bool SCATTER>
__device__ void lane_finish(const LaneView& v, const AggWs& ws, double* rhs, int t,
                            int nclip, unsigned exact, bool first, bool poisoned, double Rt,
                            double THt)
{
    const int n = v.g.n, lane = threadIdx.x & 31;
    const int I = n - kLaneBins * (t + 1);
    const int smax = lane_block_smax(n, t);
    const int s = I + lane, i = s;
    const bool slot = s >= 0 && s <= smax;
    const double xs = slot ? __ldg(v.g.x + s) : 0.0;
    const int St = slot ? -exponent_of(xs) : 0;
    double clip0 = 0.0;                                // the prefix part of the clipped slot n - 1
    double death = 0.0;
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
                Rt += r;
                THt += scale_down(th, exponent_of(__ldg(v.g.x + cut - 1)) + St);
            } else {
                clip0 = r;
            }
        }
    }
    // own part of bin i (slot i) and the w-part of slot i, owed to bin i + 1
    double b1 = 0.0, co = 0.0;
    if (slot) {
        const double sd = scalbn(__ldg(v.g.inv_dx + i), -St);
        b1 = fma(-THt, sd, Rt);
        co = THt * sd;
    }
    const double cin = __shfl_up_sync(0xffffffffu, co, 1);
    if (i >= 0) {
        double val = b1;
        if (lane >= 1) val += cin;
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
        if (lane == 31 && slot && co != 0.0) atomicAdd(rhs + i + 1, co);
    } else if (lane == 31 && t >= 1) {
        // carry into bin I + 32, the first bin of block t - 1
        ws.tcarry[t - 1] = co;
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
                                double* rhs, int s, int nclip, double* red, bool poisoned)
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
            const unsigned em = exact_mask(v, t);
            double Rt, THt;
            if (block_ticket(ws, la, n, t, em, Rt, THt))
                lane_finish<K, false>(v, ws, rhs, t, nclip, em, true, poisoned, Rt, THt);
        }
    }
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
                          unsigned& phase, int* s_flag)
{
    const int n = v.g.n;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int I = n - kLaneBins * (t + 1);
    const int smax = lane_block_smax(n, t);
    const int smin = I > 0 ? I : 0;
    const int s = I + lane;
    const bool slot = (s >= smin && s <= smax);
    double R = 0.0, TH = 0.0;
    if (v.g.geo) {
        const int Dm = min(v.g.D0, n);                 // lags summed pair by pair
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
    } else {
        slot_pairs_any<K, 1>(v.g, &v.p, s, slot, c * kLaneWarps + w, la.parts * kLaneWarps, R, TH);
    }
    sm.red[(w * 2 + 0) * 32 + lane] = R;
    sm.red[(w * 2 + 1) * 32 + lane] = TH;
    __syncthreads();
    const bool poisoned = *s_flag != 0;

    if (w == 0) {
        double Rt = 0.0, THt = 0.0;
#pragma unroll
        for (int q = 0; q < kLaneWarps; ++q) {
            Rt += sm.red[(q * 2 + 0) * 32 + lane];
            THt += sm.red[(q * 2 + 1) * 32 + lane];
        }
        const unsigned em = exact_mask(v, t);
        bool finish = true;
        if (!SCATTER && (la.parts > 1 || em != 0u)) {
            double* bp = la.part + (static_cast<size_t>(t) * la.parts + c) * 64;
            bp[lane] = Rt;
            bp[32 + lane] = THt;
            finish = block_ticket(ws, la, n, t, em, Rt, THt);
        }
        if (finish)
            lane_finish<K, SCATTER>(v, ws, rhs, t, nclip, em, !SCATTER || c == 0, poisoned, Rt, THt);
    }
    __syncthreads();
}

} // namespace pbe_gb300
