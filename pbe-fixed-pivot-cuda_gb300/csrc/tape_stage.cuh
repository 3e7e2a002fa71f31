// =============================================================================
// tape_stage.cuh -- the small parts of a Runge-Kutta stage of the tape, as device
// functions: other kernels of the stage carry them (aggregation.cu, breakage.cu).
// A stage is a chain of kernels of a few microseconds each: with a kernel of its own
// for every part, six of them and a memset, a stage of n = 3840 took 95 us.
// =============================================================================
#pragma once

#include "pbe_internal.cuh"

namespace pbe_gb300 {

// Shares of one fragment: (to lo, to lo+1). Clipped fragments put everything
// into the first share.
__device__ __forceinline__ void frag_shares(const double* __restrict__ x, int n, int lo, double v,
                                            double contrib, double& clo, double& chi)
{
    if (lo < 0 || lo >= n - 1) { clo = contrib; chi = 0.0; return; }
    const double xl = __ldg(x + lo), xh = __ldg(x + lo + 1);
    const double q = contrib / (xh - xl);
    clo = q * (xh - v);
    chi = q * (v - xl);
}

constexpr int kBrkPrepBlock = 256;     // fragments of a breakage prep block (BrkWs::clipsum)
__host__ __device__ constexpr int brk_prep_blocks(int n, int nq)
{
    return static_cast<int>((static_cast<long long>(n) * nq + kBrkPrepBlock - 1) / kBrkPrepBlock);
}

// The breakage prep of a stage by one CTA: the shares of the fragments of prep block
// `blk` from the kept brackets and selection values, S_j N_j, and the block's sum of
// what is clipped below x[0]. sh: >= blockDim/32 doubles.
__device__ __forceinline__ void brk_stage_block(const double* __restrict__ N, const double* __restrict__ x,
                                                const double* __restrict__ t_q, const double* __restrict__ bw_q,
                                                int n, int nq, const BrkWs& ws, int blk, double* sh)
{
    double clipped = 0.0;
    for (int u = threadIdx.x; u < kBrkPrepBlock; u += blockDim.x) {
        const long long idx = static_cast<long long>(blk) * kBrkPrepBlock + u;
        if (idx >= static_cast<long long>(n) * nq) break;
        const int q = static_cast<int>(idx / n), j = static_cast<int>(idx - static_cast<long long>(q) * n);
        const double v = x[j] * t_q[q], S = ws.Ssel[j], Nj = N[j];
        const int lo = ws.lo[idx];
        const bool active = (S != 0.0) && (Nj > kBreakageNMin);
        double clo, chi;
        frag_shares(x, n, lo, v, active ? S * Nj * bw_q[q] : 0.0, clo, chi);
        ws.clo[idx] = clo;
        ws.chi[idx] = chi;
        if (lo < 0) clipped += clo;                    // all of it goes to bin 0
        if (q == 0) ws.SN[j] = active ? S * Nj : 0.0;
    }
    // summed in a fixed order (most blocks have none: one barrier tells)
    if (__syncthreads_or(clipped != 0.0)) clipped = block_sum(clipped, sh);
    if (threadIdx.x == 0) ws.clipsum[blk] = clipped;
}

// Stage q of one RK4 step for bin i with k_i (same rounding as the reference's host loop):
// q = 0: acc = k; Y = N + c k.   q = 1, 2: acc += 2 k; Y = N + c k.
// q = 3: acc += k; N += dt6 acc.
__device__ __forceinline__ void rk_update(const RkStage& st, int i, double ki)
{
    if (st.q == 0) {
        st.acc[i] = ki;
        st.Y[i] = __dadd_rn(st.N[i], __dmul_rn(st.c, ki));
    } else if (st.q < 3) {
        st.acc[i] = __dadd_rn(st.acc[i], __dmul_rn(2.0, ki));
        st.Y[i] = __dadd_rn(st.N[i], __dmul_rn(st.c, ki));
    } else {
        st.N[i] = __dadd_rn(st.N[i], __dmul_rn(st.dt6, __dadd_rn(st.acc[i], ki)));
    }
}

} // namespace pbe_gb300
