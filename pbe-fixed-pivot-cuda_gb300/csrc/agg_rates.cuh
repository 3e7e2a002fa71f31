// =============================================================================
// agg_rates.cuh -- pair rates and the death polynomial of the six aggregation
// kernels, and the thread groups that the batched and VJP kernels work in.
// =============================================================================
#pragma once

#include "pbe_internal.cuh"
#include "exact_weight.cuh"

namespace pbe_gb300 {

template <int K> struct NeedH {
    static constexpr bool j = (K == 1 || K == 2 || K == 4 || K == 5);
    static constexpr bool k = (K == 1 || K == 2);
};

// Pair rate on a verified geometric grid, lag tables B = c_d * Bfactor(d),
// S = c_d * Sfactor(d) with c_d = 1/2 for d = 0 (times beta in the
// single-instance tables; the batched tables leave beta to Nj / hj).
template <int K>
__device__ __forceinline__ double rate_geo(double B, double S, double Nj, double hj,
                                           double Nk, double hk)
{
    if constexpr (K == 0 || K == 3) return (B * Nj) * Nk;
    else if constexpr (K == 1) return B * fma(hj, Nk, Nj * hk);
    else if constexpr (K == 2) return (B * hj) * hk;
    else if constexpr (K == 4) return (S * hj) * Nk;
    else return Nk * fma(S, hj, B * Nj);
}

// Lags whose pairs land on the larger member's own slot (lo = k): the rate is
// F_k * q_slot(j) with the per-slot factor F_k = N_k (h_k for Product). Not
// used for Sum, whose rate has two k-dependent terms.
template <int K>
__device__ __forceinline__ double q_slot(double B, double S, double Nj, double hj)
{
    if constexpr (K == 0 || K == 3) return B * Nj;
    else if constexpr (K == 2) return B * hj;
    else if constexpr (K == 4) return S * hj;
    else return fma(S, hj, B * Nj);
}

// sum_k beta(x_i, x_k) N_k from the moments
// M[0] = sum N/a, M[1] = sum N, M[2] = sum a N, M[3] = sum a^2 N, M[4] = sum x N.
template <int K>
__device__ __forceinline__ double death_factor(double xi, double ai, double iai,
                                               const double* M, double b0, double bbr,
                                               double bsh)
{
    if constexpr (K == 0) return b0 * M[1];
    else if constexpr (K == 1) return b0 * fma(xi, M[1], M[4]);
    else if constexpr (K == 2) return (b0 * xi) * M[4];
    else {
        double f = 0.0;
        // beta_br (a_i/a_k + a_k/a_i + 2)
        if constexpr (K == 3 || K == 5) f = bbr * (fma(ai, M[0], iai * M[2]) + 2.0 * M[1]);
        // beta_sh (a_i + a_k)^3 = beta_sh (x_i + 3 a_i^2 a_k + 3 a_i a_k^2 + x_k)
        if constexpr (K == 4 || K == 5)
            f = fma(bsh, fma(xi, M[1], (3.0 * ai) * fma(ai, M[2], M[3])) + M[4], f);
        return f;
    }
}

constexpr int kMaxGroups = kMainThreads / 32;

// A group of T threads (T a multiple of 32, T <= kMainThreads) working on one
// task; named barrier g + 1 (barrier 0 stays free for __syncthreads).
struct TileGroup {
    int g;       // group index within the CTA
    int lane;    // thread index within the group
    int T;       // group size
    __device__ __forceinline__ void sync() const
    {
        asm volatile("bar.sync %0, %1;" :: "r"(g + 1), "r"(T) : "memory");
    }
};

} // namespace pbe_gb300
