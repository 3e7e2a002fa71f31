// =============================================================================
// agg_moments.cuh -- rules of the prefix moments behind the separated pair sums
// (agg_lane.cuh derives them): which moments a kernel type needs, and which
// slots must keep their exact pair sums.
// =============================================================================
#pragma once

#include "pbe_internal.cuh"

namespace pbe_gb300 {

// Moments that kernel type K's rates need: beta(x_j, x_k) is a sum of products
// of powers of x_j and x_k, with the powers {-1/3, 0, 1/3, 2/3, 1} of x_j.
template <int K>
__device__ __forceinline__ constexpr bool need_moment(int q)
{
    return K == 0 ? q == 1 : K == 1 ? (q == 1 || q == 4) : K == 2 ? q == 4
         : K == 3 ? q <= 2 : K == 4 ? q >= 1 : true;
}

// Largest move of a bin, relative to the bin's sum of |contributions|, that the
// separated sums may make by leaving out the rounding of fl(x_j + x_k).
constexpr double kMomGuard = 2.5e-13;

// The slot's lags from D0 on must be summed pair by pair (see the file header):
// u |N_s| > kMomGuard |N_{s+1}|, u = 2^-53 x_{s+1} / dx_s (2^53 on the other
// side, so that no product underflows for subnormal N).
__device__ __forceinline__ bool mom_exact_slot(double Ns, double Nup, double xup, double inv_dx)
{
    return fabs(Nup) * (kMomGuard * 9007199254740992.0) < (xup * inv_dx) * fabs(Ns);
}

} // namespace pbe_gb300
