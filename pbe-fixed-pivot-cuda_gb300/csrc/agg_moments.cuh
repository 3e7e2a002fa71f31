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

// The same for a row of the VJP (vjp.cu), relative to its sum of |terms|.
constexpr double kVjpGuard = 5e-13;

// Window sums (agg_lane.cuh) pay on grids of about 64 sections an octave and more:
// neighbour ratio at most kWinRatio = 2^(1/64). Lags up to x_d = kWinStart x_0 are summed
// pair by pair: from there on a run has at least 6 lags (1 + x_d / x_0, within
// one), a window more than 4 bins, and costs 22 FP64 instructions against 4 a pair.
// The tables hold moments up to x^2 N in units of 2^E of x_0, E = win_exponent (a multiple
// of 3, so that cube roots scale exactly): N down to 1e-300 stays normal in them, where
// x^2 N itself would underflow, and up to 1e187 finite within kWinOctaves.
constexpr double kWinRatio = 1.0109;
constexpr double kWinStart = 6.0;
constexpr int kWinOctaves = 200;
__device__ __forceinline__ bool win_grid(const double* __restrict__ x, int n)
{
    return n >= 2 && x[1] <= kWinRatio * x[0] && exponent_of(x[n - 1]) - exponent_of(x[0]) <= kWinOctaves &&
           exponent_of(x[0]) > -900;
}
__device__ __forceinline__ int win_exponent(const double* __restrict__ x)
{
    const int E = exponent_of(x[0]);
    return 3 * ((E >= 0 ? E : E - 2) / 3);
}
// All pair rates of a population without negative entries have one sign, but with Brownian
// and shear coefficients of opposite signs (no windows then: kRatesMixed). The windows'
// rule compares sums of such rates, taken positive: the sign bit to flip. Host side (the
// comparisons at the kernel's start took 0.8 % of a tape's time).
constexpr int kRatesMixed = 1;
inline int rates_flip(int kernel, double b0, double bbr, double bsh)
{
    const bool br = kernel == 3 || kernel == 5, sh = kernel >= 4;
    if (br && sh && ((bbr < 0.0 && bsh > 0.0) || (bbr > 0.0 && bsh < 0.0))) return kRatesMixed;
    const bool neg = kernel <= 2 ? b0 < 0.0 : (br && bbr < 0.0) || (sh && bsh < 0.0);
    return neg ? static_cast<int>(0x80000000u) : 0;
}
__device__ __forceinline__ double flip_sign(double v, int flip)
{
    return __hiloint2double(__double2hiint(v) ^ flip, __double2loint(v));
}
// Moments m_{-1..6} (index m + 1) that kernel type K's windows need.
template <int K>
__device__ __forceinline__ constexpr bool need_window(int m)
{
    return (m < kMomN && need_moment<K>(m)) || (m >= 3 && need_moment<K>(m - 3));
}

} // namespace pbe_gb300
