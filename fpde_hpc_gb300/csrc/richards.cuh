// Closures of the reference's Richards problem (fpde_hpc_1d.cpp, analytic_test 0 with the van
// Genuchten-Mualem water content of cv_form 4): water content wetness :2493-2522, the inverse
// of its derivative inv_dw_dh :2523-2566 and the relative conductivity of KK :2625-2655
// (k_form 1 van Genuchten-Mualem, 2 Averianov), as functions of the suction P in metres. The
// soil constants are the reference's. The expressions keep its operation order. Its powers with
// exponents in quarters (n = 1.25, 2n = 2.5, 0.5, 2 and 3.5) are products and square roots, each
// correctly rounded (at most 2 ulps together, pow's own bound): a general pow is over a hundred
// FP64 instructions on a pipe that issues one warp instruction per 16 cycles and SM, and these
// were 11 of a node's 15. The others (0.2, 0.8, 5) are CUDA's pow; values agree with the host's
// to a few ulps.
#pragma once

namespace fpde {

constexpr double RICH_N = 1.25, RICH_S0 = 0.0736, RICH_S1 = 0.55, RICH_A = 0.066;
constexpr double RICH_SATURATED = 1e20;          // inv_dw_dh where the soil is saturated

constexpr double RICH_HN = 316.22776601683793320, RICH_H2N = 1e5;   // 100^1.25, 100^2.5

__device__ __forceinline__ double rich_pow_n(double x) { return x * sqrt(sqrt(x)); }        // x^1.25
__device__ __forceinline__ double rich_pow_2n(double x) { return (x * x) * sqrt(x); }       // x^2.5

__device__ __forceinline__ double rich_wetness(double P)
{
    const double n = RICH_N, s0 = RICH_S0, s1 = RICH_S1, a = RICH_A;
    P *= 100.0;                                   // centimetres
    if (P <= 0.0) return s1;
    return s0 + ((s1 - s0) / pow(1 + rich_pow_n(a * P), (1 - 1 / n)));
}

__device__ __forceinline__ double rich_inv_dw_dh(double P)
{
    const double n = RICH_N, s0 = RICH_S0, s1 = RICH_S1, a = RICH_A;
    if (P <= 0.0) return RICH_SATURATED;
    const double hn = RICH_HN, h2n = RICH_H2N;
    const double apn = rich_pow_n(a * P);
    const double Ch = ((((1 - n) * hn * s0 + (n - 1) * hn * s1) * apn * pow(1 + hn * apn, (1 / n))) /
                       (h2n * P * rich_pow_2n(a * P) + 2 * hn * P * apn + P));
    return Ch != 0.0 ? 1.0 / Ch : RICH_SATURATED;
}

// KK = Kr(wetness) * k_sat
__device__ __forceinline__ double rich_KK(double P, int kform, double ksat)
{
    const double n = RICH_N, s0 = RICH_S0, s1 = RICH_S1;
    const double x = (rich_wetness(P) - s0) / (s1 - s0);
    double Kr = 1.0;
    if (kform == 1) {
        const double m = 1.0 - pow(1.0 - pow(x, (1.0 / (1.0 - 1.0 / n))), (1.0 - 1.0 / n));
        Kr = sqrt(x) * (m * m);
    }
    if (kform == 2) Kr = ((x * x) * x) * sqrt(x);
    return Kr * ksat;
}

}  // namespace fpde
