// hype_div.cuh -- IEEE round-to-nearest-even FP64 reciprocal and quotient as straight
// lines of fused multiply-adds, for the bit-exact kernels.
//
// The compiler's division ends in a branch to its own slow path, which keeps
// independent divisions from overlapping; these have no branch, so the WENO weights of
// a reconstruction (reconstruction.c:163-170, 186-193, 207-215) and the two sides of a
// Riemann problem issue as interleaved chains, and quotients by one divisor share its
// reciprocal.  Methods: P. Markstein, IBM J. Res. Dev. 34 (1990), and "IA-64 and Elementary
// Functions", 2000, ch. 8; the exact-remainder property in J.-M. Muller et al., "Handbook of
// Floating-Point Arithmetic", 2010, sec. 4.3.  The callers check their operands' ranges and
// repeat with the compiler's division outside them.  tests/test_gpu_division.py compares
// both functions with IEEE division on 2^30 operand pairs per run (hype_test_division).
#pragma once
#include <cuda_runtime.h>

namespace hype {

__device__ __forceinline__ unsigned biased_exp(double x) { return (unsigned)((__double_as_longlong(x) >> 52) & 0x7ff); }

// 1/b correctly rounded, for b normal with |binary exponent| <= 1000:
//   y0 ~ 1/b: the hardware approximation (PTX rcp.approx.ftz.f64, about 20 bits, its low word zero)
//        with 2^31 as its low word: about 2^-21 more than the approximation;
//   y1 = y0 + e s, s = y0 + y0 e, e = 1 - b y0: Chebyshev's third-order iteration y0 (1 + e + e^2)
//        by Horner's rule, (1/b)(1 - e^3).  s rounds to 2^-53 of itself, 2^-73 of y1, and e^3 is below
//        2^-57, so y1 is one of the two doubles around 1/b;
//   y2 = y1 + y1 (1 - b y1), both by fma: rounds (1/b)(1 - e1^2), |e1| <= 2^-53; no midpoint
//        of two doubles lies between that and 1/b unless b is all ones (Markstein 2000, ch. 8).
// For b = 2^k (2 - 2^-52), all ones, 1/b = L (1 + 2^-53 + 2^-106 + ...), L = 2^-(k+1), lies just above
// the midpoint of L and U = L (1 + 2^-52).  y0 = L (1 + 2^-21) is above it, so e < 0, y1 above the
// midpoint by about 2^-63 L, which its rounding errors of 2^-74 L leave, and rounds to U; then
// y2 = U (1 - 2^-53 + 2^-105) = L (1 + 2^-53 + 2^-157) rounds to U, which is right.  (From y0 = L, y1 is
// the midpoint itself and both steps end on L.)
// Five fused multiply-adds, no branch.  All-ones divisors are common: the density 1 - 2^-53 that
// (alpha rho) / alpha gives in quiescent gas.
__device__ __forceinline__ double rcp_rn(double b)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    y = __hiloint2double(__double2hiint(y), (int)0x80000000u);
    const double e = fma(-b, y, 1.0);
    const double s = fma(y, e, y);
    y = fma(e, s, y);
    return fma(y, fma(-b, y, 1.0), y);
}

// a / b correctly rounded from y = rcp_rn(b): quotients by one divisor share y.  q1 = a y and one
// correction give a double next to a/b, whose remainder a - b q1 is exact; with y the correctly
// rounded 1/b the second correction rounds correctly (Markstein 1990, theorem 5).  b and a/b of
// binary exponents in [-1000, 1000] and [-900, 1000], a in [-900, 1000] or zero.  A zero's quotient
// is a zero, but +0 for -0 over a positive divisor too: callers may pass zeros only where the sign
// of a zero reaches no result (velocities, pressures and volume products end up as terms of sums
// that begin with +0).
__device__ __forceinline__ double div_rn(double a, double b, double y)
{
    double q = a * y;
    double r = fma(-b, q, a);
    q = fma(r, y, q);
    r = fma(-b, q, a);   // exact
    return fma(r, y, q);
}

// whether a, b and a/b are in div_rn's range (hype_test_division; the callers ensure it by the ranges
// of densities, pressures and weights, CrDiv and CrCheck, which that test checks too)
__device__ __forceinline__ bool div_in_range(double a, double b, double quotient)
{
    auto within = [](unsigned e, unsigned lo) { return e >= 1023u - lo && e <= 1023u + 1000u; };
    return (a == 0.0 || within(biased_exp(a), 900u)) && within(biased_exp(b), 1000u) && (a == 0.0 || within(biased_exp(quotient), 900u));
}

}  // namespace hype
