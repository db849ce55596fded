// div_rn.cuh -- correctly rounded division by a divisor whose reciprocal is known.
//
// Markstein's final correction step (P. Markstein, "IA-64 and Elementary Functions",
// Prentice Hall 2000; also M. Cornea, J. Harrison, P. T. P. Tang, "Scientific Computing
// on Itanium-based Systems", Intel Press 2002): with y = RN(1/D), the product
// q = RN(u y) is within one ulp of u / D, the residual r = u - D q is exact in one fused
// multiply-add, and RN(q + r y) is the correctly rounded quotient RN(u / D), for
// operands and quotients inside the normal range (the window below); when r is zero q is
// already the exact quotient.  y comes from __drcp_rn, formed off a recurrence's critical
// path (D does not depend on the previous step), so the dependent work per step is one
// multiply and two fused multiply-adds.
//
// The correction step is exact only while the operands and the quotient stay inside the
// normal range with room to spare: y = RN(1/D) must be normal, u - D q must be
// representable (it is about 2^-53 |u|, so u must lie well above the subnormal range)
// and q must neither overflow nor underflow.  The divisors here are Thomas pivots, and
// plan creation checks that every pivot satisfies 2^-40 <= |D| <= 2^1000
// (PRJ_ERR_NUMERIC otherwise).  With D in that range, |q| in [2^-900, 2^1000) implies
// |u| >= 2^-941, so all three conditions hold; the function tests only the quotient's
// exponent (its high word: a mask, a subtraction and a compare).
//
// A zero u gives a zero of the right sign but for u = -0 with D > 0 (there r y = +0 turns
// q = -0 into +0); that case counts as outside the window, the other zeros do not.
// Quotients outside it -- and subnormals, infinities and NaNs with them -- are the caller's to
// take from __ddiv_rn.  prj_selftest_division compares that pair with __ddiv_rn bit for bit
// on random pairs of that domain, with the window's edges weighted.
//
// The function has no branch: one per quotient kept the real and imaginary parts of a line,
// and the lines of a thread, from overlapping.  Measured on one warp, the forward Thomas step
// of a complex line takes 199 cycles with a branch in the function and 41 without.
#pragma once

namespace prj {

// smallest and largest |D| for which div_by_recip is correctly rounded inside its window
constexpr double kDivRecipMinD = 0x1p-40;
constexpr double kDivRecipMaxD = 0x1p1000;

// RN(u / D) with y = RN(1 / D); `outside` becomes non-zero when the result may differ
__device__ __forceinline__ double div_by_recip(double u, double D, double y, unsigned& outside) {
    const double q = __dmul_rn(u, y);
    const double r = __fma_rn(-D, q, u);
    // 2^-900 <= |q| < 2^1000: the biased exponent of q in [123, 2023)
    const unsigned hq = (unsigned)__double2hiint(q) & 0x7fffffffu;
    const bool q_in = hq - 0x07B00000u < 0x7E700000u - 0x07B00000u;
    // 0 for u = +0, and for u = -0 with D < 0
    const unsigned not_zero = ((unsigned)__double2hiint(u) & ~((unsigned)__double2hiint(D) & 0x80000000u)) |
                              (unsigned)__double2loint(u);
    outside |= q_in ? 0u : not_zero;
    return __fma_rn(r, y, q);
}

}  // namespace prj
