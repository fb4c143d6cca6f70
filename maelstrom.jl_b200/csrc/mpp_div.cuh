// Division by a number whose rounded reciprocal is at hand, without the division's cost in a chain:
// the quotient's estimate a rd and its residual, exact in one fused multiply-add, corrected
// (P. Markstein, IBM J. Res. Dev. 34, 1990: a faithful estimate corrected so is the rounded quotient).
// The result is the IEEE quotient bit for bit over the ranges stated, but for the sign of a zero; an
// infinite or NaN quotient stays one of the two (an infinite a gives NaN), so no finite value differs.
// Keeping infinities and -0 too (a select beside the chain) costs what is a chain of these 0.5 to 1 %
// (32^3 projection 510 -> 513 us, 64^3 1076 -> 1084, a small sparse basin 1360 -> 1374, the runs' own
// difference taken off); a branch as much as the division it avoids (a half-sweep of the coarsest solve
// at 128 threads 157 cycles, with the division 144, so 105).
// (Plain C++ but for the qualifiers: tests/test_division.py checks these statements on the CPU.)
#pragma once

namespace mpp {

// d = 1 .. 6, a level's count of open faces. Every mantissa is right for every d, down to subnormal
// quotients too, except that ties of d = 6 among those (|a / d| < 2^-126) may go the other way.
__device__ __forceinline__ float div_small(float a, float d, float rd) {
    const float q = a * rd;
    return fmaf(fmaf(-q, d, a), rd, q);
}
// Any d of ordinary size, in [2^-30, 2^30], |a| >= 2^-70 or zero; the first correction makes the estimate
// faithful.
__device__ __forceinline__ float div_rn(float a, float d, float rd) {
    float q = a * rd;
    q = fmaf(fmaf(-q, d, a), rd, q);
    return fmaf(fmaf(-q, d, a), rd, q);
}

}  // namespace mpp
