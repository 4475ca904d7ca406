// Quotients by a kept reciprocal. Nothing here needs CUDA but its function qualifiers, fabsf and
// __fmaf_rn (a fused multiply-add rounded once): the tests compile this file for the host too.
#pragma once

namespace ntr {

// a / b correctly rounded for b > 0, from y = 1 / b correctly rounded: one step brings a * y within
// an ulp of the quotient, the second rounds it correctly (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990, theorem on q + r y).
// It holds while no product or remainder underflows or overflows: 2^-80 <= |a| <= 2^40 with 2^-60 <=
// b <= 2^40 (1.2e9 random operands, none different from a / b). Zero keeps its sign; anything else
// divides, in a call, which the compiler does not run ahead of its condition: a division takes its
// long way for a zero numerator (in the pressure solve, 300 cycles a half-sweep beside the rest's 100).
__device__ __noinline__ float div_any(float a, float b) { return a / b; }
__device__ __forceinline__ float div_by(float a, float b, float y) {
    const float m = fabsf(a);
    const bool wide = b >= 0x1p-60f && b <= 0x1p40f;
    const bool fine = wide && m >= 0x1p-80f && m <= 0x1p40f;
    float q = a * y;
    float e = __fmaf_rn(-q, b, a);
    q = __fmaf_rn(e, y, q);
    e = __fmaf_rn(-q, b, a);
    q = fine ? __fmaf_rn(e, y, q) : a;
    if (!fine && !(wide && a == 0.0f)) q = div_any(a, b);
    return q;
}

}  // namespace ntr
