// exact_div.cuh -- a / b, correctly rounded, for a divisor whose reciprocal is
// known.  Free of the CUDA runtime, so that a host build of it can be checked.
#pragma once

#include <math.h>

namespace bcmc {

// a / b rounded to nearest, given inv = 1 / b rounded to nearest, by Markstein's
// method (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990): the product's residual a - q b is exact in a
// fused multiply-add, a first correction makes q one of the two neighbours of
// a / b, and the second rounds it.  For finite a and b away from the ends of the
// range, where no residual underflows (here: positions within a volume).
// tests/test_exact_div_host.py holds it to the quotient for every position of
// every volume size up to 1200 on an axis.
__device__ __forceinline__ float exact_div(float a, float b, float inv)
{
    float q = a * inv;
    q = fmaf(fmaf(-q, b, a), inv, q);
    return fmaf(fmaf(-q, b, a), inv, q);
}

}  // namespace bcmc
