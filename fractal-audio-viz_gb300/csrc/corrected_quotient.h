// Quotients by a divisor known ahead, without the division.
#pragma once

#include "scaled.h"

#ifndef __CUDA_ARCH__
#include <cmath>
#endif

namespace fx {

// x / d given r = RN(1 / d): the rounded product corrected once (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// IBM J. Res. Dev. 34(1), 1990).  The callers say where that is the IEEE
// quotient.
FX_HD float corrected_quotient(float x, float d, float r) {
#ifdef __CUDA_ARCH__
    const float q = __fmul_rn(x, r);
    return __fmaf_rn(__fmaf_rn(-q, d, x), r, q);
#else
    const float q = x * r;
    return std::fmaf(std::fmaf(-q, d, x), r, q);
#endif
}

// offset / dimension given 1 / dimension: the IEEE quotient for every integer
// and half-integer offset within a dimension up to 32768.
FX_HD float offset_quotient(float offset, float dimension, float per) {
    return corrected_quotient(offset, dimension, per);
}

// v / 255 for a palette share v in [0, 256): the IEEE quotient from 2^-100 on;
// a share below that moves no byte.
FX_HD float byte_share(float v) { return corrected_quotient(v, 255.0f, 1.0f / 255.0f); }

}  // namespace fx
