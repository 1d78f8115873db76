// IEEE double products on the integer pipe.
//
// One FP64 warp instruction takes an SM sub-partition of GB300 80 cycles; a
// product formed from four 32x32-bit multiplications takes 41 (measured on
// independent chains, operand splitting included) and runs beside the FP64
// sums.  A step of 7 products and 5 sums takes 480 cycles this way against
// 1041 with FP64 products (678 against 1100 for a warp alone).  A fallback
// product belongs behind a branch that is really taken: as a predicated
// instruction it costs its 80 cycles even when no lane needs it.
//
// The product of two 53-bit mantissas is formed exactly and rounded to
// nearest: one operand scaled by 2 and the other by 2^11 puts the top 53 or
// 54 bits in the upper word.  A tie needs the low half to be zero but for its
// top bit, so its lowest 32-bit word is zero: int_mul reports that word, and
// where it is zero the caller takes int_mul_even, which rounds ties to even.
// That happens for operands with 20 trailing zero bits between them: one
// product in 95,000 of independent full mantissas, one square in 1,024 (10
// bits suffice), and every one that follows a deep cancellation.  Operands and
// result must be normal.
#pragma once

#include "scaled.h"

namespace fx {

struct FactorA {  // mantissa * 2
    std::uint32_t h, l;
    int x;        // sign and exponent
};
struct FactorB {  // mantissa * 2^11
    std::uint32_t h, l;
    int x;
};

FX_HD std::uint32_t shift_in(std::uint32_t low, std::uint32_t high, int n) {  // upper word of (high:low) << n
#ifdef __CUDA_ARCH__
    return __funnelshift_l(low, high, n);
#else
    return (high << n) | (low >> (32 - n));
#endif
}

FX_HD FactorA factor_a(double v) {
    const std::uint32_t h = static_cast<std::uint32_t>(hi_of(v)), l = lo_of(v);
    FactorA f;
    f.h = shift_in(l, (h & 0xfffffu) | 0x100000u, 1);
    f.l = l + l;
    f.x = static_cast<int>(h & 0xfff00000u);
    return f;
}

FX_HD FactorB factor_b(double v) {
    const std::uint32_t h = static_cast<std::uint32_t>(hi_of(v)), l = lo_of(v);
    FactorB f;
    f.h = shift_in(l, (h & 0xfffffu) | 0x100000u, 11);
    f.l = l << 11;
    f.x = static_cast<int>(h & 0xfff00000u);
    return f;
}

FX_HD std::uint64_t wide_mad(std::uint32_t a, std::uint32_t b, std::uint64_t c) {
#ifdef __CUDA_ARCH__
    std::uint64_t r;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
#else
    return static_cast<std::uint64_t>(a) * b + c;
#endif
}

template <bool Even>
FX_HD double int_product(const FactorA& a, const FactorB& b, std::uint32_t& low) {
    const std::uint64_t t0 = wide_mad(a.l, b.l, 0);
    const std::uint64_t t1 = wide_mad(a.h, b.l, t0 >> 32);
    const std::uint64_t t2 = wide_mad(a.l, b.h, static_cast<std::uint32_t>(t1));
    const std::uint64_t top = wide_mad(a.h, b.h, t1 >> 32) + (t2 >> 32);
    low = low < static_cast<std::uint32_t>(t0) ? low : static_cast<std::uint32_t>(t0);
    // In [2^52, 2^54): one more bit to drop when the 54th is set.  The bit
    // below the mantissa is then the lowest bit kept here, else the next
    // word's top bit.
    const std::uint32_t c = static_cast<std::uint32_t>(top >> 53);
    const std::uint64_t r = top + ((static_cast<std::uint32_t>(t2) >> 31) | c);
    const std::uint32_t rl = static_cast<std::uint32_t>(r), rh = static_cast<std::uint32_t>(r >> 32);
#ifdef __CUDA_ARCH__
    std::uint32_t ol = __funnelshift_r(rl, rh, c);
#else
    std::uint32_t ol = static_cast<std::uint32_t>(r >> c);
#endif
    if (Even) {
        // Exactly half: the dropped bit set and nothing below it.
        const std::uint32_t next = static_cast<std::uint32_t>(t2), last = static_cast<std::uint32_t>(t0);
        const bool half = last == 0 && (c ? next == 0 && (static_cast<std::uint32_t>(top) & 1u) != 0
                                          : next == 0x80000000u);
        if (half) ol &= ~1u;
    }
    // Sign and exponent words add; the mantissa carries its leading bit.
    const std::uint32_t oh = (rh >> c) + (c << 20)
        + (static_cast<std::uint32_t>(a.x) + static_cast<std::uint32_t>(b.x) - (1024u << 20));
    return from_hilo(static_cast<int>(oh), ol);
}

// The correctly rounded product; `low` becomes zero where it may be a tie.
FX_HD double int_mul(const FactorA& a, const FactorB& b, std::uint32_t& low) { return int_product<false>(a, b, low); }

// The correctly rounded product, ties included.
FX_HD double int_mul_even(const FactorA& a, const FactorB& b) {
    std::uint32_t low = 0;
    return int_product<true>(a, b, low);
}

}  // namespace fx
