// Horner evaluation of the image series at a pixel offset (renderer.cpp:8594-8639).
//
// In ScaledComplex form a term is a product and a sum, 8 FP64 instructions
// (80 cycles each, scaled.h) and about 100 integer ones to align and
// normalise.  Scaling every coefficient by the power of two that its offset
// power carries makes the whole sum one of plain doubles of like size
// (raw_double.h): a term is then 4 integer products (int_mul.h), 4 FP64 sums
// and the rule that drops an operand more than 60 binades below the other.
// Coefficients whose scaled parts leave 2^-900 .. 2^60, or are zero, take the
// ScaledComplex step.
#pragma once

#include "int_mul.h"
#include "raw_double.h"

namespace fx {

FX_HD bool series_part(int biased) { return static_cast<unsigned>(biased - (1023 - 900)) <= 960u; }
FX_HD bool series_parts(const Sc& v, int shift) {
    return is_normal(bexp(v.re)) && is_normal(bexp(v.im)) && series_part(bexp(v.re) + shift)
        && series_part(bexp(v.im) + shift);
}
FX_HD Sc series_scaled(const Sc& v, int shift) { return sc_make(add_exp(v.re, shift), add_exp(v.im, shift), 0); }
FX_HD double unless(std::uint32_t zero, double v) {  // v, or +0 where the mask is set
    return from_hilo(hi_of(v) & static_cast<int>(~zero), lo_of(v) & ~zero);
}

// An offset's factors; a zero part (`none_*` all ones) makes its products zero.
struct SeriesFactors {
    FactorA re, im;
    std::uint32_t none_re, none_im;
};

FX_HD Sc series_times(const Sc& w, const SeriesFactors& u) {
    const FactorB fr = factor_b(w.re), fi = factor_b(w.im);
    const double rr = unless(u.none_re, int_mul_even(u.re, fr)), ii = unless(u.none_im, int_mul_even(u.im, fi));
    const double ri = unless(u.none_im, int_mul_even(u.im, fr)), ir = unless(u.none_re, int_mul_even(u.re, fi));
    return sc_make(rr - ii, ri + ir, 0);
}

// The sum of coefficient(k) offset^(k - 1) over k = 1 .. terms - 1 by Horner,
// terms > 1, and with `WithDerivative` Horner's derivative before its last
// step.
template <bool WithDerivative, typename Load>
FX_HD void series_sum(const Load& coefficient, int terms, const Sc& offset, Sc& value, Sc& poly) {
    int k = terms - 1;
    value = coefficient(k);
    poly = sc_zero();
    const int e = offset.e;
    const bool zr = is_zero(offset.re), zi = is_zero(offset.im);
    const bool fits = static_cast<unsigned>(e + (1 << 24)) <= (2u << 24) && !(zr && zi)
        && (zr || bexp(offset.re) >= 1023 - 100) && (zi || bexp(offset.im) >= 1023 - 100);
    const SeriesFactors u{factor_a(offset.re), factor_a(offset.im), zr ? ~0u : 0u, zi ? ~0u : 0u};
    const int base = -coefficient(1).e;
    while (k > 1) {
        int scale = imin(imax(base, -(1 << 28)), 1 << 28) + (k - 1) * (fits ? e : 0);
        const int enter = imin(imax(sat_add(value.e, scale), -4096), 4096);
        const int enter_poly = imin(imax(sat_add(poly.e, scale + e), -4096), 4096);
        bool raw = fits && series_parts(value, enter);
        bool started = false;
        if constexpr (WithDerivative) {
            started = !sc_is_zero(poly);
            raw = raw && (!started || series_parts(poly, enter_poly));
        }
        if (raw) {
            Sc w = series_scaled(value, enter), v = sc_zero();
            if (started) v = series_scaled(poly, enter_poly);
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
            for (;;) {
                const Sc c = coefficient(k - 1);
                const int shift = imin(imax(sat_add(c.e, scale - e), -4096), 4096);
                if (!series_parts(c, shift)) break;
                if constexpr (WithDerivative) {
                    v = started ? add_cut(series_times(v, u), w) : w;
                    started = true;
                }
                w = add_cut(series_times(w, u), series_scaled(c, shift));
                scale -= e;
                --k;
                if (k <= 1 || !series_parts(w, 0)) break;
                if constexpr (WithDerivative) {
                    if (!series_parts(v, 0)) break;
                }
            }
            // Back to the normal form: v's scale is the one before the last
            // offset power, which its next product brings in.
            value = sc_make(w.re, w.im, -scale);
            sc_normalize(value);
            if constexpr (WithDerivative) {
                if (started) {
                    poly = sc_make(v.re, v.im, -scale - e);
                    sc_normalize(poly);
                }
            }
        }
        if (k <= 1) break;
        const Sc before = value;
        value = sc_add(sc_mul(value, offset), coefficient(k - 1));
        if constexpr (WithDerivative) poly = sc_add(sc_mul(poly, offset), before);
        --k;
    }
}

}  // namespace fx
