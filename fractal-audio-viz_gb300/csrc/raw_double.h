// Extended-exponent values held as plain doubles where their range allows.
//
// A FloatExp or ScaledComplex operation (scaled.h) rounds like the IEEE
// double operation on the same values with an unbounded exponent range: the
// mantissas are doubles, powers of two are exact, and a real operand more
// than 60 binades below the other cannot move its rounded sum.  So while
// every operand and result stays in the normal double range, one FP64
// instruction per sum or product gives the same bits without aligning and
// normalising, which took about 30 integer instructions each and, inlined
// at every site, more code than the instruction cache holds (a warp waited
// 21 of 27 cycles for instructions).  Two rules remain:
//   * a ScaledComplex sum drops the whole smaller operand when the shared
//     exponents differ by more than 60 (add_cut);
//   * the sign of a zero may differ (FloatExp products and exact sums give
//     +0): a zero is accepted where it meets a nonzero value next.
// "Raw" below: a ScaledComplex whose exponent word is 0 and whose parts are
// the values themselves, not normalised.
//
// The range is 2^-400 .. 2^10 for deltas, orbit values and parameters (zooms
// to about 1e115), so products of two stay above 2^-906 even after
// cancellation, and 2^-400 .. 2^400 for Jacobian entries, which share one
// exponent and are rescaled.
//
// Measured with the alternate kernels on raw values and their escape tests
// settled in FP32 first: an 853x480 burning-ship field with planes at 1e40 in
// 28.8 ms (39.5 ms with every step aligned and normalised), the mixed 1280x720
// batch in 88 ms (217 ms); with the queue of render_alt.cu and its integer
// products since in 6.3 and 33 ms.
#pragma once

#include "scaled.h"

namespace fx {

constexpr int kRawLow = 1023 - 400;
constexpr unsigned kRawSpan = 410;    // 2^-400 .. 2^10
constexpr unsigned kJacSpan = 800;    // 2^-400 .. 2^400

FX_HD bool raw_part(double v) { return static_cast<unsigned>(bexp(v) - kRawLow) <= kRawSpan; }
FX_HD bool raw_or_zero(double v) { return raw_part(v) || is_zero(v); }
FX_HD bool raw_value(const Sc& v) { return v.e == 0 && raw_part(v.re) && raw_part(v.im); }

// The normal form of a value in either form.
FX_HD Sc normal_form(Sc v) {
    sc_normalize(v);
    return v;
}

// v as a raw value where both parts are in range or zero, else unchanged.
FX_HD Sc to_raw(const Sc& v) {
    const int e = imax(imin(v.e, 2048), -2048);
    const int br = bexp(v.re) + e, bi = bexp(v.im) + e;
    const bool zr = is_zero(v.re), zi = is_zero(v.im);
    const bool fits = (zr || (is_normal(bexp(v.re)) && static_cast<unsigned>(br - kRawLow) <= kRawSpan))
        && (zi || (is_normal(bexp(v.im)) && static_cast<unsigned>(bi - kRawLow) <= kRawSpan));
    if (!fits) return v;
    return sc_make(zr ? v.re : add_exp(v.re, e), zi ? v.im : add_exp(v.im, e), 0);
}

FX_HD double choose(bool first, double a, double b) {
    return from_hilo(first ? hi_of(a) : hi_of(b), first ? lo_of(a) : lo_of(b));
}

// sc_add on raw values (parts normal or zero).
FX_HD Sc add_cut(const Sc& a, const Sc& b) {
    const int diff = imax(bexp(a.re), bexp(a.im)) - imax(bexp(b.re), bexp(b.im));
    const double re = a.re + b.re, im = a.im + b.im;
    return sc_make(diff > 60 ? a.re : choose(diff < -60, b.re, re), diff > 60 ? a.im : choose(diff < -60, b.im, im), 0);
}

// Whether a part z + d of a raw z lies on the other side of zero than z, zero
// counting with the positive side: a positive z that d cancels exactly stays,
// a negative one crosses (a row of pixels on the real axis meets both).
FX_HD bool folds(double z, double d) {
    const std::uint64_t magnitude = 0x7fffffffffffffffull;
    return (hi_of(z) ^ hi_of(d)) < 0
        && (bits_of(d) & magnitude) >= (bits_of(z) & magnitude) + (hi_of(z) >= 0 ? 1u : 0u);
}

FX_HD double twice_raw(double v) { return is_zero(v) ? v : add_exp(v, 1); }

FX_HD double flip(double v, bool negate) {
    return from_hilo(hi_of(v) ^ (negate ? static_cast<int>(0x80000000u) : 0), lo_of(v));
}

}  // namespace fx
