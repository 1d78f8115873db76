// Extended-exponent arithmetic shared by the host table builders and the
// plain FP64 device kernels.
//
// Semantics follow the reference's FloatExp / ScaledComplex / ScaledNorm
// (renderer.cpp:7532-7824 and 8190-8475): a double mantissa normalised to
// [0.5, 1) with an int exponent, a complex pair sharing one exponent, the
// same one-shift fast paths, the same 60-exponent cut-off in aligned sums
// and the same comparison rules.  Every operation is written so that it
// performs the same IEEE-754 double operations in the same order as the
// reference release build, which has no fused multiply-add: device code that
// includes this header is compiled with --fmad=false and host code with
// -ffp-contract=off.  The frexp/ldexp replacements below are exact
// bit-level operations with one correctly rounded step for subnormal
// results, i.e. the same values glibc's frexp/scalbn return.
//
// What bounds the kernels that use it is the FP64 pipe: one warp instruction
// takes it 80 cycles of an SM sub-partition on GB300 (measured with
// dependent-free chains of DADD, DMUL, DFMA and DSETP alike), against 1 to 2
// for an integer instruction, and both run side by side.  So an FP64
// instruction is spent only where a sum or product of two full mantissas is
// rounded.  Zero and range tests, comparisons, sign changes and every
// multiplication by a power of two work on the bit patterns, and the rare
// operands those rules do not cover (subnormal, infinite, NaN) go to
// out-of-line general paths.  A complex product with its normalisation then
// takes 6 FP64 instructions where the comparisons and halvings made it 18.
// These rules alone took a 640x360 plain field at 1e30 from 3.10 to 0.98 ms and
// an 853x480 burning-ship field with planes at 1e40 from 106 to 39 ms.
#pragma once

#include <cstdint>
#include <climits>
#include <cmath>

#ifdef __CUDACC__
#define FX_HD __host__ __device__ __forceinline__
#define FX_HD_SLOW static __host__ __device__ __noinline__
#else
#define FX_HD inline
#define FX_HD_SLOW inline
#endif
// The larger operations: out of line where the including file defines
// FX_OUTLINE.  Kernels that inline dozens of them outgrow the instruction
// cache: 26 of 33 cycles per instruction went to instruction fetch in the
// alternate queue.
#ifdef FX_OUTLINE
#define FX_OP FX_HD_SLOW
#else
#define FX_OP FX_HD
#endif

namespace fx {

FX_HD std::uint64_t bits_of(double v) {
#ifdef __CUDA_ARCH__
    return static_cast<std::uint64_t>(__double_as_longlong(v));
#else
    std::uint64_t b;
    __builtin_memcpy(&b, &v, sizeof b);
    return b;
#endif
}

FX_HD double from_bits(std::uint64_t b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double(static_cast<long long>(b));
#else
    double v;
    __builtin_memcpy(&v, &b, sizeof v);
    return v;
#endif
}

// The high word (sign, exponent, top of the mantissa) and the low word.
// Register moves in PTX: with the word intrinsics (__double2hiint and the
// like) CUDA 13.0 lost the low word where fe_from takes a product.
FX_HD int hi_of(double v) {
#ifdef __CUDA_ARCH__
    int lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(v));
    (void)lo;
    return hi;
#else
    return static_cast<int>(bits_of(v) >> 32);
#endif
}

FX_HD unsigned lo_of(double v) {
#ifdef __CUDA_ARCH__
    unsigned lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(v));
    (void)hi;
    return lo;
#else
    return static_cast<unsigned>(bits_of(v));
#endif
}

FX_HD double from_hilo(int hi, unsigned lo) {
#ifdef __CUDA_ARCH__
    double v;
    asm("mov.b64 %0, {%1, %2};" : "=d"(v) : "r"(lo), "r"(hi));
    return v;
#else
    return from_bits((static_cast<std::uint64_t>(static_cast<std::uint32_t>(hi)) << 32) | lo);
#endif
}

FX_HD bool is_finite(double v) { return (hi_of(v) & 0x7ff00000) != 0x7ff00000; }
FX_HD bool is_nan(double v) { return (bits_of(v) & 0x7fffffffffffffffull) > 0x7ff0000000000000ull; }
FX_HD bool is_zero(double v) { return ((hi_of(v) & 0x7fffffff) | lo_of(v)) == 0; }
FX_HD double fabs_(double v) { return from_hilo(hi_of(v) & 0x7fffffff, lo_of(v)); }
FX_HD double neg_(double v) { return from_hilo(hi_of(v) ^ static_cast<int>(0x80000000u), lo_of(v)); }
FX_HD double copysign_(double mag, double sign) {
    return from_bits((bits_of(mag) & 0x7fffffffffffffffull) | (bits_of(sign) & 0x8000000000000000ull));
}
FX_HD int imax(int a, int b) { return a > b ? a : b; }
FX_HD int imin(int a, int b) { return a < b ? a : b; }
FX_HD double dmax(double a, double b) { return a < b ? b : a; }

// Biased exponent; 0 marks zeros and subnormals, 0x7ff infinities and NaN.
FX_HD int bexp(double v) { return (hi_of(v) >> 20) & 0x7ff; }
FX_HD bool is_normal(int be) { return static_cast<unsigned>(be - 1) < 2046u; }
// v * 2^k for a normal v whose result is normal: exact.
FX_HD double add_exp(double v, int k) { return from_hilo(hi_of(v) + (k << 20), lo_of(v)); }

// (a > b) - (a < b) for finite a and b that are not both zero: sign and
// magnitude order of the bit patterns.
FX_HD int order_of(double a, double b) {
    const long long x = static_cast<long long>(bits_of(a)), y = static_cast<long long>(bits_of(b));
    const long long r = (x & y) < 0 ? y - x : (x > y ? 1 : (x < y ? -1 : 0));
    return r > 0 ? 1 : (r < 0 ? -1 : 0);
}

// Exponent sum, saturated to the int range.
FX_HD int sat_add(int a, int b) {
#ifdef __CUDA_ARCH__
    int r;
    asm("add.sat.s32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
#else
    const long long v = static_cast<long long>(a) + b;
    return v > INT_MAX ? INT_MAX : (v < INT_MIN ? INT_MIN : static_cast<int>(v));
#endif
}

// x * 2^n with a single round-to-nearest-even step (glibc scalbn semantics).
FX_HD_SLOW double scale2_general(double x, int n) {
    std::uint64_t b = bits_of(x);
    int be = static_cast<int>((b >> 52) & 0x7ff);
    if (be == 0x7ff || (b << 1) == 0) return x;  // inf, nan, +-0
    if (be == 0) {
        // Subnormal input: lift it into the normal range exactly first.
        x = x * 18014398509481984.0;  // 2^54
        b = bits_of(x);
        be = static_cast<int>((b >> 52) & 0x7ff);
        n -= 54;
    }
    if (n > 4096) n = 4096;
    if (n < -4096) n = -4096;
    const int ne = be + n;
    if (ne >= 1 && ne <= 2046) {
        return from_bits((b & ~(0x7ffull << 52)) | (static_cast<std::uint64_t>(ne) << 52));
    }
    if (ne > 2046) return copysign_(from_bits(0x7ff0000000000000ull), x);
    // Subnormal or zero result: move the value to the smallest normal binade
    // (exact), then apply the remaining power of two in one multiplication,
    // which is the only rounding.
    const double y = from_bits((b & ~(0x7ffull << 52)) | (1ull << 52));
    const int r = ne - 1;  // <= -1
    if (r < -54) return copysign_(0.0, x);
    return y * from_bits(static_cast<std::uint64_t>(1023 + r) << 52);
}

FX_HD double scale2(double x, int n) {
    n = imin(imax(n, -4096), 4096);
    const int be = bexp(x);
    if (is_normal(be) && is_normal(be + n)) return add_exp(x, n);
    if (is_zero(x)) return x;
    return scale2_general(x, n);
}

// A subnormal moved into the normal range: v * 2^54, exact.
FX_HD_SLOW double lift54(double v) { return v * 18014398509481984.0; }

// frexp: mantissa in [0.5, 1) and exponent; zero/inf/nan returned unchanged
// with exponent 0.
FX_HD double split2(double x, int* e) {
    std::uint64_t b = bits_of(x);
    int be = static_cast<int>((b >> 52) & 0x7ff);
    if (be == 0x7ff || (b << 1) == 0) { *e = 0; return x; }
    int bias = 0;
    if (be == 0) {
        x = x * 18014398509481984.0;  // 2^54, exact
        b = bits_of(x);
        be = static_cast<int>((b >> 52) & 0x7ff);
        bias = 54;
    }
    *e = be - 1022 - bias;
    return from_bits((b & ~(0x7ffull << 52)) | (0x3feull << 52));
}

FX_HD int sat_exp(long long v) {
    if (v > static_cast<long long>(INT_MAX)) return INT_MAX;
    if (v < static_cast<long long>(INT_MIN)) return INT_MIN;
    return static_cast<int>(v);
}

// ---------------------------------------------------------------- FloatExp
struct Fe {
    double m;
    int e;
};

FX_HD Fe fe_make(double m, int e) { Fe r; r.m = m; r.e = e; return r; }
FX_HD Fe fe_zero() { return fe_make(0.0, 0); }
FX_HD bool fe_finite(const Fe& a) { return is_finite(a.m); }
FX_HD bool fe_is_zero(const Fe& a) { return is_zero(a.m); }

// FloatExp::from_parts (renderer.cpp:7551-7561).
FX_HD Fe fe_from(double value, int exponent) {
    const int be = bexp(value);
    if (is_normal(be)) return fe_make(add_exp(value, 1022 - be), sat_add(exponent, be - 1022));
    if (is_zero(value) || is_nan(value)) return fe_make(value, 0);
    if (be != 0) return fe_make(value, exponent);  // infinite: frexp's exponent is 0
    const double lifted = lift54(value);
    const int shift = bexp(lifted) - 1022;
    return fe_make(add_exp(lifted, -shift), sat_add(exponent, shift - 54));
}

FX_HD Fe fe_neg(const Fe& a) { return fe_make(neg_(a.m), a.e); }
FX_HD Fe fe_abs(const Fe& a) { return fe_make(fabs_(a.m), a.e); }

// fe_add (renderer.cpp:8197-8235): a sum at or above 1 is halved once, one
// below 0.5 normalised.
FX_OP Fe fe_add(Fe a, Fe b) {
    if (is_zero(a.m)) return b;
    if (is_zero(b.m)) return a;
    const bool swap = b.e > a.e;
    const double hm = swap ? b.m : a.m, lm = swap ? a.m : b.m;
    const int he = swap ? b.e : a.e, le = swap ? a.e : b.e;
    const unsigned diff = static_cast<unsigned>(he) - static_cast<unsigned>(le);
    if (diff > 60u) return fe_make(hm, he);
    const double m = hm + scale2(lm, -static_cast<int>(diff));
    const int be = bexp(m);
    if (!is_normal(be)) return fe_from(m, he);
    const int shift = be >= 1023 ? 1 : be - 1022;
    return fe_make(add_exp(m, -shift), sat_add(he, shift));
}

FX_HD Fe fe_sub(const Fe& a, const Fe& b) { return fe_add(a, fe_neg(b)); }

// Result of a product or quotient: halved once at or above 1, doubled once
// below 0.5 (fe_mul / fe_div, renderer.cpp:8241-8291).  `e` is the exponent
// sum or difference; its saturation matters only for values that no orbit of
// at most 131,072 bits reaches.
FX_HD Fe fe_step(double m, int e) {
    const int be = bexp(m);
    if (be >= 1023) {
        if (be == 0x7ff) return fe_from(m, 0);
        return fe_make(add_exp(m, -1), sat_add(e, 1));
    }
    if (be >= 1022) return fe_make(m, e);
    return fe_make(be > 0 ? add_exp(m, 1) : m * 2.0, sat_add(e, -1));
}

FX_OP Fe fe_mul(Fe a, Fe b) {
    if (is_zero(a.m) || is_zero(b.m)) return fe_zero();
    return fe_step(a.m * b.m, sat_add(a.e, b.e));
}

// fe_mul(a, fe_from(s, 0)) for s = +2 or -2 (`minus`), without the product.
FX_HD Fe fe_twice(const Fe& a, bool minus) {
    if (is_zero(a.m)) return fe_zero();
    const double m = minus ? neg_(a.m) : a.m;
    return is_finite(m) ? fe_make(m, sat_add(a.e, 1)) : fe_make(m, 0);
}

FX_HD Fe fe_mul(const Fe& a, double b) { return fe_mul(a, fe_from(b, 0)); }

// fe_div (renderer.cpp:8272-8291).
FX_OP Fe fe_div(Fe a, Fe b) {
    if (is_zero(a.m)) return fe_zero();
    const double m = a.m / b.m;
    const long long d = static_cast<long long>(a.e) - b.e;
    return fe_step(m, sat_exp(d));
}

FX_HD Fe fe_sqr(const Fe& a) { return fe_mul(a, a); }

// fe_sqrt (renderer.cpp:8297-8315).
FX_HD Fe fe_sqrt(const Fe& a) {
    if (is_zero(a.m)) return a;
    long long e = a.e;
    double m = a.m;
    if (m < 0.0 || !is_finite(m)) return fe_from(sqrt(m), 0);
    if (e % 2 != 0) {
        m *= 2.0;
        --e;
        return fe_make(sqrt(m) * 0.5, sat_exp(e / 2 + 1));
    }
    return fe_make(sqrt(m), sat_exp(e / 2));
}

// fe_compare (renderer.cpp:8317-8340).
FX_HD int fe_cmp(const Fe& a, const Fe& b) {
    if (!fe_finite(a)) return fe_finite(b) ? 1 : 0;
    if (!fe_finite(b)) return -1;
    const bool an = hi_of(a.m) < 0, bn = hi_of(b.m) < 0;
    if (is_zero(a.m)) return is_zero(b.m) ? 0 : -1;
    if (is_zero(b.m)) return an ? -1 : 1;
    if (an != bn) return an ? -1 : 1;
    if (a.e != b.e) return (a.e < b.e) == an ? 1 : -1;
    return order_of(a.m, b.m);
}

// fe_cmp(a, 0) as its callers use it: > 0 and >= 0.
FX_HD bool fe_positive(const Fe& a) { return !fe_finite(a) || (hi_of(a.m) >= 0 && !is_zero(a.m)); }
FX_HD bool fe_at_least_zero(const Fe& a) { return !fe_finite(a) || hi_of(a.m) >= 0 || is_zero(a.m); }

FX_HD Fe fe_min(const Fe& a, const Fe& b) { return fe_cmp(a, b) <= 0 ? a : b; }

struct Fec {
    Fe re;
    Fe im;
};

FX_HD Fec fec_make(const Fe& re, const Fe& im) { Fec r; r.re = re; r.im = im; return r; }
FX_HD Fec fec_add(const Fec& a, const Fec& b) { return fec_make(fe_add(a.re, b.re), fe_add(a.im, b.im)); }
FX_HD Fec fec_sub(const Fec& a, const Fec& b) { return fec_make(fe_sub(a.re, b.re), fe_sub(a.im, b.im)); }
FX_HD Fec fec_mul(const Fec& a, const Fec& b) {
    return fec_make(fe_sub(fe_mul(a.re, b.re), fe_mul(a.im, b.im)),
                    fe_add(fe_mul(a.re, b.im), fe_mul(a.im, b.re)));
}
FX_HD Fec fec_scale(const Fec& a, const Fe& b) { return fec_make(fe_mul(a.re, b), fe_mul(a.im, b)); }
FX_HD Fe fec_norm2(const Fec& a) { return fe_add(fe_sqr(a.re), fe_sqr(a.im)); }
FX_HD bool fec_finite(const Fec& a) { return fe_finite(a.re) && fe_finite(a.im); }

// Escape threshold as FloatExp: 4 (classic) or 1e8 (Kalles high bailout).
FX_HD Fe escape_r2_fe(int mode) { return mode == 1 ? fe_from(1.0e8, 0) : fe_from(4.0, 0); }
FX_HD double escape_r2_d(int mode) { return mode == 1 ? 1.0e8 : 4.0; }

// |R + D|^2 - R_escape^2 in FloatExp (renderer.cpp:8374-8390).
FX_HD Fe fec_escape_margin(const Fec& r, const Fec& d, int mode) {
    const Fe cross = fe_twice(fe_add(fe_mul(r.re, d.re), fe_mul(r.im, d.im)), false);
    const Fe ref_margin = fe_sub(fec_norm2(r), escape_r2_fe(mode));
    return fe_add(fe_add(ref_margin, cross), fec_norm2(d));
}

// ---------------------------------------------------------- ScaledComplex
struct Sc {
    double re;
    double im;
    int e;
};

struct Nrm {
    double m;
    int e;
};

FX_HD Sc sc_make(double re, double im, int e) { Sc r; r.re = re; r.im = im; r.e = e; return r; }
FX_HD Sc sc_zero() { return sc_make(0.0, 0.0, 0); }
FX_HD Sc sc_one() { return sc_make(1.0, 0.0, 0); }
FX_HD bool sc_is_zero(const Sc& a) {
    return (((hi_of(a.re) | hi_of(a.im)) & 0x7fffffff) | lo_of(a.re) | lo_of(a.im)) == 0;
}
FX_HD bool sc_finite(const Sc& a) { return is_finite(a.re) && is_finite(a.im); }
FX_HD Nrm nrm_make(double m, int e) { Nrm r; r.m = m; r.e = e; return r; }

// ScaledComplex::normalize (renderer.cpp:7611-7656).
// The exponent of max(|re|, |im|) as frexp gives it, for parts that are both
// zero or subnormal, or not finite (0: zero, infinite or NaN).  Scalars only
// in and out: passing the pair through memory, by reference or as a struct,
// let the compiler (CUDA 13.0, sm_100 and up) mix up two such pairs.
FX_HD_SLOW int sc_general_shift(double re, double im) {
    const double mag = dmax(fabs_(re), fabs_(im));
    int shift = 0;
    (void)split2(mag, &shift);
    return shift;
}

FX_HD void sc_normalize(Sc& v) {
    const int be = imax(bexp(v.re), bexp(v.im));
    int shift = be - 1022;
    if (!is_normal(be)) {
        // A NaN in the imaginary part beside a zero real part clears both, as
        // the reference's magnitude comparison has it.
        if (is_zero(v.re) && (is_zero(v.im) || is_nan(v.im))) {
            v.re = 0.0;
            v.im = 0.0;
            v.e = 0;
            return;
        }
        shift = sc_general_shift(v.re, v.im);
    }
    if (shift == 0) return;
    v.re = scale2(v.re, -shift);
    v.im = scale2(v.im, -shift);
    v.e = sat_add(v.e, shift);
}

// ScaledComplex::from_float_exp (renderer.cpp:7658-7675).
FX_OP Sc sc_from_fe(Fe re, Fe im) {
    if (is_zero(re.m) && is_zero(im.m)) return sc_zero();
    const int common = imax(re.e, im.e);
    const unsigned rd = static_cast<unsigned>(common) - static_cast<unsigned>(re.e);
    const unsigned id = static_cast<unsigned>(common) - static_cast<unsigned>(im.e);
    Sc r = sc_make(rd > 1074u ? 0.0 : scale2(re.m, -static_cast<int>(rd)),
                   id > 1074u ? 0.0 : scale2(im.m, -static_cast<int>(id)), common);
    sc_normalize(r);
    return r;
}

// sc_add (renderer.cpp:7678-7698).
FX_OP Sc sc_add(Sc a, Sc b) {
    if (sc_is_zero(a)) return b;
    if (sc_is_zero(b)) return a;
    const bool swap = b.e > a.e;
    const Sc hi = sc_make(swap ? b.re : a.re, swap ? b.im : a.im, swap ? b.e : a.e);
    const Sc lo = sc_make(swap ? a.re : b.re, swap ? a.im : b.im, swap ? a.e : b.e);
    const unsigned diff = static_cast<unsigned>(hi.e) - static_cast<unsigned>(lo.e);
    if (diff > 60u) return hi;
    const int d = static_cast<int>(diff);
    Sc r = sc_make(hi.re + scale2(lo.re, -d), hi.im + scale2(lo.im, -d), hi.e);
    sc_normalize(r);
    return r;
}

FX_HD Sc sc_neg(const Sc& a) { return sc_make(neg_(a.re), neg_(a.im), a.e); }
FX_HD Sc sc_conj(const Sc& a) { return sc_make(a.re, neg_(a.im), a.e); }
FX_HD Sc sc_sub(const Sc& a, const Sc& b) { return sc_add(a, sc_neg(b)); }

// sc_mul (renderer.cpp:7712-7722).
FX_OP Sc sc_mul(Sc a, Sc b) {
    if (sc_is_zero(a) || sc_is_zero(b)) return sc_zero();
    Sc r = sc_make(a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re, sat_add(a.e, b.e));
    sc_normalize(r);
    return r;
}

// sc_mul(a, a): the two equal cross products are one product, doubled.
FX_OP Sc sc_sqr(Sc a) {
    if (sc_is_zero(a)) return sc_zero();
    const double cross = a.re * a.im;
    Sc r = sc_make(a.re * a.re - a.im * a.im, is_normal(bexp(cross)) ? add_exp(cross, 1) : cross + cross,
                   sat_add(a.e, a.e));
    sc_normalize(r);
    return r;
}

// sc_double (renderer.cpp:7724-7733): exact doubling through the exponent.
FX_HD Sc sc_twice(const Sc& a) {
    if (sc_is_zero(a)) return sc_zero();
    return sc_make(a.re, a.im, sat_add(a.e, 1));
}

// sc_norm_squared (renderer.cpp:7740-7770).
FX_OP Nrm sc_norm2(Sc a) {
    const double inf = from_bits(0x7ff0000000000000ull);
    if (!sc_finite(a)) return nrm_make(inf, INT_MAX);
    const double n = a.re * a.re + a.im * a.im;
    if (is_zero(n)) return nrm_make(0.0, 0);
    const int be = bexp(n);
    if (be == 0x7ff) return nrm_make(inf, INT_MAX);
    // One doubling or halving into [0.5, 1), as the reference.
    const int shift = be >= 1023 ? 1 : (be < 1022 ? -1 : 0);
    const long long e = 2LL * a.e + shift;
    if (e > INT_MAX && shift >= 0) return nrm_make(inf, INT_MAX);
    if (e < INT_MIN && shift <= 0) return nrm_make(0.0, 0);
    return nrm_make(be > 0 ? add_exp(n, -shift) : n * 2.0, static_cast<int>(e));
}

// sc_compare_norm (renderer.cpp:7772-7781).
FX_HD int nrm_cmp(const Nrm& a, const Nrm& b) {
    if (!is_finite(a.m)) return is_finite(b.m) ? 1 : 0;
    if (!is_finite(b.m)) return -1;
    if (is_zero(a.m)) return is_zero(b.m) ? 0 : -1;
    if (is_zero(b.m)) return hi_of(a.m) >= 0 ? 1 : -1;
    if (a.e != b.e) return a.e < b.e ? -1 : 1;
    return order_of(a.m, b.m);
}

FX_HD bool nrm_outside(const Nrm& n, int mode) {
    const Fe t = escape_r2_fe(mode);
    return nrm_cmp(n, nrm_make(t.m, t.e)) > 0;
}

// m * 2^e truncated to a float without the FP64 pipe: relative error below
// 2^-23, 0 below the float range, infinity above it (for |e| < 2^20).
FX_HD float float_of(double m, int e) {
    const int h = hi_of(m);
    const int fe = ((h >> 20) & 0x7ff) - 896 + e;
    std::uint32_t b = static_cast<std::uint32_t>(h) & 0x80000000u;
    if (fe >= 255) {
        b |= 0x7f800000u;
    } else if (fe > 0) {
        b |= (static_cast<std::uint32_t>(fe) << 23) | ((static_cast<std::uint32_t>(h) << 3) & 0x7fffffu) | (lo_of(m) >> 29);
    }
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float v;
    __builtin_memcpy(&v, &b, sizeof v);
    return v;
#endif
}

FX_HD double sc_re_d(const Sc& a) { return scale2(a.re, a.e); }
FX_HD double sc_im_d(const Sc& a) { return scale2(a.im, a.e); }

// scaled_norm_to_double / scaled_norm_from_double (renderer.cpp:7801-7823).
FX_HD double nrm_to_d(const Nrm& n) {
    if (is_zero(n.m)) return 0.0;
    const double dbl_max = 1.7976931348623157e308;
    if (!is_finite(n.m)) return dbl_max;
    const double v = scale2(n.m, n.e);
    return is_finite(v) ? dmax(0.0, v) : dbl_max;
}

FX_HD Nrm nrm_from_d(double v) {
    if (!(v > 0.0) || !is_finite(v)) {
        return v > 0.0 ? nrm_make(1.7976931348623157e308, 0) : nrm_make(0.0, 0);
    }
    int e = 0;
    const double m = split2(v, &e);
    return nrm_make(m, e);
}

FX_HD Fe sc_part_fe(const Sc& v, bool imaginary) { return fe_from(imaginary ? v.im : v.re, v.e); }
FX_HD Fec sc_to_fec(const Sc& v) { return fec_make(sc_part_fe(v, false), sc_part_fe(v, true)); }

// Signed escape margin |Z + d|^2 - R^2 (renderer.cpp:8400-8425).
FX_HD Fe sc_escape_margin(const Sc& ref, const Sc& d, int mode) {
    return fec_escape_margin(sc_to_fec(ref), sc_to_fec(d), mode);
}

// sc_norm_squared_with_delta given the margin (renderer.cpp:8445-8453).
FX_HD Nrm nrm_from_margin(const Fe& margin, int mode) {
    const Fe n = fe_add(escape_r2_fe(mode), margin);
    return nrm_make(n.m, n.e);
}

}  // namespace fx
