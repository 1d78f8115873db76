"""CPU: the extended-exponent arithmetic of csrc/scaled.h against its plain
definition.

scaled.h decides zero tests, comparisons, normalisations and powers of two on
bit patterns.  Here every operation is compared, bit for bit, with the
definition written with frexp, ldexp and floating-point comparisons
(renderer.cpp:7532-7824, 8190-8475), on seeded operands: random, sparse and
nearly equal mantissas, zeros of both signs, subnormals, infinities and NaN,
exponents near and far apart.  Host build; the device build runs the same
code and is compared with the reference's fields by test_gpu_parity.py.  The
raw-double sums of csrc/raw_double.h are compared with the same definitions,
and the integer products of csrc/int_mul.h with the FP64 product.
"""

from __future__ import annotations

import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fractal-audio-viz_gb300", "csrc")

DRIVER = r"""
#include "int_mul.h"
#include "raw_double.h"
#include "scaled.h"
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
using namespace fx;
using u64 = std::uint64_t;

// The definitions.
static int sat(long long v) { return v > INT_MAX ? INT_MAX : (v < INT_MIN ? INT_MIN : (int)v); }
static Fe d_from(double v, int e) {
    if (v == 0.0 || v != v) return fe_make(v, 0);
    int s = 0;
    double m = std::isinf(v) ? v : std::frexp(v, &s);
    return fe_make(m, sat((long long)e + s));
}
static Fe d_add(Fe a, Fe b) {
    if (a.m == 0.0) return b;
    if (b.m == 0.0) return a;
    if (b.e > a.e) { Fe t = a; a = b; b = t; }
    const long long diff = (long long)a.e - b.e;
    if (diff > 60) return a;
    const double m = a.m + std::ldexp(b.m, -(int)diff);
    if (m == 0.0 || !std::isfinite(m)) return d_from(m, a.e);
    if (std::fabs(m) >= 1.0) return fe_make(m * 0.5, sat((long long)a.e + 1));
    if (std::fabs(m) >= 0.5) return fe_make(m, a.e);
    return d_from(m, a.e);
}
static Fe d_step(double m, long long e) {
    if (!std::isfinite(m)) return d_from(m, 0);
    if (std::fabs(m) >= 1.0) return fe_make(m * 0.5, sat(e + 1));
    if (std::fabs(m) < 0.5) return fe_make(m * 2.0, sat(e - 1));
    return fe_make(m, sat(e));
}
static Fe d_mul(Fe a, Fe b) { return a.m == 0.0 || b.m == 0.0 ? fe_zero() : d_step(a.m * b.m, (long long)a.e + b.e); }
static Fe d_div(Fe a, Fe b) { return a.m == 0.0 ? fe_zero() : d_step(a.m / b.m, (long long)a.e - b.e); }
static int d_cmp(Fe a, Fe b) {
    if (!std::isfinite(a.m)) return std::isfinite(b.m) ? 1 : 0;
    if (!std::isfinite(b.m)) return -1;
    if (a.m == 0.0) return b.m == 0.0 ? 0 : -1;
    if (b.m == 0.0) return a.m > 0.0 ? 1 : -1;
    if ((a.m < 0.0) != (b.m < 0.0)) return a.m < 0.0 ? -1 : 1;
    if (a.e != b.e) return (a.e < b.e) == (a.m < 0.0) ? 1 : -1;
    return (a.m > b.m) - (a.m < b.m);
}
static void d_normalize(Sc& v) {
    const double mag = std::fabs(v.re) < std::fabs(v.im) ? std::fabs(v.im) : std::fabs(v.re);
    if (mag == 0.0) { v = sc_zero(); return; }
    if (!std::isfinite(mag)) return;
    int s = 0;
    std::frexp(mag, &s);
    v.re = std::ldexp(v.re, -s);
    v.im = std::ldexp(v.im, -s);
    v.e = sat((long long)v.e + s);
}
static bool d_zero(Sc a) { return a.re == 0.0 && a.im == 0.0; }
static Sc d_scadd(Sc a, Sc b) {
    if (d_zero(a)) return b;
    if (d_zero(b)) return a;
    if (b.e > a.e) { Sc t = a; a = b; b = t; }
    const long long diff = (long long)a.e - b.e;
    if (diff > 60) return a;
    Sc r = sc_make(a.re + std::ldexp(b.re, -(int)diff), a.im + std::ldexp(b.im, -(int)diff), a.e);
    d_normalize(r);
    return r;
}
static Sc d_scmul(Sc a, Sc b) {
    if (d_zero(a) || d_zero(b)) return sc_zero();
    Sc r = sc_make(a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re, sat((long long)a.e + b.e));
    d_normalize(r);
    return r;
}
static Nrm d_norm2(Sc a) {
    if (!std::isfinite(a.re) || !std::isfinite(a.im)) return nrm_make(INFINITY, INT_MAX);
    const double n = a.re * a.re + a.im * a.im;
    if (n == 0.0) return nrm_make(0.0, 0);
    if (!std::isfinite(n)) return nrm_make(INFINITY, INT_MAX);
    const Fe r = d_step(n, 2LL * a.e);
    return nrm_make(r.m, r.e);
}
static int d_ncmp(Nrm a, Nrm b) {
    if (!std::isfinite(a.m)) return std::isfinite(b.m) ? 1 : 0;
    if (!std::isfinite(b.m)) return -1;
    if (a.m == 0.0 || b.m == 0.0) return (a.m > b.m) - (a.m < b.m);
    return a.e != b.e ? (a.e < b.e ? -1 : 1) : (a.m > b.m) - (a.m < b.m);
}
static Sc d_fromfe(Fe re, Fe im) {
    if (re.m == 0.0 && im.m == 0.0) return sc_zero();
    const int c = re.e > im.e ? re.e : im.e;
    const long long rd = (long long)re.e - c, id = (long long)im.e - c;
    Sc r = sc_make(rd < -1074 ? 0.0 : std::ldexp(re.m, (int)rd), id < -1074 ? 0.0 : std::ldexp(im.m, (int)id), c);
    d_normalize(r);
    return r;
}

static std::mt19937_64 g(20240);
static long bad = 0;
static bool same(double a, double b) { return (a != a && b != b) || !std::memcmp(&a, &b, 8); }
static void check(const char* what, bool ok) { if (!ok && bad++ < 10) std::printf("%s\n", what); }
static void eq(const char* w, Fe a, Fe b) { check(w, same(a.m, b.m) && a.e == b.e); }
static void eq(const char* w, Nrm a, Nrm b) { check(w, same(a.m, b.m) && a.e == b.e); }
static void eq(const char* w, Sc a, Sc b) { check(w, same(a.re, b.re) && same(a.im, b.im) && a.e == b.e); }
static double mant() {
    u64 m = g();
    if (g() % 4 == 0) m &= ~((1ull << (g() % 52)) - 1);
    if (g() % 16 == 0) m |= (1ull << (g() % 52)) - 1;
    return from_bits((m & 0x800fffffffffffffull) | (1022ull << 52));
}
static double any() {
    switch (g() % 12) {
        case 0: return 0.0;
        case 1: return -0.0;
        case 2: return from_bits(0x7ff0000000000000ull | (g() & (1ull << 63)));
        case 3: return from_bits(0x7ff8000000000000ull);
        case 4: return from_bits(g() & 0x800fffffffffffffull);
        case 5: return from_bits(g());
        default: return mant();
    }
}
static int base = 0;
static int near_e() { return g() % 4 ? base + (int)(g() % 140) - 70 : base + (int)(g() % 6000) - 3000; }
static Fe real() {
    const double m = g() % 12 ? mant() : any();
    if (m == 0.0 || m != m) return fe_make(m, 0);
    return std::isinf(m) ? fe_make(m, near_e()) : fe_make(std::fabs(m) >= 0.5 && std::fabs(m) < 1.0 ? m : mant(), near_e());
}
static Sc pair() {
    double a = mant(), b = mant();
    const int k = g() % 9;
    if (k == 0 || k == 2) a = 0.0;
    if (k == 1 || k == 2) b = 0.0;
    if (k == 3) a = std::ldexp(a, -(int)(g() % 1100));
    if (k == 4) b = std::ldexp(b, -(int)(g() % 1100));
    if (g() % 40 == 0) a = any();
    if (g() % 40 == 0) b = any();
    return sc_make(a, b, near_e());
}
int main(int, char** argv) {
    const long rounds = std::atol(argv[1]);
    for (long i = 0; i < rounds; ++i) {
        base = (int)(g() % 2000000) - 1000000;
        Fe a = real(), b = real();
        if (g() % 3 == 0) { b = a; if (g() % 2) b.m = -b.m; b.m = from_bits(bits_of(b.m) ^ (is_finite(b.m) ? g() & 3 : 0)); }
        eq("fe_add", fe_add(a, b), d_add(a, b));
        eq("fe_sub", fe_sub(a, b), d_add(a, fe_make(-b.m, b.e)));
        eq("fe_mul", fe_mul(a, b), d_mul(a, b));
        eq("fe_div", fe_div(a, b), d_div(a, b));
        eq("fe_twice", fe_twice(a, false), d_mul(a, d_from(2.0, 0)));
        eq("fe_twice minus", fe_twice(a, true), d_mul(a, d_from(-2.0, 0)));
        check("fe_cmp", fe_cmp(a, b) == d_cmp(a, b));
        check("fe_positive", fe_positive(a) == (d_cmp(a, fe_zero()) > 0));
        check("fe_at_least_zero", fe_at_least_zero(a) == (d_cmp(a, fe_zero()) >= 0));
        const double v = any();
        const int e = near_e(), n = (int)(g() % 2400) - 1200;
        eq("fe_from", fe_from(v, e), d_from(v, e));
        check("scale2", same(scale2(v, n), std::ldexp(v, n)));
        Sc s = pair(), t = pair();
        if (g() % 4 == 0) { t = s; t.re = -t.re; if (g() % 2) t.im = -t.im; }
        eq("sc_add", sc_add(s, t), d_scadd(s, t));
        eq("sc_sub", sc_sub(s, t), d_scadd(s, sc_make(-t.re, -t.im, t.e)));
        eq("sc_mul", sc_mul(s, t), d_scmul(s, t));
        eq("sc_norm2", sc_norm2(s), d_norm2(s));
        eq("sc_from_fe", sc_from_fe(a, b), d_fromfe(a, b));
        const Nrm p = d_norm2(s), q = d_norm2(t);
        check("nrm_cmp", nrm_cmp(p, q) == d_ncmp(p, q));
        Sc u = s, w;
        u.re = g() % 30 ? std::ldexp(u.re, (int)(g() % 200) - 100) : any();
        u.im = g() % 30 ? std::ldexp(u.im, (int)(g() % 2200) - 1100) : any();
        w = u;
        sc_normalize(u);
        d_normalize(w);
        eq("sc_normalize", u, w);
        // Raw doubles (raw_double.h): parts in range or zero.
        const int top = (int)(g() % 380) - 375;
        auto part = [&](int e) { return g() % 10 ? std::ldexp(mant(), e - (int)(g() % 20)) : 0.0; };
        Sc x = sc_make(part(top), part(top), 0), y = sc_make(part(top), part(top), 0);
        if (g() % 2) { const int e = -(int)(g() % 130); y.re = std::ldexp(y.re, e < -370 - top ? 0 : e); y.im = std::ldexp(y.im, e < -370 - top ? 0 : e); }
        if (g() % 6 == 0) { y.re = -x.re; if (g() % 2 && !is_zero(x.im)) y.im = from_bits(bits_of(x.im) ^ (g() & 1) ^ (1ull << 63)); }
        Sc xn = x, yn = y, sum = add_cut(x, y);
        d_normalize(xn);
        d_normalize(yn);
        d_normalize(sum);
        Sc want = d_scadd(xn, yn);
        check("add_cut", sum.re == want.re && sum.im == want.im && sum.e == want.e);
        eq("to_raw", normal_form(to_raw(xn)), xn);
        check("to_raw in range", to_raw(xn).e == 0 || d_zero(xn));
        // Integer products: normal operands and result.
        const double fa = std::ldexp(mant(), (int)(g() % 800) - 400), fb = std::ldexp(mant(), (int)(g() % 800) - 400);
        std::uint32_t low = ~0u;
        const double product = int_mul(factor_a(fa), factor_b(fb), low);
        check("int_mul", low == 0 || same(product, fa * fb));
        check("int_mul_even", same(int_mul_even(factor_a(fa), factor_b(fb)), fa * fb));
        // Products of short mantissas: exact ones and ties.
        const int bits = (int)(g() % 30) + 1;
        const double ga = (double)(2 * (g() % (1ull << bits)) + 1), gb = (double)(2 * (g() % (1ull << (53 - bits))) + 1);
        check("int_mul_even tie", same(int_mul_even(factor_a(ga), factor_b(gb)), ga * gb));
        if (is_finite(s.re) && is_finite(s.im)) { Sc n = s; d_normalize(n); eq("to_raw any", normal_form(to_raw(n)), n); }
    }
    std::printf("bad %ld\n", bad);
    return bad ? 1 : 0;
}
"""

def test_scaled_arithmetic_matches_its_definition(tmp_path):
    source = tmp_path / "driver.cpp"
    source.write_text(DRIVER)
    binary = tmp_path / "driver"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I" + CSRC, str(source), "-o", str(binary)],
                   check=True)
    done = subprocess.run([str(binary), "2000000"], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout
    assert done.stdout.strip() == "bad 0"
