"""CPU: the image series summed on scaled doubles against Horner's rule.

csrc/raw_series.h scales the coefficients by the powers of two that the
offset carries and sums plain doubles.  Value and derivative are compared,
bit for bit, with the ScaledComplex steps (renderer.cpp:8594-8639) on seeded
series: falling, growing and ragged coefficients of full and of few bits,
real ones, operands about 60 binades apart, offsets on an axis, far smaller
than the radius, of extreme exponents, and zero.  Host build of the device's
code.
"""

from __future__ import annotations

import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fractal-audio-viz_gb300", "csrc")

DRIVER = r"""
#include "raw_series.h"
#include <cstdio>
#include <cstdlib>
#include <random>
using namespace fx;

static std::mt19937_64 rng(20261);
static int pick(int n) { return static_cast<int>(rng() % static_cast<unsigned>(n)); }
static double mantissa(int kind) {
    double m = 1.0 + static_cast<double>(rng() >> 12) * 0x1p-52;
    if (kind == 1) m = 1.0 + pick(8) * 0.125;          // few bits: ties
    if (kind == 2) m = 1.0 + pick(1 << 26) * 0x1p-26;
    return (rng() & 1 ? -m : m) * 0.5;
}
static bool same(const Sc& a, const Sc& b) {
    return bits_of(a.re) == bits_of(b.re) && bits_of(a.im) == bits_of(b.im) && a.e == b.e;
}
int main(int argc, char** argv) {
    const int count = std::atoi(argv[1]), shape = std::atoi(argv[2]);
    long long bad = 0;
    for (int n = 0; n < count; ++n) {
        const int terms = 2 + pick(31), kind = pick(3);
        int e = -pick(400);
        if (shape == 3) e = -100000 - pick(100000);
        if (shape == 4) e = pick(2) ? -(1 << 25) : 40;
        const int fall = shape == 1 ? -1 : (shape == 2 ? 30 : pick(12));  // binades per term below the radius
        Sc c[33], offset = sc_make(mantissa(kind), mantissa(pick(3)), e);
        offset.re = add_exp(offset.re, -pick(6) * pick(25));
        if (pick(8) == 0) offset.re = pick(2) ? 0.0 : -0.0;
        if (pick(8) == 0) offset.im = pick(2) ? 0.0 : -0.0;
        sc_normalize(offset);
        for (int k = 0; k < terms; ++k) {
            const int spread = shape == 5 ? pick(130) - 65 : pick(4);
            c[k] = sc_make(mantissa(kind), add_exp(mantissa(kind), -pick(3) * pick(30)), spread - k * (e + fall));
            if (shape == 6) c[k].im = 0.0;
            if (shape == 7 && pick(5) == 0) c[k] = sc_make(0.0, pick(2) ? 0.25 : 0.0, 7);
            sc_normalize(c[k]);
        }
        Sc value = c[terms - 1], poly = sc_zero(), got, slope, plain_got, unused;
        for (int k = terms - 1; k > 1; --k) {
            poly = sc_add(sc_mul(poly, offset), value);
            value = sc_add(sc_mul(value, offset), c[k - 1]);
        }
        const auto load = [&](int k) { return c[k]; };
        series_sum<true>(load, terms, offset, got, slope);
        series_sum<false>(load, terms, offset, plain_got, unused);
        // The sign of a zero part does not reach a field; the rest must match.
        const auto plus = [](Sc v) { return sc_make(v.re + 0.0, v.im + 0.0, v.e); };
        if (!same(plus(got), plus(value)) || !same(plus(plain_got), plus(value)) || !same(plus(slope), plus(poly))) {
            if (bad++ < 3) std::printf("case %d: terms %d e %d got %a %a %d want %a %a %d\n", n, terms, e, got.re,
                                       got.im, got.e, value.re, value.im, value.e);
        }
    }
    std::printf("mismatches %lld\n", bad);
    return bad != 0;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    folder = tmp_path_factory.mktemp("series")
    source, binary = folder / "driver.cpp", folder / "driver"
    source.write_text(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I" + CSRC, str(source), "-o", str(binary)],
                   check=True)
    return str(binary)


@pytest.mark.parametrize("shape", range(8))
def test_series_sum_equals_horner(driver, shape):
    done = subprocess.run([driver, "200000", str(shape)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout
