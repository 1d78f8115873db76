"""The burning ship where a part of Z + d is exactly zero.

A step takes its folded form where a part of Z + d lies on the other side of
zero than Z; zero counts with the positive side (alternate_delta_step,
renderer.cpp:11933-12034).  Both forms have the same value and round
differently, so a row of pixels on the real axis tells them apart.  The rule
is compared with the sign of the sum on the CPU, and rendered points with the
plain definition in Python floats (one IEEE operation per FloatExp one, exact
while no exponent leaves the double range): iterations and the escape norms
bit for bit.
"""

from __future__ import annotations

import math
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fractal-audio-viz_gb300", "csrc")

DRIVER = r"""
#include "raw_double.h"
#include <cmath>
#include <cstdio>
#include <random>
int main() {
    std::mt19937_64 rng(5);
    long bad = 0, crossed = 0, zeros = 0;
    for (int n = 0; n < 2000000; ++n) {
        const int e = -390 + static_cast<int>(rng() % 400);
        double z = std::ldexp(0.5 + 0.5 * static_cast<double>(rng() >> 12) / 4503599627370496.0, e);
        if (rng() & 1) z = -z;
        double d = -z;
        switch (rng() % 6) {
            case 0: break;
            case 1: d = std::nextafter(-z, -2 * z); break;
            case 2: d = std::nextafter(-z, 0.0); break;
            case 3: d = std::ldexp(-z, static_cast<int>(rng() % 5) - 2); break;
            case 4: d = z; break;
            default: d = (rng() & 1) ? 0.0 : -0.0;
        }
        const double sum = z + d;  // exact sign: no gradual underflow in this range
        const bool want = (z >= 0.0) != (sum >= 0.0);
        if (fx::folds(z, d) != want) ++bad;
        crossed += want;
        zeros += sum == 0.0;
    }
    std::printf("bad %ld of %ld crossings, %ld zero sums\n", bad, crossed, zeros);
    return bad != 0 || crossed == 0 || zeros == 0;
}
"""


def test_crossing_rule_is_the_sign_of_the_sum(tmp_path):
    source, binary = tmp_path / "driver.cpp", tmp_path / "driver"
    source.write_text(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I" + CSRC, str(source), "-o", str(binary)],
                   check=True)
    done = subprocess.run([str(binary)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout


def _nearest(fixed: int, bits: int) -> float:
    """fixed * 2^-bits rounded to a double."""
    return fixed / (1 << bits)


def _ship_orbit(re: str, im: str, cap: int):
    """Reference orbit (doubles) and |Z|^2 - 4 (double) from fixed point."""
    from fractions import Fraction
    bits = 400
    one = 1 << bits
    cr, ci = (int(Fraction(t) * one) for t in (re, im))
    zr = zi = 0
    orbit, margins = [], []
    for _ in range(cap + 1):
        norm = zr * zr + zi * zi
        orbit.append((_nearest(zr, bits), _nearest(zi, bits)))
        margins.append(_nearest(norm - (4 << (2 * bits)), 2 * bits))
        if norm > 4 << (2 * bits):
            break
        zr, zi = ((zr * zr - zi * zi) >> bits) + cr, ((2 * abs(zr * zi)) >> bits) + ci
    return orbit, margins


def _shared(v):  # shared exponent
    return max(math.frexp(v[0])[1] if v[0] else -5000, math.frexp(v[1])[1] if v[1] else -5000)


def _add(a, b):
    """A ScaledComplex sum: an operand 60 binades below the other is dropped."""
    if a == (0.0, 0.0):
        return b
    if b == (0.0, 0.0):
        return a
    apart = _shared(a) - _shared(b)
    return a if apart > 60 else (b if apart < -60 else (a[0] + b[0], a[1] + b[1]))


def _ship_point(orbit, margins, dc, cap):
    """(iterations, |z|^2 at the escape, |z|^2 before it), or None."""
    c, d = orbit[1], dc
    total = _add(c, d)
    for it in range(1, cap):
        (zr, zi), (dr, di) = orbit[it], d
        tr, ti = zr + dr, zi + di
        if (zr >= 0.0) != (tr >= 0.0) or (zi >= 0.0) != (ti >= 0.0):
            nr = (tr * tr - ti * ti) + ((c[0] - orbit[it + 1][0]) + dc[0])
            ni = 2.0 * (abs(tr) * abs(ti)) + ((c[1] - orbit[it + 1][1]) + dc[1])
        else:
            rs, cs = (-1.0 if zr < 0.0 else 1.0), (-1.0 if zi < 0.0 else 1.0)
            ar, ai = abs(zr), abs(zi)
            nr = (2.0 * rs * (ar * dr) - 2.0 * cs * (ai * di)) + (dr * dr - di * di) + dc[0]
            ni = (2.0 * cs * (ar * di) + 2.0 * rs * (ai * dr)) + 2.0 * rs * cs * (dr * di) + dc[1]
        d = (nr, ni)
        zr, zi = orbit[it + 1]
        before, total = total, _add((zr, zi), d)
        if (margins[it + 1] + 2.0 * (zr * nr + zi * ni)) + (nr * nr + ni * ni) > 0.0:
            return it + 1, total[0] * total[0] + total[1] * total[1], before[0] * before[0] + before[1] * before[1]
    return None


@pytest.mark.gpu
@pytest.mark.parametrize("re", ["-1.5", "-1.62", "-1.9"])
@pytest.mark.parametrize("im", ["4.375e-14", "-4.375e-14"])
def test_points_on_the_real_axis(package, product, re, im):
    native = package.native
    orbit, margins = _ship_orbit(re, im, 300)
    zoom, cap, count = b"1e12", len(orbit) - 2, 1000  # before the reference itself escapes
    rng = np.random.default_rng(17)
    real = 0.26 - float(re) + rng.uniform(0.0, 1.0, count) * np.exp2(-rng.integers(0, 6, count))
    imag = np.full(count, -float(im))
    imag[::5] *= 1.0 + 2.0 ** -52  # and one step beside the axis
    options = native.RenderOptions(disable_bla=1, disable_cycle=1)
    handle = native.create_reference(product, re, im, zoom, cap, 256, 8, formula="burning-ship", options=options)
    try:
        _, planes = native.render_points(product, handle, zoom, real, imag, np.zeros(count, dtype=np.int32), cap,
                                         options=options, planes=True)
    finally:
        product.fractal_destroy_reference(handle)
    want = [_ship_point(orbit, margins, (float(x), float(y)), cap) for x, y in zip(real, imag)]
    assert sum(w is not None for w in want) > count // 2
    np.testing.assert_array_equal(planes["orbit_iteration"], [cap if w is None else w[0] - 1 for w in want])
    np.testing.assert_array_equal(planes["test1"], [0.0 if w is None else w[1] for w in want])
    np.testing.assert_array_equal(planes["test2"], [0.0 if w is None else w[2] for w in want])
