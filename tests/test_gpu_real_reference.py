"""GPU: references on the real axis, whose orbits have zero parts.

Points around such references equal the plain definition in Python floats
(alternate_delta_step, renderer.cpp:11933-12034; one IEEE operation per scaled
one while no exponent leaves the double range): iterations and the escape
norms bit for bit.  Mandelbrot fields equal the oracle's.  And a reference on
the axis does not hold a field up: the same view of a Julia set with its
centre moved by 1e-4 of its height, off the axis, makes steps with the same
sums and as many products.
"""

from __future__ import annotations

import numpy as np
import pytest

from .test_axis_crossing import _add, _ship_orbit, _ship_point

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _real_orbit(z: float, c: float, cap: int):
    """z <- z^2 + c for dyadic start and parameter, exact, as doubles, and
    |z|^2 - 4; both maps are this one on the axis."""
    from fractions import Fraction
    bits = 400
    one = 1 << bits
    z, c = int(Fraction(z) * one), int(Fraction(c) * one)
    orbit, margins = [], []
    for _ in range(cap + 2):
        orbit.append((z / one, 0.0))
        margins.append((z * z - (4 << (2 * bits))) / (1 << (2 * bits)))
        z = ((z * z) >> bits) + c
    return orbit, margins


def _twice(v):
    return 2.0 * v[0], 2.0 * v[1]


def _mul(a, b):
    return a[0] * b[0] - a[1] * b[1], a[0] * b[1] + a[1] * b[0]


def _point(formula, orbit, margins, dc, cap):
    it = 0 if formula == "julia" else 1
    d = dc
    total = _add(orbit[it], d)
    while it < cap:
        z = orbit[it]
        if formula == "tricorn":
            zc, conj = (z[0], -z[1]), (d[0], -d[1])
            d = _add(_twice(_mul(zc, conj)), _add(_mul(conj, conj), dc))
        else:
            d = _add(_twice(_mul(z, d)), _mul(d, d))
        it += 1
        (zr, zi), (nr, ni) = orbit[it], d
        before, total = total, _add((zr, zi), d)
        if (margins[it] + 2.0 * (zr * nr + zi * ni)) + (nr * nr + ni * ni) > 0.0:
            return it, total[0] * total[0] + total[1] * total[1], before[0] * before[0] + before[1] * before[1]
    return None


@pytest.mark.parametrize("formula,re", [("burning-ship", "-1.5"), ("burning-ship", "-1.75"), ("burning-ship", "0.25"),
                                        ("tricorn", "-1.5"), ("tricorn", "-1.75"), ("julia", "0.3125"), ("julia", "1.25")])
def test_points_around_a_real_centre(package, product, formula, re):
    native = package.native
    zoom, cap, count = b"1e6", 60, 2000
    constant = -1.75
    rng = np.random.default_rng(23)
    real = rng.normal(size=count) * np.exp2(-rng.integers(0, 40, count))
    imag = rng.normal(size=count) * np.exp2(-rng.integers(0, 40, count))
    imag[::11] = 0.0
    options = native.RenderOptions(disable_bla=1, disable_cycle=1, series_min_terms=32, series_max_terms=32)
    handle = native.create_reference(product, re, "0", zoom, cap, 256, 32, formula=formula,
                                     julia=(repr(constant), "0") if formula == "julia" else ("0", "0"), options=options)
    try:
        _, planes = native.render_points(product, handle, zoom, real, imag, np.zeros(count, dtype=np.int32), cap,
                                         options=options, planes=True)
    finally:
        product.fractal_destroy_reference(handle)
    if formula == "burning-ship":
        orbit, margins = _ship_orbit(re, "0", cap + 2)
        want = [_ship_point(orbit, margins, (float(x), float(y)), cap) for x, y in zip(real, imag)]
    else:
        orbit, margins = (_real_orbit(float(re), constant, cap) if formula == "julia"
                          else _real_orbit(0.0, float(re), cap))
        want = [_point(formula, orbit, margins, (float(x), float(y)), cap) for x, y in zip(real, imag)]
    first = 0 if formula == "julia" else 1
    # A point outside from the start escapes there, before any step.
    norms = [(orbit[first][0] + x) ** 2 + (orbit[first][1] + y) ** 2 for x, y in zip(real, imag)]
    chosen = [i for i, n in enumerate(norms) if n < 3.9]
    assert len(chosen) > count // 2 and sum(want[i] is not None for i in chosen) > 100
    raw = [cap if want[i] is None else want[i][0] - first for i in chosen]
    np.testing.assert_array_equal(planes["orbit_iteration"][chosen], raw)
    np.testing.assert_array_equal(planes["test1"][chosen], [0.0 if want[i] is None else want[i][1] for i in chosen])
    np.testing.assert_array_equal(planes["test2"][chosen], [0.0 if want[i] is None else want[i][2] for i in chosen])


@pytest.mark.parametrize("re,cap", [("-1.62", 2000), ("-2", 1500), ("-1.7548776662466927", 1500)])
def test_mandelbrot_field_around_a_real_centre(package, product, oracle_port, re, cap):
    native = package.native
    fields = []
    for library in (product, oracle_port):
        handle = native.create_reference(library, re, "0", b"1e12", cap, 256, 32)
        try:
            fields.append(native.render_reference(library, handle, 65, 49, b"1e12", cap))
        finally:
            library.fractal_destroy_reference(handle)
    np.testing.assert_array_equal(fields[0].view(np.uint32), fields[1].view(np.uint32))


def test_real_centre_does_not_hold_the_field_up(package, product):
    native = package.native
    width, height, cap = 160, 101, 4000
    times = []
    for im in ("0", "2.8e-16"):
        handle = native.create_reference(product, "0.3", im, b"1e12", cap, 256, 32, formula="julia", julia=("-1.75", "0"))
        try:
            best = 1e9
            for _ in range(6):
                native.render_reference(product, handle, width, height, b"1e12", cap)
                best = min(best, product.fractal_gb300_last_kernel_ms())
            times.append(best)
        finally:
            product.fractal_destroy_reference(handle)
    print(f"on the axis {times[0]:.3f} ms, beside it {times[1]:.3f} ms")
    assert times[0] < 2.0 * times[1]
