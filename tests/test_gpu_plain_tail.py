"""GPU: the plain Mandelbrot form's double tail and image series against the
oracle.

The tail runs steps whose escape, rebase and cycle tests FP32 estimates
settle, the others exactly; the series sums scaled doubles.  Views from the
whole set's neighbourhood to 1e50: odd sizes (offsets with a zero part), a
centre on the real axis (orbit values with a zero part), escaping centres (exact
steps past the reference's end), interiors (cycle
tests, the 64-rebase limit), the high bailout, strict and cycle-free renders.
Fields, iteration and test planes equal the oracle bit for bit.
"""

from __future__ import annotations

import numpy as np
import pytest

from .golden import cases as case_defs

pytestmark = pytest.mark.gpu

REAL = ("-1.7548776662466927", "0.0")
OUTSIDE = ("-0.7436438870371587", "0.1318259042053")  # escapes: pixels go past the reference's end
VIEWS = [("fhd_stack_e50", 4.0, 161, 91, 3000, {}), ("fhd_stack_e50", 12.5, 97, 65, 8000, {}),
         ("fhd_stack_e50", 30.0, 161, 90, 60000, {"escape_radius_mode": 1}), ("fhd_stack_e50", 50.0, 131, 77, 100000, {}),
         ("field_640x360_e30", 30.0, 160, 91, 50000, {"disable_cycle": 1}),
         ("field_640x360_e30", 29.0, 65, 33, 50000, {"strict": 1}), (REAL, 6.0, 97, 65, 2000, {}),
         (REAL, 3.0, 65, 65, 1500, {"strict": 1, "strict_cycle": 1}), (REAL, 11.0, 33, 17, 4000, {"disable_bla": 1}),
         (OUTSIDE, 6.0, 97, 65, 3000, {}), (OUTSIDE, 9.0, 97, 64, 3000, {"escape_radius_mode": 1}),
         (OUTSIDE, 3.0, 65, 65, 1200, {"strict": 1, "strict_cycle": 1}), (("0.26", "0.0"), 1.5, 97, 65, 1500, {})]


@pytest.mark.parametrize("planes", [False, True])
@pytest.mark.parametrize("view", VIEWS)
def test_plain_field_equals_oracle(package, product, oracle_port, view, planes):
    native, atlas = package.native, package.atlas
    centre, log_zoom, width, height, cap, flags = view
    if isinstance(centre, str):
        entry = case_defs.centres()[centre]
        x, y = entry["re"], entry["im"]
    else:
        x, y = centre
    options = native.RenderOptions()
    for name, value in flags.items():
        setattr(options, name, value)
    arguments = (width, height, atlas.zoom_text(log_zoom), x, y, cap, atlas.precision_bits(x, y, log_zoom), True)
    got = native.render_fractal(product, *arguments, options=options, planes=planes)
    want = native.render_fractal(oracle_port, *arguments, options=options, planes=planes)
    if planes:
        got, got_planes = got
        want, want_planes = want
        for key in ("orbit_iteration", "test1", "test2"):
            np.testing.assert_array_equal(got_planes[key], want_planes[key], err_msg=key)
        np.testing.assert_allclose(got_planes["phase"], want_planes["phase"], rtol=1e-12, atol=1e-300)
        # The estimate is one complex quotient: a part's error is relative to
        # the pair's modulus.
        modulus = np.hypot(want_planes["de_x"], want_planes["de_y"])
        for key in ("de_x", "de_y"):
            assert (np.abs(got_planes[key] - want_planes[key]) <= 1e-12 * modulus).all(), key
    np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
