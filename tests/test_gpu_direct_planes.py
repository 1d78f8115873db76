"""GPU: render planes of direct fields through the resuming launches.

Planes of the four formulas, from fields whose long orbits go through one and
through several resuming launches, equal the oracle's: iterations, values and
escape norms bit for bit (phase and distance estimate pass through the
libraries' atan2, hypot and logarithm).  The formulas without a derivative
plane take the same steps with planes as without, so their fields may not take
half as long again.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VIEWS = [("mandelbrot", b"1", "-0.6", "0.1", 320, 181, 1500), ("mandelbrot", b"1", "-0.6", "0.0", 641, 361, 1500),
         ("julia", b"1", "0.0", "0.0", 801, 401, 2000), ("burning-ship", b"1", "-0.5", "-0.3", 801, 401, 1500),
         ("tricorn", b"50", "-0.3", "-0.1", 320, 181, 1500), ("tricorn", b"50", "-0.3", "-0.1", 801, 401, 1500)]


@pytest.mark.parametrize("formula,zoom,x,y,width,height,cap", VIEWS)
def test_planes_equal_oracle(package, product, oracle_port, formula, zoom, x, y, width, height, cap):
    def render(library):
        return package.native.render_fractal(library, width, height, zoom, x, y, cap, 256, False, threads=0,
                                             formula=formula, julia=(-0.7269, 0.1889), planes=True)

    field, planes = render(product)
    want, expected = render(oracle_port)
    np.testing.assert_array_equal(field.view(np.uint32), want.view(np.uint32))
    for name in ("orbit_iteration", "test1", "test2"):
        np.testing.assert_array_equal(planes[name], expected[name], err_msg=name)
    np.testing.assert_allclose(planes["phase"], expected["phase"], rtol=1e-12, atol=1e-300)
    # The estimate is a complex quotient: each part is off relative to its modulus.
    modulus = np.hypot(expected["de_x"], expected["de_y"])
    for name in ("de_x", "de_y"):
        off = np.abs(planes[name] - expected[name])
        assert (off <= 1e-12 * modulus).all(), (name, float(off.max()))


@pytest.mark.parametrize("formula", ["burning-ship", "tricorn"])
def test_planes_without_a_derivative_cost_no_steps(package, product, formula):
    def best(planes):
        times = []
        for _ in range(8):
            package.native.render_fractal(product, 64, 36, b"1", "-0.3", "-0.1", 4000, 128, False, formula=formula,
                                          planes=planes)
            times.append(product.fractal_gb300_last_kernel_ms())
        return min(times)

    without, with_planes = best(False), best(True)
    print(f"{formula}: {without:.3f} ms, with planes {with_planes:.3f} ms")
    assert with_planes < 1.5 * without
