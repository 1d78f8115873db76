"""GPU: the alternate formulas' queue over several launches against one.

Lists of more than 16,384 points run in up to eight launches, long orbits
spilled from each to the next; shorter ones run in one.  A point's result
does not depend on its list, so a long list must equal its pieces bit for
bit, planes included.  The lists hold offsets with zero parts (the axes of an
odd-sized view) and the reference centre itself.
"""

from __future__ import annotations

import math

import numpy as np
import pytest

from .golden import cases as case_defs

pytestmark = pytest.mark.gpu

CASES = [("julia", "julia_fixed_1", 24.0, 6000), ("julia", "julia_fixed_2", 9.0, 3000),
         ("burning-ship", "burning_ship_deep", 24.0, 4000), ("tricorn", "tricorn_deep", 30.0, 4000),
         ("tricorn", "tricorn_boundary", 7.0, 3000)]


@pytest.mark.parametrize("planes", [False, True])
@pytest.mark.parametrize("formula,key,log_zoom,cap", CASES)
def test_long_list_equals_its_pieces(package, product, formula, key, log_zoom, cap, planes):
    native, atlas = package.native, package.atlas
    c = case_defs.centres()[key]
    julia = (c["c_re"], c["c_im"]) if formula == "julia" else ("0", "0")
    zoom = atlas.zoom_text(log_zoom)
    handle = native.create_reference(product, c["re"], c["im"], zoom, cap,
                                     atlas.precision_bits(c["re"], c["im"], log_zoom), 32, formula=formula,
                                     julia=julia)
    try:
        count = 16_384 + 4_321
        rng = np.random.default_rng(11)
        radius = (rng.uniform(-2.0, 0.15, count) - log_zoom) * math.log2(10.0)
        angle = rng.uniform(0.0, 2.0 * math.pi, count)
        exponents = np.ceil(radius).astype(np.int32)
        magnitude = np.exp2(radius - exponents)
        real, imag = magnitude * np.cos(angle), magnitude * np.sin(angle)
        real[::97] = 0.0
        imag[::89] = 0.0

        def render(part):
            return native.render_points(product, handle, zoom, real[part], imag[part], exponents[part], cap,
                                        planes=planes)

        whole, whole_planes = render(slice(0, count))
        for start in range(0, count, 8192):
            part = slice(start, min(start + 8192, count))
            field, arrays = render(part)
            np.testing.assert_array_equal(whole[part].view(np.uint32), field.view(np.uint32))
            for name in arrays or {}:
                np.testing.assert_array_equal(whole_planes[name][part], arrays[name], err_msg=name)
    finally:
        product.fractal_destroy_reference(handle)
