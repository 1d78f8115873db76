"""The alternate formulas' launches: how many, and several against one.

Fields and lists of more than 131,072 pixels run in eight launches, long
orbits spilled from each to the next; shorter ones run in one (counted on a
stand-in CUDA runtime).  A point's result does not depend on its list, so on
the GPU a long list must equal its pieces bit for bit, planes included.
"""

from __future__ import annotations

import math

import numpy as np
import pytest

from . import fake_cuda
from .golden import cases as case_defs


def test_launches_of_a_field(package, tmp_path):
    out = fake_cuda.run(fake_cuda.link(package, tmp_path), """
options = native.RenderOptions()
field = (ctypes.c_float * (512 * 512))()
handle = native.create_reference(lib, "0.3", "0.4", b"1e12", 500, 256, 8, formula="tricorn")
counts = []
for width, height in ((3, 1), (512, 256), (512, 257)):
    for _ in range(2):  # the first call also makes the reference's tables
        before = lib.fake_launches()
        check(lib.fractal_gb300_render_reference_device(field, None, width, height, b"1e12", ctypes.c_void_p(handle), 500,
                                                        3, 256, ctypes.byref(options), 0, None))
    counts.append(lib.fake_launches() - before)
print(*counts)
""")
    assert list(map(int, out.split())) == [1, 1, 8]


CASES = [("julia", "julia_fixed_1", 24.0, 6000), ("julia", "julia_fixed_2", 9.0, 3000),
         ("burning-ship", "burning_ship_deep", 24.0, 4000), ("tricorn", "tricorn_deep", 30.0, 4000),
         ("tricorn", "tricorn_boundary", 7.0, 3000)]


@pytest.mark.gpu
@pytest.mark.parametrize("planes", [False, True])
@pytest.mark.parametrize("escape_mode", [0, 1])
@pytest.mark.parametrize("formula,key,log_zoom,cap", CASES)
def test_long_list_equals_its_pieces(package, product, formula, key, log_zoom, cap, escape_mode, planes):
    native, atlas = package.native, package.atlas
    c = case_defs.centres()[key]
    julia = (c["c_re"], c["c_im"]) if formula == "julia" else ("0", "0")
    zoom = atlas.zoom_text(log_zoom)
    options = native.RenderOptions(escape_radius_mode=escape_mode)
    handle = native.create_reference(product, c["re"], c["im"], zoom, cap,
                                     atlas.precision_bits(c["re"], c["im"], log_zoom), 32, formula=formula,
                                     julia=julia, options=options)
    try:
        count = 131_072 + 4_321
        rng = np.random.default_rng(29)
        radius = (rng.uniform(-2.0, 0.15, count) - log_zoom) * math.log2(10.0)
        angle = rng.uniform(0.0, 2.0 * math.pi, count)
        exponents = np.ceil(radius).astype(np.int32)
        magnitude = np.exp2(radius - exponents)
        real, imag = magnitude * np.cos(angle), magnitude * np.sin(angle)
        real[::97] = 0.0
        imag[::89] = 0.0

        def render(part):
            return native.render_points(product, handle, zoom, real[part], imag[part], exponents[part], cap,
                                        options=options, planes=planes)

        whole, whole_planes = render(slice(0, count))
        for start in range(0, count, 70_000):
            part = slice(start, min(start + 70_000, count))
            field, arrays = render(part)
            np.testing.assert_array_equal(whole[part].view(np.uint32), field.view(np.uint32))
            for name in arrays or {}:
                np.testing.assert_array_equal(whole_planes[name][part], arrays[name], err_msg=name)
    finally:
        product.fractal_destroy_reference(handle)
