"""GPU: the centre pixel of odd-sized fields in the FP32 form.

That pixel is the reference orbit itself: its delta stays zero through every
block.  Its count must be the FP64 form's, whatever the orbit's length and
the blocks' limit, and with derivative planes as without.
"""

from __future__ import annotations

import ctypes

import pytest

from .golden import cases as case_defs

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

VIEWS = [("fhd_stack_e50", 45.0, 33, 17, 137000, 64), ("fhd_stack_e50", 20.0, 1, 1, 60000, 2),
         ("fhd_stack_e50", 50.0, 65, 1, 100000, 7), ("field_e100", 90.0, 17, 33, 137000, 64),
         ("field_640x360_e30", 30.0, 31, 31, 50000, 5)]


@pytest.mark.parametrize("key,log_zoom,width,height,cap,block", VIEWS)
def test_centre_pixel_follows_the_reference(package, product, key, log_zoom, width, height, cap, block):
    native, atlas = package.native, package.atlas
    c = case_defs.centres()[key]
    zoom = atlas.zoom_text(log_zoom)
    handle = native.create_reference(product, c["re"], c["im"], zoom, cap,
                                     atlas.precision_bits(c["re"], c["im"], log_zoom), 32)
    counts = torch.zeros((2, width * height), dtype=torch.int32, device="cuda")
    field = torch.empty(width * height, dtype=torch.float32, device="cuda")
    try:
        options = native.RenderOptions()
        for form in (0, 1):
            status = product.fractal_gb300_render_reference_device(
                ctypes.c_void_p(field.data_ptr()), ctypes.c_void_p(counts[form].data_ptr()), width, height, zoom,
                ctypes.c_void_p(handle), cap, 3, block, ctypes.byref(options), form, None)
            assert status == 0, native.last_error(product)
        torch.cuda.synchronize()
    finally:
        product.fractal_destroy_reference(handle)
    centre = (height // 2) * width + width // 2
    assert int(counts[0, centre]) == int(counts[1, centre]) > 0
