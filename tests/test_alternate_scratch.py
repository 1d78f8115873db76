"""CPU: device memory that the alternate formulas' queue takes for its lists.

A call takes what its field needs: a short point list a few kilobytes, a field
that one launch does no spill list, and a batch lists for the lanes that carry
such fields only.  The host side runs on a stand-in CUDA runtime.
"""

from __future__ import annotations

import pytest

from . import fake_cuda

PRELUDE = """
options = native.RenderOptions()
field = (ctypes.c_float * (1024 * 1024))()
def reference(formula):
    return native.create_reference(lib, "0.3", "0.4", b"1e12", 500, 256, 8, formula=formula)
tricorn, mandelbrot = reference("tricorn"), reference("mandelbrot")
def single(width, height, handle=tricorn):
    check(lib.fractal_gb300_render_reference_device(field, None, width, height, b"1e12", ctypes.c_void_p(handle), 500, 3, 256,
                                                    ctypes.byref(options), 0, None))
def batch(handles, width, height):
    frames = (native.Field * len(handles))()
    for i, handle in enumerate(handles):
        frames[i].field, frames[i].zoom_text, frames[i].reference = ctypes.addressof(field), b"1e12", handle
        frames[i].width, frames[i].height, frames[i].max_iter = width, height, 500
    check(lib.fractal_gb300_render_fields_device(frames, len(handles), None, None, 3, 256, ctypes.byref(options), 0, 0, None))
def taken(call, *arguments):
    before = lib.fake_allocated()
    call(*arguments)
    return lib.fake_allocated() - before
single(1, 1, mandelbrot), single(1, 1)
"""
MB = 1 << 20
SLOT = 2 * (1 << 18) * 128


@pytest.fixture(scope="module")
def library(package, tmp_path_factory):
    return fake_cuda.link(package, tmp_path_factory.mktemp("fake"))


def test_lists_fit_the_field(library):
    few, one_launch, large, again = map(int, fake_cuda.run(library, PRELUDE + """
print(taken(single, 3, 1), taken(single, 512, 256), taken(single, 1024, 1024), taken(single, 1024, 1024))
""").split())
    assert few <= 64 * 1024
    assert one_launch <= 24 * MB
    assert SLOT - 24 * MB <= large <= SLOT + 24 * MB
    assert again == 0


def test_lists_are_for_the_lanes_with_such_fields(library):
    alone, beside, two = map(int, fake_cuda.run(library, PRELUDE + """
print(taken(batch, [tricorn], 1024, 1024), taken(batch, [mandelbrot] * 5 + [tricorn] + [mandelbrot] * 4, 1024, 1024),
      taken(batch, [tricorn, tricorn, mandelbrot], 1024, 1024))
""").split())
    assert alone >= SLOT
    assert beside <= 16 * MB
    assert SLOT <= two <= 2 * (SLOT + 24 * MB)
