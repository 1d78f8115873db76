"""CPU: a scratch buffer is clear before the first launch that may use it.

The library's streams do not wait for the default stream, so a clear that is
still running there would zero what a kernel has written since: pixels parked
on a list, claim counters, generation marks.  The host side runs on a stand-in
CUDA runtime; first calls, calls that grow a buffer and calls on a caller's
stream may not launch while a new buffer's clear is in flight.
"""

from __future__ import annotations

import pytest

from . import fake_cuda

CODE = """
stream = ctypes.c_void_p(lib.fake_stream())
options = native.RenderOptions()
field = (ctypes.c_float * (512 * 512))()
def direct(width, height, stream):
    check(lib.fractal_gb300_render_direct_device(field, None, width, height, b"1", b"-0.5", b"0.0", 500, {direct}, 0.0, 0.0,
                                                 ctypes.byref(options), stream))
def deep(width, height, stream):
    frames = (native.Field * 2)()
    for i in range(2):
        frames[i].field = ctypes.addressof(field)
        frames[i].zoom_text, frames[i].reference, frames[i].width = b"1e12", handle, width
        frames[i].height, frames[i].max_iter = height, 500
    check(lib.fractal_gb300_render_fields_device(frames, 2, None, None, 3, 256, ctypes.byref(options), 1, {flags}, stream))
handle = native.create_reference(lib, "0.3", "0.4", b"1e12", 500, 256, 8, formula={formula!r}, julia=("-0.7", "0.2"))
for call in (direct, deep):
    for width, height in ((16, 16), (200, 180), (500, 400)):
        for target in (None, stream):
            call(width, height, target)
print(lib.fake_launches(), lib.fake_hazards())
"""


@pytest.fixture(scope="module")
def library(package, tmp_path_factory):
    return fake_cuda.link(package, tmp_path_factory.mktemp("fake"))


@pytest.mark.parametrize("formula,flags", [("burning-ship", 0), ("julia", 1), ("tricorn", 0)])
def test_no_launch_while_a_new_buffer_is_cleared(library, formula, flags):
    ids = {"julia": 1, "burning-ship": 2, "tricorn": 3}
    launches, hazards = map(int, fake_cuda.run(library, CODE.format(direct=ids[formula], flags=flags, formula=formula)).split())
    assert launches > 0
    assert hazards == 0


def test_the_cost_network_workspace_is_clear_before_its_first_layer(library):
    launches, hazards = map(int, fake_cuda.run(library, """
        lib.fractal_gb300_costnet_create.restype = ctypes.c_void_p
        lib.fractal_gb300_costnet_predict.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p,
                                                      ctypes.c_void_p]
        net = lib.fractal_gb300_costnet_create(7)
        assert net, native.last_error(lib)
        stream = lib.fake_stream()
        rows = (ctypes.c_uint16 * (1024 * 320 + 8))()
        x = (ctypes.addressof(rows) + 15) // 16 * 16
        out = (ctypes.c_float * 1024)()
        for count in (128, 1024):
            check(lib.fractal_gb300_costnet_predict(net, x, count, ctypes.addressof(out), stream))
        print(lib.fake_launches(), lib.fake_hazards())
        """).split())
    assert launches > 0
    assert hazards == 0
