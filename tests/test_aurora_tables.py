"""CPU: the aurora palette's tables follow the thread's device.

The tables lie in scratch memory that a thread gives back when it changes its
device.  The host side runs on a stand-in CUDA runtime with two devices, whose
allocator hands a freed address out again.
"""

from __future__ import annotations

import pytest

from . import fake_cuda

PRELUDE = """
stream = ctypes.c_void_p(lib.fake_stream())
field, rgb = (ctypes.c_float * 4096)(), (ctypes.c_uint8 * 12288)()
options = native.RenderOptions()
lib.fractal_gb300_colourise_device.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int,
                                               *[ctypes.c_double] * 4, ctypes.c_void_p]
def colour(cap=2000, phase=0.3, vocal=0.4, pitch=0.5, on=stream):
    check(lib.fractal_gb300_colourise_device(ctypes.addressof(field), ctypes.addressof(rgb), 64, 64, cap, phase, vocal,
                                             0.7, pitch, on))
def render():
    check(lib.fractal_gb300_render_direct_device(field, None, 32, 32, b"1", b"-0.5", b"0.0", 100, 0, 0.0, 0.0,
                                                 ctypes.byref(options), stream))
"""


@pytest.fixture(scope="module")
def library(package, tmp_path_factory):
    return fake_cuda.link(package, tmp_path_factory.mktemp("fake"))


def test_waves_are_uploaded_again_after_another_device(library):
    out = fake_cuda.run(library, PRELUDE + """
lib.fake_devices(2)
uploads = []
for device, call in ((0, colour), (0, colour), (1, render), (0, colour)):
    lib.fake_device(device)
    before = lib.fake_uploaded()
    call()
    uploads.append(lib.fake_uploaded() - before)
print(*uploads)
""")
    first, again, other, back = map(int, out.split())
    assert first == 8000 * 8 and again == 0 and other == 0
    assert back == first
