"""The aurora palette's tables: when they are made, and for whom.

The tables lie in scratch memory that a thread gives back when it changes its
device.  The host side runs on a stand-in CUDA runtime with two devices, whose
allocator hands a freed address out again; the palette is made once for
unchanged controls and again for any other.  On the GPU, palettes that
alternate between two streams without a wait colour each frame as alone.
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


def test_palette_is_made_once_for_unchanged_controls(library):
    out = fake_cuda.run(library, PRELUDE + """
launches = []
for change in ({}, {}, dict(on=None), dict(phase=0.4), dict(phase=0.4), {}, dict(vocal=0.5), dict(pitch=0.9), dict(cap=999),
               dict(cap=40000), dict(cap=40000), {}, {}):
    before = lib.fake_launches()
    colour(**change)
    launches.append(lib.fake_launches() - before)
print(*launches)
""")
    # One launch colours the field; the palette's own where a control changed.
    assert list(map(int, out.split())) == [2, 1, 1, 2, 1, 2, 2, 2, 2, 2, 1, 2, 1]


@pytest.mark.gpu
def test_palettes_on_two_streams(package, product):
    import ctypes
    torch = pytest.importorskip("torch")
    width, height, frames = 1920, 1080, 12
    field = (torch.arange(width * height, device="cuda", dtype=torch.float32) * 0.731) % 2003.0
    streams = [torch.cuda.Stream() for _ in range(2)]
    controls = [(2000, 0.3), (2000, 0.3), (2000, 1.7), (1500, 1.7)]

    def colour(rgb, index, stream):
        cap, phase = controls[index]
        status = product.fractal_gb300_colourise_device(
            ctypes.c_void_p(field.data_ptr()), ctypes.c_void_p(rgb.data_ptr()), width, height, cap,
            ctypes.c_double(phase), ctypes.c_double(0.4), ctypes.c_double(0.7), ctypes.c_double(0.5),
            ctypes.c_void_p(stream.cuda_stream))
        assert status == 0, package.native.last_error(product)

    def empty():
        return torch.zeros(width * height * 3, dtype=torch.uint8, device="cuda")

    torch.cuda.synchronize()
    alone = []
    for index in range(len(controls)):
        alone.append(empty())
        torch.cuda.synchronize()
        colour(alone[-1], index, streams[0])
        torch.cuda.synchronize()
    made = [empty() for _ in range(frames)]
    torch.cuda.synchronize()
    for n, rgb in enumerate(made):
        colour(rgb, (n * 5 // 3) % len(controls), streams[n % 2])
    torch.cuda.synchronize()
    for n, rgb in enumerate(made):
        assert torch.equal(rgb, alone[(n * 5 // 3) % len(controls)]), n
