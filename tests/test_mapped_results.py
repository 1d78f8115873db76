"""CPU: whose pages a host call asks for.

Results of 4 MB and more are mapped before the copy, each buffer once; smaller
calls ask for nothing, which costs more than their copy gains.  The host side
runs on a stand-in CUDA runtime that counts the requests.
"""

from __future__ import annotations

from . import fake_cuda


def test_only_large_results_are_mapped(package, tmp_path):
    out = fake_cuda.run(fake_cuda.link(package, tmp_path), """
import numpy as np
def asked(call):
    before = lib.fake_mapped()
    call()
    return lib.fake_mapped() - before
def render(width, height, planes):
    native.render_fractal(lib, width, height, b"1", "-0.5", "0.0", 100, 128, False, planes=planes)
def colour(width, height):
    native.colourise(lib, np.zeros(width * height, np.float32), width, height, 100, 0.1, 0.2, 0.3, 0.4)
print(asked(lambda: render(960, 540, False)), asked(lambda: render(320, 180, True)), asked(lambda: colour(1280, 720)),
      asked(lambda: render(1920, 1080, False)), asked(lambda: render(640, 360, True)), asked(lambda: colour(1920, 1080)))
""")
    small, small_planes, small_rgb, large, planes, rgb = map(int, out.split())
    assert (small, small_planes, small_rgb) == (0, 0, 0)
    page = 65536
    for got, bytes_ in ((large, 1920 * 1080 * 4), (planes, 640 * 360 * 52), (rgb, 1920 * 1080 * 3)):
        assert bytes_ <= got <= bytes_ + 14 * page
