"""The direct queue's launches: how many, and what each leaves to the next.

On the CPU (stand-in CUDA runtime): a batch whose caps the first launch's
budget covers gets no resuming launch, a small one gets one, a larger one
three.  On the GPU: fields on both sides of those lines, and one whose long
orbits overfill the spill list, equal the same fields rendered by the
no-allocation entry, which has no list and runs every pixel in its first
launch.
"""

from __future__ import annotations

import ctypes
import os
import subprocess

import pytest

from . import fake_cuda
from .conftest import ROOT


def test_resuming_launches(package, tmp_path):
    out = fake_cuda.run(fake_cuda.link(package, tmp_path), """
options = native.RenderOptions()
field = (ctypes.c_float * (512 * 512))()
counts = []
for width, height, cap in ((64, 36, 256), (64, 36, 257), (512, 512, 256), (512, 512, 257), (513, 512, 256),
                           (513, 512, 257), (900, 800, 100), (900, 800, 5000)):
    before = lib.fake_launches()
    check(lib.fractal_gb300_render_direct_device(field, None, width, height, b"1", b"-0.5", b"0.0", cap, 0, 0.0, 0.0,
                                                 ctypes.byref(options), None))
    counts.append(lib.fake_launches() - before)
print(*counts)
""")
    # The coordinate tables, the fresh pixels, and the resuming launches.
    assert list(map(int, out.split())) == [2, 3, 2, 3, 2, 5, 2, 5]


def test_marks_tell_launches_apart(tmp_path):
    """A list is written by every other launch: an entry that one of them left
    out must not pass for its own with the mark of the one before."""
    source, binary = tmp_path / "driver.cpp", tmp_path / "driver"
    source.write_text("""
#include "device.h"
#include <set>
int main() {
    std::set<unsigned long long> marks{0ull};  // 0: a cleared entry
    for (unsigned long long generation = 1; generation <= 1000; ++generation) {
        for (int launch = 0; launch < fgb::kDirectLaunches; ++launch) {
            if (!marks.insert(fgb::spill_mark(generation, launch)).second) return 1;
        }
    }
    return 0;
}
""")
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(fake_cuda.PACKAGE_DIR, "csrc"),
                    "-I" + os.path.join(ROOT, "include"), "-I" + fake_cuda.cuda_include(), str(source), "-o", str(binary)],
                   check=True)
    subprocess.run([str(binary)], check=True)


_ARGS = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_char_p, ctypes.c_char_p,
         ctypes.c_char_p, ctypes.c_int, ctypes.c_int, ctypes.c_double, ctypes.c_double, ctypes.c_void_p,
         ctypes.c_void_p]
SEA = (b"4.5e5", b"-0.743643887037151", b"0.13182590420533", (0.0, 0.0))
VIEWS = [("mandelbrot", SEA, 512, 512, 3000), ("mandelbrot", SEA, 513, 512, 3000), ("mandelbrot", SEA, 200, 112, 256),
         ("burning-ship", (b"20", b"-1.76", b"-0.03", (0.0, 0.0)), 257, 255, 4000),
         ("julia", (b"1", b"0.0", b"0.0", (-0.7269, 0.1889)), 1101, 619, 4000),
         ("tricorn", (b"30", b"-1.4", b"0.01", (0.0, 0.0)), 801, 401, 4000),
         # 646,000 pixels past the budget, of 524,288 entries.
         ("burning-ship", (b"1", b"-0.5", b"-0.3", (0.0, 0.0)), 3840, 2160, 600)]


@pytest.mark.gpu
@pytest.mark.parametrize("formula,view,width,height,cap", VIEWS)
def test_spilled_pixels_equal_pixels_kept(package, product, formula, view, width, height, cap):
    torch = pytest.importorskip("torch")
    zoom, x, y, julia = view
    options = package.native.RenderOptions()
    results = []
    for name in ("fractal_gb300_render_direct_device", "fractal_gb300_render_direct_device_noalloc"):
        function = getattr(product, name)
        function.restype, function.argtypes = ctypes.c_int, _ARGS
        field = torch.full((width * height,), -1.0, dtype=torch.float32, device="cuda")
        counts = torch.zeros(width * height, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        status = function(field.data_ptr(), counts.data_ptr(), width, height, zoom, x, y, cap,
                          package.native.FORMULA_IDS[formula], *julia, ctypes.addressof(options), None)
        assert status == 0, package.native.last_error(product)
        torch.cuda.synchronize()
        results.append((field, counts))
    assert int((results[1][1] > 256).sum()) > 1000 or cap <= 256
    assert torch.equal(results[0][0].view(torch.int32), results[1][0].view(torch.int32))
    assert torch.equal(results[0][1], results[1][1])
