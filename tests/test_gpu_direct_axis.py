"""GPU: direct views with a row of pixels exactly on the real axis.

The imaginary part of such an orbit is a zero at every step.  The fields equal
the same fields of the no-allocation entry, which keeps every pixel in its
first launch, for the four formulas and for parameters with either zero; and
the row does not hold the field up: its step has one product and one sum where
another's has three and three, so with the same cap the view takes no more
than twice the time of the view one row smaller, whose longest orbits run to
the cap too.
"""

from __future__ import annotations

import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

_ARGS = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_char_p, ctypes.c_char_p,
         ctypes.c_char_p, ctypes.c_int, ctypes.c_int, ctypes.c_double, ctypes.c_double, ctypes.c_void_p,
         ctypes.c_void_p]


def _call(package, product, name, formula, x, y, width, height, cap, julia, field, counts, stream=None):
    function = getattr(product, name)
    function.restype, function.argtypes = ctypes.c_int, _ARGS
    options = package.native.RenderOptions()
    status = function(field.data_ptr(), counts.data_ptr(), width, height, b"1", x, y, cap,
                      package.native.FORMULA_IDS[formula], *julia, ctypes.addressof(options),
                      stream.cuda_stream if stream else None)
    assert status == 0, package.native.last_error(product)


def _buffers(width, height):
    pixels = width * height
    return (torch.full((pixels,), -1.0, dtype=torch.float32, device="cuda"),
            torch.zeros(pixels, dtype=torch.int32, device="cuda"))


@pytest.mark.parametrize("formula,x,y,julia", [
    ("mandelbrot", b"-0.6", b"0.0", (0.0, 0.0)), ("mandelbrot", b"-0.6", b"-0.0", (0.0, 0.0)),
    ("burning-ship", b"-0.5", b"0.0", (0.0, 0.0)), ("burning-ship", b"-0.5", b"-0.0", (0.0, 0.0)),
    ("tricorn", b"-0.4", b"0.0", (0.0, 0.0)), ("tricorn", b"-0.4", b"-0.0", (0.0, 0.0)),
    ("julia", b"0.0", b"0.0", (-1.25, 0.0)), ("julia", b"0.0", b"0.0", (-1.31, -0.0))])
def test_axis_row_equals_the_row_kept(package, product, formula, x, y, julia):
    width, height, cap = 401, 225, 5000
    results = []
    torch.cuda.synchronize()
    for name in ("fractal_gb300_render_direct_device", "fractal_gb300_render_direct_device_noalloc"):
        field, counts = _buffers(width, height)
        torch.cuda.synchronize()
        _call(package, product, name, formula, x, y, width, height, cap, julia, field, counts)
        torch.cuda.synchronize()
        results.append((field, counts))
    assert torch.equal(results[0][0].view(torch.int32), results[1][0].view(torch.int32))
    assert torch.equal(results[0][1], results[1][1])


def test_axis_row_does_not_hold_the_field_up(package, product):
    stream = torch.cuda.Stream()

    def best(height):
        field, counts = _buffers(400, height)
        times = []
        for _ in range(6):
            start, stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            start.record(stream)
            _call(package, product, "fractal_gb300_render_direct_device", "mandelbrot", b"-0.6", b"0.0", 400, height,
                  5000, (0.0, 0.0), field, counts, stream)
            stop.record(stream)
            stop.synchronize()
            times.append(start.elapsed_time(stop))
        return min(times[1:])

    even, odd = best(224), best(225)
    print(f"even {even:.3f} ms, odd {odd:.3f} ms")
    assert odd < 2.0 * even
