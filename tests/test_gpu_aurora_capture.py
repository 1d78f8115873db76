"""GPU: the aurora colour call recorded into a caller's graph.

In relaxed mode a recorded call, made after an ordinary one on the same or on
another stream, replays to the same bytes on new fields, and ordinary calls
go on afterwards.
"""

from __future__ import annotations

import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("same_stream", [True, False])
def test_recorded_call_replays(package, product, same_stream):
    width, height, cap = 640, 361, 2000
    ramp = torch.arange(width * height, device="cuda", dtype=torch.float32)
    field = (ramp * 0.731) % 2003.0
    rgb = torch.zeros(width * height * 3, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.Stream()
    other = stream if same_stream else torch.cuda.Stream()

    def colour(on, phase=0.3):
        status = product.fractal_gb300_colourise_device(
            ctypes.c_void_p(field.data_ptr()), ctypes.c_void_p(rgb.data_ptr()), width, height, cap,
            ctypes.c_double(phase), ctypes.c_double(0.4), ctypes.c_double(0.7), ctypes.c_double(0.5),
            ctypes.c_void_p(on.cuda_stream))
        assert status == 0, package.native.last_error(product)

    torch.cuda.synchronize()
    colour(other)
    torch.cuda.synchronize()
    first = rgb.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
        colour(stream)
    rgb.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(rgb, first)
    # Ordinary calls go on, on either stream.
    field.copy_((ramp * 0.417) % 1999.0)
    torch.cuda.synchronize()
    results = []
    for on in (other, stream):
        rgb.zero_()
        torch.cuda.synchronize()
        colour(on)
        torch.cuda.synchronize()
        results.append(rgb.clone())
    assert torch.equal(results[0], results[1])
    assert not torch.equal(results[0], first)
    rgb.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(rgb, results[0])
