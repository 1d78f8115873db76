"""GPU: a time budget bounds the pixels that blocks alone take to the cap.

Deep inside a component every pixel of these fields is interior and its delta
never outgrows the block radius; the cap is a whole number of the longest
blocks past the first index, and the corners lie inside the blocks' input
radius.  So no single step is made, and the field runs in the queue's start of
new pixels.  With a budget far below the field's time the unfinished pixels
are NaN and the finished ones equal the unbudgeted render's.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Centre near an attracting fixed point, no axis crossed by the orbit.
VIEWS = [("burning-ship", "-0.1075", "0.04"), ("tricorn", "-0.1", "0.05")]


@pytest.mark.parametrize("formula,x,y", VIEWS)
def test_budget_stops_the_start_of_new_pixels(package, product, formula, x, y):
    native = package.native
    zoom, cap, width, height = b"1e14", 32 * 4096 + 1, 2880, 2880
    handle = native.create_reference(product, x, y, zoom, cap, 256, 8, formula=formula)
    try:
        def render(budget):
            field = native.render_reference(product, handle, width, height, zoom, cap,
                                            options=native.RenderOptions(time_budget_ms=budget))
            return field, product.fractal_gb300_last_kernel_ms()

        render(0)
        unbudgeted, whole_ms = render(0)
        field, ms = render(1)
    finally:
        product.fractal_destroy_reference(handle)
    print(f"{formula}: {whole_ms:.2f} ms, with the budget {ms:.2f} ms, {int(np.isnan(field).sum())} unfinished")
    np.testing.assert_array_equal(unbudgeted, np.float32(cap))
    assert whole_ms > 4.0, whole_ms  # a budget of 1 ms must cut it
    unfinished = np.isnan(field)
    assert unfinished.any()
    np.testing.assert_array_equal(field[~unfinished], unbudgeted[~unfinished])
