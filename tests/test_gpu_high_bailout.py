"""GPU: the high bailout in the FP32 form costs its steps, not repeated turns.

With |z| up to 1e4 an orbit takes some five steps more, and the norm of a
small total is quantised more coarsely, so that a rebase at index 0 may leave
the same state again.  Such pixels go on at once; as 64 equal turns they were
the longest of a field by far, four times the kernel's time with the usual
bailout.  It may take two and a half times that, the extra steps and the
coarser turns of the few pixels that need them, and the smooth values agree.
"""

from __future__ import annotations

import numpy as np
import pytest

from .golden import cases as case_defs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("key,log_zoom", [("fhd_stack_e50", 30.0), ("field_e100", 50.0)])
def test_high_bailout_takes_its_steps(package, product, key, log_zoom):
    native, atlas = package.native, package.atlas
    c = case_defs.centres()[key]
    zoom, cap, width, height = atlas.zoom_text(log_zoom), 20_000, 200, 112
    times, fields = [], []
    for mode in (0, 1):
        options = native.RenderOptions(escape_radius_mode=mode, backend=native.BACKEND_CUDA)
        handle = native.create_reference(product, c["re"], c["im"], zoom, cap,
                                         atlas.precision_bits(c["re"], c["im"], log_zoom), 32, options=options)
        try:
            best = 1e9
            for _ in range(12):
                field = native.render_reference(product, handle, width, height, zoom, cap, options=options)
                best = min(best, product.fractal_gb300_last_kernel_ms())
        finally:
            product.fractal_destroy_reference(handle)
        times.append(best)
        fields.append(field)
    print(f"{key}: {times[0] * 1e3:.1f} us, with the high bailout {times[1] * 1e3:.1f} us")
    both = np.isfinite(fields[0]) & np.isfinite(fields[1]) & (fields[0] < cap) & (fields[1] < cap)
    assert both.sum() > width * height // 2
    assert np.abs(fields[1][both] - fields[0][both]).max() < 2.0  # smooth values hardly depend on the bailout
    assert times[1] < 2.5 * times[0]
