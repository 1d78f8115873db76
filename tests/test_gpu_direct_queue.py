"""GPU: the direct queue's launches and products against the oracle.

Pixels past the first launch's budget are spilled and resumed by the later
launches; whole-set views spill enough for the lists, odd heights put a row
of pixels on the real axis (products with an exact zero), and views of the
period-2 and period-3 bulbs' centres pass near zero (products of few bits,
ties included).  Alone the products run on the integer pipe, in a batch
beside the FP32 queue in FP64; both must equal the oracle bit for bit.
"""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from .golden import cases as case_defs

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

VIEWS = [("-0.6", "0.0", 0.0, 641, 361, 5000), ("-0.6123", "0.0317", 0.05, 1101, 619, 3000),
         ("-1.0", "0.0", 1.1, 255, 129, 4000), ("-1.7548776662466927", "0.0", 1.9, 320, 181, 6000),
         ("-0.1225611668766536", "0.7448617666197442", 1.5, 320, 180, 6000), ("0.3", "0.5", 2.5, 97, 33, 2000)]


def _oracle(package, oracle_port, view):
    x, y, log_zoom, width, height, cap = view
    return package.native.render_fractal(oracle_port, width, height, package.atlas.zoom_text(log_zoom), x, y, cap, 256,
                                         False, threads=0)


@pytest.mark.parametrize("view", VIEWS)
def test_direct_view_equals_oracle(package, product, oracle_port, view):
    x, y, log_zoom, width, height, cap = view
    field = torch.empty(width * height, dtype=torch.float32, device="cuda")
    status = product.fractal_gb300_render_direct_device(
        ctypes.c_void_p(field.data_ptr()), None, width, height, package.atlas.zoom_text(log_zoom), x.encode(),
        y.encode(), cap, 0, 0.0, 0.0, ctypes.byref(package.native.RenderOptions()), None)
    assert status == 0, package.native.last_error(product)
    steps = ctypes.c_ulonglong(0)
    assert product.fractal_gb300_last_direct_steps(ctypes.byref(steps)) == 0
    want = _oracle(package, oracle_port, view)
    np.testing.assert_array_equal(field.cpu().numpy().view(np.uint32), want.view(np.uint32))


def test_direct_level_beside_the_fp32_queue_equals_itself_alone(package, product):
    """The whole-set level of a ladder, batched with FP32-queue levels: counts
    equal the level's alone (its smooth value is the FP32 one there)."""
    c = case_defs.centres()["fhd_stack_e50"]
    levels = [lv for lv in case_defs.fhd_stack_levels() if lv[0] in (0, 13, 20, 30)]
    stack = package.atlas.KeyframeStack(product, c["re"], c["im"], levels, step=0.9030899869919435)
    try:
        width, height = 641, 361
        fields = torch.empty((len(levels), width * height), dtype=torch.float32, device="cuda")
        counts = torch.empty((len(levels), width * height), dtype=torch.int32, device="cuda")
        targets = [(fields[i].data_ptr(), counts[i].data_ptr()) for i in range(len(levels))]
        stack.render_batch_device(targets, width, height, form=1)
        torch.cuda.synchronize()
        alone_field = torch.empty(width * height, dtype=torch.float32, device="cuda")
        alone = torch.empty(width * height, dtype=torch.int32, device="cuda")
        for i, keyframe in enumerate(stack.keyframes):
            if keyframe.reference is None:
                stack.render_device(keyframe, alone_field.data_ptr(), alone.data_ptr(), width, height, form=0)
                torch.cuda.synchronize()
                assert torch.equal(alone, counts[i]), keyframe.level
    finally:
        stack.close()
