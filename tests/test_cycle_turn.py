"""The alternate queue's cycle tests.

On the CPU: a pixel that runs ahead of its lane (csrc/cycle_turn.h) never
makes a step that a cycle test follows, whatever mixture of blocks and single
steps it takes, since the list it waits on keeps no cycle state.  On the GPU:
fields above one launch's 131,072 pixels, with interior regions and caps well
above the first cycle test, equal the same fields without cycle tests (an
interior pixel is at the cap either way, and no view here has an orbit that
stays within the test's 2^-39 and escapes later).
"""

from __future__ import annotations

import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fractal-audio-viz_gb300", "csrc")

DRIVER = r"""
#include "cycle_turn.h"
#include <cstdio>
#include <random>
int main() {
    std::mt19937 rng(3);
    long steps = 0, lost = 0, waits = 0, off = 0;
    for (int n = 0; n < 20000; ++n) {
        const bool cycle = n % 4 != 0;
        int it = static_cast<int>(rng() % 2100);
        while (it < 6000) {
            if (!fx::turn_before_listing(cycle, it)) {
                ++waits;
                off += !cycle;
                break;
            }
            if (rng() % 3 == 0) {  // a block: no cycle test after it
                it += 1 << (rng() % 9);
            } else {
                ++it;
                ++steps;
                lost += cycle && it >= 2048 && it % 32 == 0;
            }
        }
    }
    std::printf("%ld steps, %ld with a cycle test, %ld waits, %ld without cycle tests\n", steps, lost, waits, off);
    return lost != 0 || off != 0 || waits == 0;
}
"""


def test_no_cycle_state_begins_before_a_pixel_is_listed(tmp_path):
    source, binary = tmp_path / "driver.cpp", tmp_path / "driver"
    source.write_text(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + CSRC, str(source), "-o", str(binary)], check=True)
    done = subprocess.run([str(binary)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("planes", [False, True])
@pytest.mark.parametrize("formula,x,y,zoom,julia", [
    ("burning-ship", "-0.1075", "0.04", b"1e6", ("0", "0")), ("burning-ship", "-1.7548776662466927", "0", b"1e6", ("0", "0")),
    ("tricorn", "-0.1", "0.05", b"1e6", ("0", "0")), ("julia", "0.1", "0.1", b"1e6", ("-0.12", "0.74"))])
def test_cycle_tests_change_no_value(package, product, formula, x, y, zoom, julia, planes):
    native = package.native
    width, height, cap = 512, 260, 6000
    fields = []
    for off in (0, 1):
        options = native.RenderOptions(strict=0, disable_cycle=off)
        handle = native.create_reference(product, x, y, zoom, cap, 192, 8, formula=formula, julia=julia, options=options)
        try:
            out = native.render_reference(product, handle, width, height, zoom, cap, options=options, planes=planes)
        finally:
            product.fractal_destroy_reference(handle)
        fields.append(out if planes else (out, {}))
    (with_tests, planes_with), (without, planes_without) = fields
    assert (without == np.float32(cap)).any()
    np.testing.assert_array_equal(with_tests.view(np.uint32), without.view(np.uint32))
    for name in planes_without:
        np.testing.assert_array_equal(planes_with[name], planes_without[name], err_msg=name)
