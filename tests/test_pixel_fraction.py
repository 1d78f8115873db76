"""CPU: the integer division of csrc/pixel_fraction.h.

A pixel's fraction of the view must be the rounded FP64 quotient for every
index, both coordinate modes and odd, even, smallest and largest dimensions,
past the integer form's limit too.  Host build of the device's code.
"""

from __future__ import annotations

import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fractal-audio-viz_gb300", "csrc")

DRIVER = r"""
#include "pixel_fraction.h"
#include <cstdio>
int main() {
    const int dims[] = {1, 2, 3, 4, 5, 7, 16, 97, 320, 321, 360, 640, 853, 960, 1000, 1080, 1920, 3840, 4320, 7680, 7681,
                        32767, 32768, 32769, 40000, 65537};
    long long bad = 0;
    for (int dim : dims) {
        for (int mode = 0; mode < 2; ++mode) {
            for (int i = 0; i < dim; ++i) {
                const double origin = mode == 1 ? static_cast<double>(dim / 2) : static_cast<double>(dim - 1) / 2.0;
                const double want = (static_cast<double>(i) - origin) / static_cast<double>(dim);
                if (fx::bits_of(fx::pixel_fraction(i, dim, mode)) != fx::bits_of(want)) ++bad;
            }
        }
    }
    std::printf("bad %lld\n", bad);
    return bad != 0;
}
"""


def test_fraction_equals_the_fp64_quotient(tmp_path):
    driver, binary = tmp_path / "driver.cpp", tmp_path / "driver"
    driver.write_text(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I" + CSRC, str(driver), "-o", str(binary)],
                   check=True)
    done = subprocess.run([str(binary)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout
