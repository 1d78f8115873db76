"""CPU: the quotients formed without a division (csrc/corrected_quotient.h).

Pixel offsets over view dimensions: every offset of each dimension up to 2048
and of every 61st beyond it to 32768.  Palette shares over 255: every 251st
float from 2^-100 to 256, and below that no share changes a byte.
"""

from __future__ import annotations

import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fractal-audio-viz_gb300", "csrc")

DRIVER = r"""
#include "corrected_quotient.h"
#include <cstdio>
#include <cstring>
int main() {
    long bad = 0, offsets = 0, shares = 0;
    for (int n = 1; n <= 32768; n += n < 2048 ? 1 : 61) {
        const float d = static_cast<float>(n), per = 1.0f / d;
        for (int twice = -n; twice <= n; ++twice) {
            const float offset = 0.5f * static_cast<float>(twice);
            const float got = fx::offset_quotient(offset, d, per), want = offset / d;
            bad += std::memcmp(&got, &want, sizeof got) != 0;
            ++offsets;
        }
    }
    const float low = 0x1p-100f, high = 256.0f;
    unsigned from, to;
    std::memcpy(&from, &low, 4);
    std::memcpy(&to, &high, 4);
    for (unsigned bits = from; bits < to; bits += 251) {
        float v;
        std::memcpy(&v, &bits, 4);
        const float got = fx::byte_share(v), want = v / 255.0f;
        bad += std::memcmp(&got, &want, sizeof got) != 0;
        ++shares;
    }
    for (float v = low; v > 0.0f; v *= 0.37f) bad += !(fx::byte_share(v) >= 0.0f && fx::byte_share(v) < 0x1p-100f);
    bad += fx::byte_share(0.0f) != 0.0f;
    std::printf("bad %ld of %ld offsets and %ld shares\n", bad, offsets, shares);
    return bad != 0;
}
"""


def test_quotients_equal_the_division(tmp_path):
    source, binary = tmp_path / "driver.cpp", tmp_path / "driver"
    source.write_text(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I" + CSRC, str(source), "-o", str(binary)],
                   check=True)
    done = subprocess.run([str(binary)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout
