"""CPU: mapping a caller's pages (csrc/host_pages.h) changes no byte.

Ranges of a mapping with written, fresh, read-only and unmapped neighbours,
aligned and not, from below the size limit up: the bytes stay as they were,
and what cannot be mapped is left alone.
"""

from __future__ import annotations

import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fractal-audio-viz_gb300", "csrc")

DRIVER = r"""
#include "host_pages.h"
#include <cstdio>
#include <cstdlib>
#include <cstring>
int main() {
    const std::size_t page = static_cast<std::size_t>(sysconf(_SC_PAGESIZE)), size = 64 * page + (1 << 20);
    auto* m = static_cast<unsigned char*>(mmap(nullptr, size, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
    if (m == MAP_FAILED) return 2;
    for (std::size_t i = 0; i < size; i += 3 * page + 17) m[i] = static_cast<unsigned char>(i * 7 + 1);
    unsigned char* copy = static_cast<unsigned char*>(std::malloc(size));
    std::memcpy(copy, m, size);
    munmap(m + size / page * page - page, page);
    const std::size_t kept = size / page * page - page;
    mprotect(m + 20 * page, page, PROT_READ);
    int bad = 0;
    const std::size_t starts[] = {0, 1, 37, page, 5 * page + 9, 19 * page + 3};
    const std::size_t lengths[] = {0, 1, fgb::kMapFrom - 1, fgb::kMapFrom, 3 * page + 1, size / 2, size};
    for (std::size_t start : starts) {
        for (std::size_t length : lengths) {
            fgb::map_pages(m + start, length);
            if (std::memcmp(m, copy, kept) != 0) ++bad;
        }
    }
    fgb::map_pages(nullptr, 1 << 20);
    std::printf("bad %d\n", bad);
    return bad != 0;
}
"""


def test_mapping_pages_changes_no_byte(tmp_path):
    source, binary = tmp_path / "driver.cpp", tmp_path / "driver"
    source.write_text(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + CSRC, str(source), "-o", str(binary)], check=True)
    done = subprocess.run([str(binary)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout
