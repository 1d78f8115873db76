"""CPU: a fresh buffer's pages are resident once they have been mapped.

csrc/host_pages.h asks the kernel for a caller's whole range before the GPU
copies into it.  The test asks the kernel which pages of a fresh mapping are
resident (mincore) before and after, for ranges that begin and end inside a
page; it is skipped where the kernel does not know the request.
"""

from __future__ import annotations

import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fractal-audio-viz_gb300", "csrc")

DRIVER = r"""
#include "host_pages.h"
#include <cerrno>
#include <cstdio>
#include <vector>
int main() {
    const std::size_t page = static_cast<std::size_t>(sysconf(_SC_PAGESIZE)), pages = 512, size = pages * page;
    for (const std::size_t start : {std::size_t{0}, std::size_t{1}, 3 * page + 17, 200 * page - 1}) {
        for (const std::size_t length : {fgb::kMapFrom, 5 * page + 3 + fgb::kMapFrom, size - 300 * page}) {
            void* m = mmap(nullptr, size, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
            if (m == MAP_FAILED) return 2;
            madvise(m, size, MADV_NOHUGEPAGE);
            std::vector<unsigned char> resident(pages);
            if (mincore(m, size, resident.data()) != 0) return 2;
            for (unsigned char r : resident) {
                if (r & 1) return 3;
            }
            fgb::map_pages(static_cast<char*>(m) + start, length);
            if (mincore(m, size, resident.data()) != 0) return 2;
            const std::size_t first = start / page, end = (start + length + page - 1) / page;
            for (std::size_t i = 0; i < pages; ++i) {
                const bool want = i >= first && i < end;
                if (((resident[i] & 1) != 0) != want) {
                    std::printf("start %zu length %zu: page %zu %s resident\n", start, length, i, want ? "not" : "is");
                    void* probe = mmap(nullptr, page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
                    return madvise(probe, page, 23) != 0 && errno == EINVAL ? 77 : 1;
                }
            }
            munmap(m, size);
        }
    }
    return 0;
}
"""


def test_mapped_pages_are_resident(tmp_path):
    source, binary = tmp_path / "driver.cpp", tmp_path / "driver"
    source.write_text(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + CSRC, str(source), "-o", str(binary)], check=True)
    done = subprocess.run([str(binary)], capture_output=True, text=True)
    if done.returncode == 77:
        pytest.skip("the kernel does not map a range on request")
    assert done.returncode == 0, done.stdout
