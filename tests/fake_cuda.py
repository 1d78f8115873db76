"""The library's host side on a stand-in CUDA runtime (fake_cuda.cpp)."""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
import textwrap

from .conftest import PACKAGE_DIR, ROOT

PRELUDE = """
import ctypes, sys
sys.path.insert(0, {root!r})
from tests.conftest import load_package
package = load_package()
native = package.native
lib = native.load({path!r}, gb300=True)
lib.fake_stream.restype = ctypes.c_void_p
for name in ("fake_launches", "fake_hazards", "fake_allocated", "fake_uploaded", "fake_mapped"):
    getattr(lib, name).restype = ctypes.c_longlong
def check(status):
    assert status == 0, native.last_error(lib)
"""


def cuda_include() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")


def link(package, directory) -> str:
    """The library's objects with the stand-in runtime; returns the path."""
    built = os.path.dirname(package.build())
    sources = sorted(os.listdir(os.path.join(PACKAGE_DIR, "csrc")))
    objects = [os.path.join(built, name + ".o") for name in sources if name.endswith((".cu", ".cpp"))]
    include = cuda_include()
    path = os.path.join(str(directory), "libfake.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I" + include,
                    os.path.join(ROOT, "tests", "fake_cuda.cpp"), *objects, "-o", path, "-ldl", "-lpthread"], check=True)
    return path


def run(path: str, code: str) -> str:
    """`code` in a fresh process with the library loaded as `lib`."""
    source = PRELUDE.format(root=ROOT, path=path) + textwrap.dedent(code)
    done = subprocess.run([sys.executable, "-c", source], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout + done.stderr
    return done.stdout
