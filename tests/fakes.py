"""A Python process with failing CUDA runtime calls (tests/native/fake_cuda.c,
TEST INFRASTRUCTURE): ``run`` executes a snippet there, in which ``fake`` is
the preloaded library's handle, and returns what it printed."""
from __future__ import annotations

import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

HEAD = """
import ctypes as C, sys
import numpy as np
sys.path[:0] = [{root!r}, {tests!r}]
class _Fake:
    lib = C.CDLL({lib!r})
    def __setattr__(self, name, value):
        C.c_int.in_dll(self.lib, name).value = value
    def __getattr__(self, name):
        return C.c_int.in_dll(self.lib, name).value
fake = _Fake()
"""


def _library() -> str:
    from opencal_gb300 import nvbuild
    src = os.path.join(HERE, "native", "fake_cuda.c")
    out = os.path.join(HERE, "native", "build", "libfake_cuda.so")
    if not os.path.exists(out) or os.path.getmtime(out) < os.path.getmtime(src):
        os.makedirs(os.path.dirname(out), exist_ok=True)
        cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvbuild.nvcc())))
        subprocess.run([os.environ.get("CC", "gcc"), "-shared", "-fPIC", "-O1", "-I" + os.path.join(cuda, "include"),
                        "-o", out, src, "-L" + os.path.join(cuda, "lib64"), "-Wl,--no-as-needed", "-lcudart", "-ldl",
                        "-Wl,-rpath," + os.path.join(cuda, "lib64")], check=True)
    return out


def run(code: str, timeout: float = 300) -> str:
    lib = _library()
    env = dict(os.environ, LD_PRELOAD=lib)
    r = subprocess.run([sys.executable, "-c", HEAD.format(root=ROOT, tests=HERE, lib=lib) + code], env=env, cwd=ROOT,
                       capture_output=True, text=True, timeout=timeout)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
