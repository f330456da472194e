"""The library's host code on a stand-in CUDA runtime (cudart.cpp)."""
import ctypes
import os
import shutil
import subprocess

from macaw_gb300 import build as _build
from macaw_gb300 import capi

HERE = os.path.dirname(os.path.abspath(__file__))


def fake_runtime(directory):
    """Link the library's objects with the stand-in; returns the shared library's path."""
    _build.build()
    objs = [os.path.join(_build.BUILD, s.replace(".cu", ".o")) for s in _build.SOURCES]
    out = os.path.join(str(directory), "libmacaw_fake.so")
    root = os.path.dirname(os.path.dirname(os.path.realpath(_build.nvcc())))
    subprocess.run([shutil.which("g++") or "c++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic",
                    "-I", os.path.join(root, "include"), os.path.join(HERE, "cudart.cpp"), *objs, "-o", out],
                   check=True)
    return out


class Fake:
    """Controls of the stand-in of the library loaded from `path`."""

    def __init__(self, path):
        self.lib = ctypes.CDLL(path)
        self.lib.fake_log.restype = ctypes.c_char_p

    def reset(self):
        self.lib.fake_device(0)
        self.lib.fake_pending(0)
        self.lib.fake_fail(b"")
        self.lib.fake_status(0)
        self.lib.fake_clear()

    def launches(self):
        """(kernel, grid x, grid y) of the launches since the last reset or call of this."""
        lines = [x.split("@") for x in self.lib.fake_log().decode().split()]
        self.lib.fake_clear()
        return [(name, *map(int, grid.split(","))) for name, grid in lines]

    def kernels(self):
        return [x[0] for x in self.launches()]


def use(monkeypatch, path):
    """Let the Python binding load the library of fake_runtime for one test."""
    monkeypatch.setattr(capi, "LIBPATH", path)
    monkeypatch.setattr(capi, "_lib", None)
    fake = Fake(path)
    fake.reset()
    return fake
