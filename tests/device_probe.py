"""The library's scalar device functions over arrays (tests/device/probe.cu), for the
tests that hold them against the operations they stand for."""
import ctypes as C
import functools
import os
import subprocess
import tempfile

import numpy as np
import pytest

from hbtplus_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


class Probe:
    def __init__(self, path):
        self.lib = C.CDLL(path)

    def call(self, name, x, out, *args):
        """name(x, [more arrays,] n, scalars..., got, want): the function's results over the
        rows and those of the operation it stands for."""
        arrays = [np.ascontiguousarray(a) for a in (x, *args) if isinstance(a, np.ndarray)]
        scalars = [C.c_float(a) if isinstance(a, np.float32) else
                   C.c_double(a) if isinstance(a, float) else a
                   for a in args if not isinstance(a, np.ndarray)]
        n = len(arrays[0])
        got, want = np.zeros(n, out), np.zeros(n, out)
        assert getattr(self.lib, name)(*(C.c_void_p(a.ctypes.data) for a in arrays), n, *scalars,
                                       C.c_void_p(got.ctypes.data),
                                       C.c_void_p(want.ctypes.data)) == 0
        return got, want

    @staticmethod
    def same_bits(got, want, *inputs):
        bits = np.uint64 if got.dtype == np.float64 else np.uint32
        bad = np.flatnonzero(got.view(bits) != want.view(bits))
        assert not len(bad), (len(bad), [(got[i], want[i], *(a[i] for a in inputs))
                                         for i in bad[:5]])


@functools.cache
def _build():
    folder = tempfile.TemporaryDirectory()
    so = os.path.join(folder.name, "probe.so")
    r = subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-shared", "--cudart", "static", "-o", so,
                        os.path.join(HERE, "device", "probe.cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return Probe(so), folder


@pytest.fixture(scope="session")
def probe():
    return _build()[0]
