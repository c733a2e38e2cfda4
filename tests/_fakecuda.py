"""The library's host code on a runtime without a GPU (tests/fake_cudart.cpp).

``load()`` links the library's own objects with that runtime and returns the
ctypes library with the API's signatures and the ``fake_*`` controls.
"""
from __future__ import annotations

import ctypes
import os
import subprocess
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
OOM = 2  # cudaErrorMemoryAllocation
_lib = _dir = None


def load():
    global _lib, _dir
    if _lib is not None:
        return _lib
    from amrvac_b200 import _lib as api
    from amrvac_b200 import build
    build.build()
    objs = [os.path.join(build.BUILD, u.replace(".cu", ".o")) for u in build.UNITS]
    if not all(os.path.exists(o) for o in objs):
        build.build(force=True)
    _dir = tempfile.TemporaryDirectory()
    out = os.path.join(_dir.name, "libfake.so")
    inc = os.path.join(os.path.dirname(os.path.dirname(build.NVCC)), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", inc, "-o", out,
                    os.path.join(HERE, "fake_cudart.cpp"), *objs], check=True)
    L = ctypes.CDLL(out)
    for name, res, args in api.SIGNATURES:
        fn = getattr(L, name)
        fn.restype, fn.argtypes = res, args
    L.fake_log.restype = ctypes.c_char_p
    L.fake_used.restype = ctypes.c_size_t
    L.fake_capacity.argtypes = [ctypes.c_size_t]
    _lib = L
    return L


class Fake:
    """One test's view: a fresh log, contexts made through the C API."""

    def __init__(self):
        self.L = load()
        self.L.fake_reset()

    def create(self, **kw):
        from amrvac_b200 import make_cfg
        h = ctypes.c_void_p()
        cfg = make_cfg(**kw)
        assert self.L.amrvac_gpu_create(ctypes.byref(cfg), ctypes.byref(h)) == 0, self.error()
        return h

    def grid(self, h, n):
        import numpy as np
        nx = (ctypes.c_int * 3)(*(list(n) + [1] * (3 - len(n))))
        lo, hi = np.zeros(3), np.ones(3)
        dp = ctypes.POINTER(ctypes.c_double)
        return self.L.amrvac_gpu_set_uniform_grid(h, nx, lo.ctypes.data_as(dp), hi.ctypes.data_as(dp))

    def error(self):
        return self.L.amrvac_gpu_last_error().decode()

    def fail(self, fn, after=0, times=1, err=OOM):
        self.L.fake_fail(fn.encode(), after, times, err)

    def log(self):
        return self.L.fake_log().decode().splitlines()

    def clear(self):
        self.L.fake_clear_log()
