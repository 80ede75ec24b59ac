"""The device-side helpers of the GPU tests (tests/device_forms.cu), compiled on first use."""
import ctypes
import functools
import os
import subprocess
import tempfile

import numpy as np

from medusa_b200 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


@functools.lru_cache(maxsize=None)
def library() -> ctypes.CDLL:
    out = os.path.join(tempfile.mkdtemp(prefix="device_forms"), "device_forms.so")
    subprocess.check_call([B.nvcc(), "-shared", os.path.join(HERE, "device_forms.cu"), "-o", out, "-std=c++17", "-O2",
                           "-Xcompiler", "-fPIC", "-I", B.CSRC, "-I", B.INCLUDE] + B.ARCH)
    L = ctypes.CDLL(out)
    L.hold_start.argtypes = [ctypes.c_int] * 4
    L.hold_start.restype = ctypes.c_void_p
    L.hold_running.argtypes = [ctypes.c_void_p]
    L.hold_end.argtypes = [ctypes.c_void_p]
    L.faces.argtypes = [ctypes.c_longlong, ctypes.c_double, ctypes.c_void_p, ctypes.c_void_p]
    for f in (L.form_f32, L.form_f64):
        f.argtypes = [ctypes.c_int, ctypes.c_longlong] + [ctypes.c_void_p] * 3
    return L


class Hold:
    """`sms` SMs filled for `ms` milliseconds, one CTA each, on a stream of its own; running()
    says whether they still are.  Ends by itself."""

    def __init__(self, sms: int, threads: int, smem: int, ms: int):
        self._L = library()
        self._h = self._L.hold_start(sms, threads, smem, ms)
        assert self._h, "hold_start failed"

    def __enter__(self):
        return self

    def running(self) -> bool:
        return bool(self._L.hold_running(self._h))

    def __exit__(self, *a):
        self._L.hold_end(self._h)


def form(k: int, a: np.ndarray, b: np.ndarray) -> np.ndarray:
    """The sweeps' arithmetic helper k of the arrays' type on the GPU (form_kernel)."""
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b, dtype=a.dtype)
    out = np.empty_like(a)
    f = library().form_f32 if a.dtype == np.float32 else library().form_f64
    assert f(k, b.size, a.ctypes.data, b.ctypes.data, out.ctypes.data) == 0
    return out


def faces(gam: float, states: np.ndarray) -> np.ndarray:
    """[n][2][3] states to [n][13]: face_kernel's columns."""
    states = np.ascontiguousarray(states, dtype=np.float64)
    out = np.empty((states.shape[0], 13))
    assert library().faces(states.shape[0], gam, states.ctypes.data, out.ctypes.data) == 0
    return out
