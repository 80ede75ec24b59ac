"""The device-side helpers of the GPU tests (tests/device_forms.cu), compiled on first use."""
import ctypes
import functools
import os
import subprocess
import tempfile

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
