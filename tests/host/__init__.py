"""The library's host code on a CUDA runtime without a device (fake_cuda.cpp)."""
import ctypes
import os
import subprocess

from ivr_gb300 import _lib, api, build

HERE = os.path.dirname(os.path.abspath(__file__))
SOURCES = ["ivr_api.cpp", "ivr_frame.cpp", "ivr_colormap.cpp", "ivr_learn.cpp"]


def load(directory) -> ctypes.CDLL:
    """Compiles the host code with the stand-in runtime and declares what it
    exports of the ABI, and the stand-in's own controls."""
    so = os.path.join(str(directory), "libivr_host.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fPIC", "-shared", "-ffp-contract=off", "-Wl,-Bsymbolic",
                    "-I" + os.path.join(build.ROOT, "include"), "-I" + build.CSRC, "-I" + build.CUDA_INC,
                    *[os.path.join(build.CSRC, s) for s in SOURCES], os.path.join(HERE, "fake_cuda.cpp"), "-o", so],
                   check=True)
    lib = ctypes.CDLL(so)
    for name, (res, args) in _lib.SIGNATURES.items():
        fn = getattr(lib, name, None)  # (the server is not part of it)
        if fn is not None:
            fn.restype, fn.argtypes = res, args
    lib.fake_first_race.restype = ctypes.c_char_p
    for name in ("fake_in_use", "fake_mallocs", "fake_launches", "fake_early"):
        getattr(lib, name).restype = ctypes.c_size_t
    lib.fake_capacity.argtypes = [ctypes.c_size_t]
    lib.fake_fail_malloc.argtypes = lib.fake_fail_more.argtypes = lib.fake_fail_launch.argtypes = [ctypes.c_long]
    lib.cudaStreamCreateWithFlags.argtypes = [ctypes.POINTER(ctypes.c_void_p), ctypes.c_uint]
    lib.cudaDeviceSynchronize.argtypes = []
    lib.cudaStreamBeginCapture.argtypes = [ctypes.c_void_p, ctypes.c_int]
    lib.cudaStreamEndCapture.argtypes = [ctypes.c_void_p, ctypes.POINTER(ctypes.c_void_p)]
    return lib


class HostContext(api.Context):
    """api.Context on such a library."""

    def __init__(self, lib, hbm_budget: int = 0):
        self.lib = lib
        h = ctypes.c_void_p()
        assert lib.ivr_create(0, hbm_budget, ctypes.byref(h)) == 0
        self.h = h

    def stream(self) -> int:
        s = ctypes.c_void_p()
        assert self.lib.cudaStreamCreateWithFlags(ctypes.byref(s), 1) == 0
        return s.value
