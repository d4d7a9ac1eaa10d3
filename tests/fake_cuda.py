"""The library's host code over a stand-in for the CUDA runtime (tests/native/fake_cudart.cpp), for
CPU tests of the order of its work, of its error paths and of which kernels a call takes."""
import ctypes
import glob
import os
import shutil
import subprocess

from conftest import ROOT


def build(folder: str) -> str:
    """Links the library's objects (built if need be) with the stand-in; returns the library."""
    from mcrt_gb300 import native_build
    native_build.build()
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    out = os.path.join(folder, "libmcrt_fake.so")
    objs = [os.path.join(native_build.LIB_DIR, s + ".o") for s in native_build.CU_SOURCES + native_build.CPP_SOURCES]
    # -Bsymbolic: the stand-in's functions also where another library of the process has these names
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread", f"-I{cuda}/include",
                    os.path.join(ROOT, "tests", "native", "fake_cudart.cpp"), *objs, "-Wl,-Bsymbolic",
                    "-Wl,--no-undefined", "-o", out], check=True, capture_output=True)
    return out


class Fake:
    """One instance of the library with its own process-wide state, in the package's place."""

    def __init__(self, built: str, monkeypatch):
        from mcrt_gb300 import _native as N
        folder = os.path.dirname(built)
        path = os.path.join(folder, f"instance{len(glob.glob(os.path.join(folder, 'instance*')))}.so")
        shutil.copy(built, path)
        self.lib = ctypes.CDLL(path)
        for name, (res, args) in N.EXPORTS.items():
            fn = getattr(self.lib, name)
            fn.restype, fn.argtypes = res, args
        for name in ("fake_pending", "fake_nulls", "fake_open_captures"):
            getattr(self.lib, name).restype = ctypes.c_longlong
        self.lib.fake_launch.restype = ctypes.c_char_p
        monkeypatch.setattr(N, "_lib", self.lib)

    def fail(self, function: str, nth: int = 1, error: int = 2):
        """The nth next call of `function` fails (2: out of memory)."""
        self.lib.fake_fail(function.encode(), nth, error)

    def polls_read(self, value: int):
        """What a copy to page-locked memory brings: the finished-path counter."""
        self.lib.fake_poll(ctypes.c_longlong(value))

    def kernels(self) -> list:
        """The kernels launched since the last call, by name."""
        names = [self.lib.fake_launch(i).decode() for i in range(self.lib.fake_launches())]
        self.lib.fake_forget()
        return names
