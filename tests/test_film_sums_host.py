"""The arithmetic of the parallel ordered float sums, on the CPU (film.cu's increments are host and
device code): -0.0 adds nothing, and the sum composed from increments has the bits of the plain loop."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def sums(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("film") / "libfilm_sums_host.so")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run([os.path.join(cuda, "bin", "nvcc"), "-gencode=arch=compute_103a,code=sm_103a", "-std=c++17", "-O2",
                    "-shared", "-Xcompiler", "-fPIC,-ffp-contract=off",
                    os.path.join(ROOT, "tests", "native", "film_sums_host.cu"), "-o", out], check=True,
                   capture_output=True)
    lib = ctypes.CDLL(out)
    lib.film_sums_ordered.restype = ctypes.c_float
    return lib


def _ordered(lib, x, run):
    x = np.ascontiguousarray(x, np.float32)
    redone, ties = ctypes.c_longlong(0), (ctypes.c_longlong * 2)()
    s = lib.film_sums_ordered(x.ctypes.data_as(ctypes.c_void_p), ctypes.c_longlong(x.size), run,
                              ctypes.byref(redone), ties)
    return np.float32(s), redone.value, list(ties)


def _loop(x):
    s = np.float32(0)
    with np.errstate(over="ignore"):
        for v in np.asarray(x, np.float32).ravel():
            s = np.float32(s + v)
    return s


@pytest.mark.parametrize("e", [1, 2, 24, 25, 127, 151, 253, 254])
def test_a_signed_zero_adds_nothing(e, sums):
    out = (ctypes.c_int * 2)()
    for bits in (0x00000000, 0x80000000):
        sums.film_sums_inc(ctypes.c_uint(bits), e, out)
        assert list(out) == [0, 0], f"bits {bits:#x} in binade {e}"


@pytest.mark.parametrize("run", [1, 8, 256, 1000])
def test_signed_zeros_take_no_run_out_of_the_scheme(run, sums):
    rng = np.random.default_rng(1)
    x = rng.uniform(0.5, 1.0, 20000).astype(np.float32)
    x[::3] = 0.0
    want, plain, _ = _ordered(sums, x, run)
    x[::3] = -0.0
    got, redone, _ = _ordered(sums, x, run)
    assert got.view(np.int32) == want.view(np.int32) == _loop(x).view(np.int32)
    assert redone == plain
