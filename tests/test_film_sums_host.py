"""The arithmetic of the parallel ordered float sums, on the CPU (film.cu's increments are host and
device code): the sum composed from increments has the bits of the plain loop, on sequences whose
ties are counted, at even and at odd multiples of the sum's unit; and -0.0 adds nothing."""
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


@pytest.mark.parametrize("run", [1, 7, 8, 256, 1000])
@pytest.mark.parametrize("first,low", [(2.0 ** 20, 10), (2.0 ** 23, 12), (2.0 ** -3, 8), (3.0 * 2.0 ** 40, 9)])
def test_ties_go_to_even_from_either_parity(first, low, run, sums):
    """Odd multiples of half an ulp of the first addend, mixed with whole ulps and with values
    beside the tie: the sum stays in the first addend's binade, so each odd one is a tie."""
    rng = np.random.default_rng(low)
    half = np.spacing(np.float32(first)).astype(np.float64) / 2
    k = rng.integers(0, 2 ** low, 6000)
    x = (k * half).astype(np.float32)
    beside = rng.uniform(size=x.size) < 0.2
    x[beside] = np.nextafter(x[beside], np.float32(np.inf))
    x = np.concatenate([[np.float32(first)], x]).astype(np.float32)
    assert x.astype(np.float64).sum() < 2.0 ** (np.floor(np.log2(first)) + 1)
    got, redone, ties = _ordered(sums, x, run)
    assert got.view(np.int32) == _loop(x).view(np.int32)
    assert redone == 1  # the first run only, which holds the first addend
    assert min(ties) > 500, ties
