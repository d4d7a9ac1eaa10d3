import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

GOLDEN = os.path.join(ROOT, "tests", "golden")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (sm_103a) and the native library")


def pytest_collection_modifyitems(items):
    """The seam tests run the reference's own renderer over this library.  Where neither its sources
    nor a build of them are present they cannot run, as the other tests that need the reference."""
    from oracle.oracle import SEAM_SO
    from oracle.stage_reference import checkout_dir, source_dir
    if os.path.exists(SEAM_SO) or checkout_dir() is not None or source_dir() is not None:
        return
    for item in items:
        if item.path.name == "test_seams_gpu.py":
            item.add_marker(pytest.mark.skip(reason="reference sources not present on this machine"))


def golden(name: str):
    return np.load(os.path.join(GOLDEN, name))


@pytest.fixture(scope="session")
def native():
    from mcrt_gb300 import _native
    return _native.load()


@pytest.fixture(scope="session")
def cuda_device():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("a gpu-marked test ran without a CUDA device")
    torch.cuda.init()
    return torch.device("cuda:0")
