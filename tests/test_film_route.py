"""Which kernels Reinhard tone mapping launches: an image of one chunk of 2,048 pixels is summed by
one kernel, larger ones by three.  On the CPU, over a stand-in for the CUDA runtime."""
import re

import numpy as np
import pytest

import fake_cuda


@pytest.fixture(scope="module")
def built(tmp_path_factory):
    return fake_cuda.build(str(tmp_path_factory.mktemp("fake")))


@pytest.mark.parametrize("pixels,sums", [(1, 1), (527, 1), (2047, 1), (2048, 1), (2049, 3), (4097, 3)])
def test_reinhard_kernels_by_image_size(pixels, sums, built, monkeypatch):
    from mcrt_gb300 import film
    cuda = fake_cuda.Fake(built, monkeypatch)
    film.tonemap(np.ones((1, pixels, 3), np.float32), "reinhard")
    names = [re.search(r"k_film_[a-z_]+", k).group() for k in cuda.kernels()]
    means = next(i for i, k in enumerate(names) if k.startswith("k_film_means"))
    assert means == sums - 1 and len(names) == sums + 1
    assert cuda.lib.fake_pending() == 0
