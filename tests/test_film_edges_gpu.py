"""Reinhard's ordered channel sums on images with signed zeros: the bits of the oracle, which adds
one pixel after another in float."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(img):
    from mcrt_gb300 import film
    from oracle import oracle as O
    want = O.film_tonemap(img, True)
    got = film.tonemap(img.copy(), "reinhard")
    nan = np.isnan(want)
    assert np.array_equal(nan, np.isnan(got))
    assert np.array_equal(got[~nan].view(np.int32), want[~nan].view(np.int32))


@pytest.mark.parametrize("share", [0.01, 0.5, 1.0])
@pytest.mark.parametrize("pixels", [1, 2047, 2049, 30011])
def test_signed_zeros_in_reinhard_sums(pixels, share, cuda_device):
    rng = np.random.default_rng(pixels)
    img = rng.uniform(0.0, 2.0, (1, pixels, 3)).astype(np.float32)
    img[rng.uniform(size=img.shape) < share] = -0.0
    _check(img)
