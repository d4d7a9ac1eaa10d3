"""Reinhard's ordered channel sums on images with signed zeros and with many exact ties: the bits
of the oracle, which adds one pixel after another in float."""
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


def _ties(x):
    """Exact ties of the ordered float sum of x that leave it in its binade, by the parity of the
    sum's multiple of its unit."""
    s, count = np.float32(0), [0, 0]
    for v in x:
        r = np.float32(s + v)
        half = np.spacing(s) / np.float32(2)
        exact = np.float64(s) + np.float64(v)  # multiples of half, fewer than 2^53 of them
        if np.spacing(r) == np.spacing(s) and abs(exact - np.float64(r)) == np.float64(half):
            count[int(s.view(np.int32)) & 1] += 1
        s = r
    return count


@pytest.mark.parametrize("pixels", [3000, 30011])
@pytest.mark.parametrize("first,low", [(2.0 ** 20, 9), (2.0 ** 23, 8), (3.0 * 2.0 ** 40, 7)])
def test_reinhard_sums_round_ties_to_even_from_either_parity(first, low, pixels, cuda_device):
    """A large first pixel, then multiples of half its ulp, odd and even ones: the sums of r, g and
    b stay in its binade, so every odd multiple is a tie, over one chunk of pixels and over many."""
    rng = np.random.default_rng(low)
    half = np.spacing(np.float32(first)).astype(np.float64) / 2
    img = (rng.integers(0, 2 ** low, (1, pixels, 3)) * half).astype(np.float32)
    img[0, 0] = first
    for c in range(3):
        assert min(_ties(img[0, :, c])) > pixels // 12
    _check(img)
