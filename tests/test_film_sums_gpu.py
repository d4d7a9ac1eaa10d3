"""Reinhard's channel means are float sums in pixel order; the parallel sums must give their
bits.  Images that reach each of its branches: ends of chunks, ties (up and down with the
parity of the sum), many additions below half an ulp, zeros in front, subnormals, addends far
larger than the sum, sums that overflow, and the channels it hands to one thread (negative,
infinite, NaN).  The oracle sums one pixel after another in float."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _flat(n, value):
    return np.full((1, n, 3), value, np.float32)


def _case(name):
    rng = np.random.default_rng(3)
    if name.startswith("pixels"):
        return rng.uniform(0.0, 4.0, (1, int(name[6:]), 3)).astype(np.float32)
    img = rng.uniform(0.0, 1.0, (61, 257, 3)).astype(np.float32)
    if name == "ones":          # exact up to 2^24
        return _flat(70001, 1.0)
    if name == "ties":          # 1 + odd multiples of 2^-23 against sums of every parity
        return (1.0 + 2.0 ** -23 * rng.integers(0, 2, (40, 1001, 3))).astype(np.float32)
    if name == "half_ulp":      # additions of exactly half an ulp of a large sum, and just beside it
        img = np.full((33, 999, 3), 0.5, np.float32)
        img[0, 0] = 2.0 ** 23
        img[::2] = np.nextafter(np.float32(0.5), np.float32(1.0))
        return img
    if name == "below":         # everything after the first pixel is lost
        img[:] = 1e-3
        img[0, 0] = 1e6
        return img
    if name == "dark_lead":
        img[:40] = 0.0
        return img
    if name == "subnormal":
        return (img * np.float32(1e-41)).astype(np.float32)
    if name == "jumps":         # each binade entered by a large step
        img[:] = 0.0
        img.reshape(-1, 3)[::700] = (2.0 ** np.arange(0, 23)).reshape(-1, 1)[:len(img.reshape(-1, 3)[::700])]
        return img
    if name == "wide":
        return np.exp2(rng.uniform(-30, 30, img.shape)).astype(np.float32)
    if name == "overflow":
        return _flat(5000, 3e38)
    if name == "negative":
        img[3, 5] = (-2.0, 0.5, 0.25)
        return img
    if name == "infinite":
        img[7, 9, 1] = np.inf
        return img
    if name == "nan":
        img[60, 3, 2] = np.nan
        return img
    raise ValueError(name)


@pytest.mark.parametrize("name", ["pixels1", "pixels7", "pixels2047", "pixels2048", "pixels2049", "pixels4097",
                                  "pixels785001", "ones", "ties", "half_ulp", "below", "dark_lead", "subnormal",
                                  "jumps", "wide", "overflow", "negative", "infinite", "nan"])
def test_reinhard_means_keep_the_bits_of_the_ordered_sum(name, cuda_device):
    from mcrt_gb300 import film
    from oracle import oracle as O
    img = _case(name)
    want = O.film_tonemap(img, True)
    got = film.tonemap(img.copy(), "reinhard")
    nan = np.isnan(want)
    assert np.array_equal(nan, np.isnan(got))
    assert np.array_equal(got[~nan].view(np.int32), want[~nan].view(np.int32))
