"""The bin guess of the centre-per-lane passes, on the CPU: for bins that start
at 0 whose thresholds lie within 1/256 of a bin of their edges, the category of
every d^2 up to R^2 is the guess g = floor(sqrt(d^2) * scale + 1/2) or g + 1,
also with the root off by 2^-23 and the product by an eighth of a bin, and one
compare with the threshold of g + 1 decides."""
import numpy as np
import pytest


def category(d2, nbins, rmax):
    """The histogram's category: 1 + bin, nbins + 1 at and above rmax."""
    x = np.sqrt(d2.astype(np.float32)).astype(np.float64)
    b = np.floor((x * (1.0 / rmax * nbins)).astype(np.float32)).astype(np.int64)
    return np.where((x <= rmax) & (b < nbins), 1 + b, nbins + 1)


def thresholds(nbins, rmax):
    """The smallest d^2 of each category, by bisection over the bit patterns."""
    k = np.arange(1, nbins + 2)
    lo = np.zeros(k.size, dtype=np.int64)
    hi = np.full(k.size, np.float32(4.0 * rmax * rmax).view(np.int32), dtype=np.int64)
    while np.any(lo < hi):
        mid = (lo + hi) // 2
        up = category(mid.astype(np.int32).view(np.float32), nbins, rmax) >= k
        lo, hi = np.where(up | (lo >= hi), lo, mid + 1), np.where(up & (lo < hi), mid, hi)
    return np.concatenate([[0.0], lo.astype(np.int32).view(np.float32), [np.inf]]).astype(np.float32)


@pytest.mark.parametrize("rmax,rincr", [(1.0, 0.01), (2.0, 0.005), (2.5, 0.01), (1.569, 0.037), (0.7, 0.0007)])
def test_guess_and_one_threshold_name_the_category(rmax, rincr):
    rmax, rincr = float(np.float32(rmax)), float(np.float32(rincr))
    nbins = int(rmax / rincr)
    T = thresholds(nbins, rmax)
    scale = np.float32(1.0 / rmax * nbins)
    edge = np.sqrt(T[1:-1].astype(np.float64)) * float(scale)
    assert np.abs(edge - np.arange(nbins + 1)).max() < 1 / 256  # the rule applies
    rng = np.random.default_rng(nbins)
    top = np.float32(rmax) * np.float32(rmax)
    bits = T[1:-1].view(np.int32).astype(np.int64)
    near = np.clip(bits[:, None] + np.arange(-4, 5), 0, top.view(np.int32)).ravel()
    d2 = np.concatenate([near.astype(np.int32).view(np.float32), rng.uniform(0, top, 50000).astype(np.float32), [0, top]])
    d2 = d2[d2 <= top]
    want = category(d2, nbins, rmax)
    root = np.sqrt(d2.astype(np.float64))
    for rel in (-2.0 ** -23, 0.0, 2.0 ** -23):
        for off in (-0.125, 0.0, 0.125):
            g = np.clip(np.floor(root * (1 + rel) * float(scale) + 0.5 + off), 0, nbins + 1).astype(np.int64)
            assert np.all((want == g) | (want == g + 1))
            assert np.array_equal(g + (T[g + 1] <= d2), want)
