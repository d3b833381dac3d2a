"""Bounds and fall-backs of the centre-per-lane passes: results at the limits of
their counters, and what a pass does without the buffers only its faster form
needs.  Counts are whole numbers and must be equal."""
import numpy as np
import pytest

from paraprobe_gb300 import native as N

pytestmark = pytest.mark.gpu


def _pairs(types):
    return [[a] for a in types for b in types], [[b] for a in types for b in types]


def test_sparse_bins_of_one_lattice(ctx):
    """More than 2^16 centres a block of the grid, all of whose nearest sparse
    ions fall in one bin: a cubic lattice with every 64th site of type 2.  The
    bin counts every centre; nothing spills into the bins beside it."""
    side, a = 220, 0.25
    assert side ** 3 > ctx.sm_count() * 65536
    g = np.arange(side, dtype=np.float32) * np.float32(a)
    xyz = np.empty((side, side, side, 3), dtype=np.float32)
    xyz[..., 0], xyz[..., 1], xyz[..., 2] = g[:, None, None], g[None, :, None], g[None, None, :]
    labels = np.ones((side, side, side), dtype=np.uint8)
    labels[2::4, 2::4, 2::4] = 2  # at most 3.47 a from any site, 4 a from one another
    n, n2 = labels.size, int((labels == 2).sum())
    cid = ctx.upload(xyz.reshape(-1, 3), labels.reshape(-1))
    ctx.surfdist(cid, np.full(n, 100.0, dtype=np.float32))
    trg, env = _pairs((1, 2))
    ctx.tasks(trg, env)
    ctx.hist(0.0, 5 * a, 7 * a)  # one bin [0, 5 a) and what lies above
    try:
        ctx.set_option("knn_walks", 1)
        ctx.run(cid, N.PP_1NN)
        one, tests = ctx.fetch(), ctx.run_tests()
        ctx.set_option("knn_walks", 2)
        ctx.run(cid, N.PP_1NN)
        two = ctx.fetch()
        assert ctx.run_tests() != tests  # two walks and a count, not one walk
    finally:
        ctx.set_option("knn_walks", 0)
        ctx.free(cid)
    want = np.zeros((4, 3), dtype=np.uint64)
    want[:, 1] = [n - n2, n - n2, n2, n2]  # (1, 1), (1, 2), (2, 1), (2, 2)
    assert np.array_equal(one.reshape(4, 3), want)
    assert np.array_equal(two.reshape(4, 3), want)
