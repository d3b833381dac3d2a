"""Bounds and fall-backs of the centre-per-lane passes: results at the limits of
their counters, and what a pass does without the buffers only its faster form
needs.  Counts are whole numbers and must be equal."""
import numpy as np
import pytest

from paraprobe_gb300 import native as N
from paraprobe_gb300 import synth

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


@pytest.mark.parametrize("flags", [N.PP_RDF, N.PP_MKNN, N.PP_RDF | N.PP_MKNN])
@pytest.mark.parametrize("symmetric", [1, 0])
def test_passes_without_their_scratch(ctx, oracle, flags, symmetric):
    """A device without room for the buffers of a pass's faster form: whichever
    of them is the first that is missing, the pass gives the same counts, and
    one that ends up on the per-centre scan prepares nothing it does not use."""
    spec = synth.cylinder_specimen(n=24000, radius=3.0, height=18.0, fractions=(0.95, 0.04, 0.01), seed=11, nseg=48,
                                   stack=4.0)
    d2 = np.where(np.arange(len(spec.xyz)) % 11 == 0, 1.0, 10.0).astype(np.float32)
    trg, env = _pairs((1, 2, 3))
    hist, ks = (0.0, 0.01, 1.5), [9, 1] if flags & N.PP_MKNN else []
    cid = ctx.upload(spec.xyz, spec.labels)
    ctx.surfdist(cid, d2)
    ctx.tasks(trg, env)
    ctx.hist(*hist)
    ctx.set_option("symmetric", symmetric)
    ctx.set_option("knn_walks", 2)

    def run():
        before = N.kernel_launches()
        ctx.run(cid, flags, ks)
        return ctx.fetch(), ctx.stats(), ctx.last_kernel(), N.kernel_launches() - before, ctx.run_tests()

    try:
        run()
        ctx.set_option("lanes", 0)
        scan = run()
        ctx.set_option("lanes", 1)
        got = []
        for limit in range(8):
            ctx.set_option("scratch", limit)
            got.append(run())
        ctx.set_option("scratch", -1)
        got.append(run())
    finally:
        for name, value in (("symmetric", 1), ("knn_walks", 0), ("lanes", 1), ("scratch", -1)):
            ctx.set_option(name, value)
        ctx.free(cid)
    ref = oracle.spatstat(spec.xyz, spec.labels, d2, *hist, flags, trg, env, ks)
    for bins, st, *_ in [scan] + got:
        assert np.array_equal(bins, ref["bins"]) and st["pairs"] == ref["pairs"] and st["centres"] == ref["centres"]
    assert scan[2] == got[0][2] == "k_scan" and scan[3] == got[0][3]
    assert got[-1][2] != "k_scan"
    if flags & N.PP_MKNN:  # two walks, one walk without the sparse list, the per-centre scan
        assert len({g[4] for g in got}) == 3


@pytest.mark.parametrize("flags", [N.PP_MKNN, N.PP_MKNN | N.PP_RDF])
@pytest.mark.parametrize("fractions", [(0.97, 0.02, 0.01), (0.5, 0.45, 0.05)])
@pytest.mark.parametrize("ks", [[8, 1], [10, 1], [16, 2], [20, 19]])
def test_two_walks_when_asked_for(ctx, oracle, flags, fractions, ks):
    """knn_walks = 2 takes two walks wherever the sets allow, also where one walk
    would be the cheaper: the tests it counts are others than one walk's."""
    spec = synth.cylinder_specimen(n=24000, radius=3.0, height=18.0, fractions=fractions, seed=5, nseg=48, stack=4.0)
    d2 = np.full(len(spec.xyz), 10.0, dtype=np.float32)
    trg, env = _pairs((1, 2, 3))
    hist = (0.0, 0.01, 1.5)
    cid = ctx.upload(spec.xyz, spec.labels)
    ctx.surfdist(cid, d2)
    ctx.tasks(trg, env)
    ctx.hist(*hist)
    try:
        tests, bins = {}, {}
        for walks in (1, 2):
            ctx.set_option("knn_walks", walks)
            ctx.run(cid, flags, ks)
            bins[walks], tests[walks] = ctx.fetch(), ctx.run_tests()
    finally:
        ctx.set_option("knn_walks", 0)
        ctx.free(cid)
    assert tests[1] != tests[2]
    ref = oracle.spatstat(spec.xyz, spec.labels, d2, *hist, flags, trg, env, ks)
    assert np.array_equal(bins[1], ref["bins"]) and np.array_equal(bins[2], ref["bins"])


@pytest.mark.parametrize("flags,ks", [(N.PP_RDF, []), (N.PP_MKNN, [10, 1]), (N.PP_RDF | N.PP_MKNN, [20, 2])])
@pytest.mark.parametrize("symmetric,walks", [(1, 2), (0, 1)])
@pytest.mark.parametrize("sigma", [0.05, 0.3, 0.8])
def test_chunks_shared_by_warps(ctx, oracle, flags, ks, symmetric, walks, sigma):
    """A ball of very many ions in a thin cloud, down to one cell of them: its
    chunks are listed and shared, and every batch is taken once."""
    rng = np.random.default_rng(8)
    xyz = rng.uniform(0, 14, (20000, 3))
    xyz[:4000] = [7.1, 6.9, 7.0] + sigma * rng.normal(size=(4000, 3))
    xyz = rng.permutation(xyz).astype(np.float32)
    n = len(xyz)
    labels = rng.choice(np.array([1, 2, 3], dtype=np.uint8), n, p=[0.9, 0.07, 0.03])
    d2 = np.where(np.arange(n) % 13 == 0, 0.1, 50.0).astype(np.float32)
    trg, env = _pairs((1, 2, 3))
    hist = (0.0, 0.01, 1.0)
    cid = ctx.upload(xyz, labels)
    ctx.surfdist(cid, d2)
    ctx.tasks(trg, env)
    ctx.hist(*hist)
    ctx.set_option("symmetric", symmetric)
    ctx.set_option("knn_walks", walks)
    try:
        if flags == N.PP_RDF | N.PP_MKNN:  # a place so full keeps an untuned pass of both on the per-centre scan
            ctx.run(cid, flags, ks)
            assert ctx.last_kernel() == "k_scan"
            ctx.tuning(cid, 4.0, ((2 | 2 << 8 | 2 << 12) << 16) | N.PP_TILE_LANES)
        launches, got = {}, {}
        without = 1 if symmetric and flags == N.PP_RDF else 2  # the buffers asked for before the list
        for limit in (without, -1):
            ctx.set_option("scratch", limit)
            ctx.run(cid, flags, ks)
            before = N.kernel_launches()
            ctx.run(cid, flags, ks)
            got[limit], launches[limit] = (ctx.fetch(), ctx.stats(), ctx.run_tests()), N.kernel_launches() - before
            assert ctx.last_kernel() != "k_scan"
    finally:
        for name, value in (("symmetric", 1), ("knn_walks", 0), ("scratch", -1)):
            ctx.set_option(name, value)
        ctx.free(cid)
    if flags == N.PP_RDF and sigma < 0.1:
        assert launches[-1] == launches[without] + 1
        assert got[without][2] == got[-1][2]  # the same tests
    ref = oracle.spatstat(xyz, labels, d2, *hist, flags, trg, env, ks)
    for bins, st, _ in got.values():
        assert np.array_equal(bins, ref["bins"]) and st["pairs"] == ref["pairs"] and st["centres"] == ref["centres"]


@pytest.mark.parametrize("targets", [[[1], [2], [1, 3]], [[2], [3], [2, 3]], [[3]]])
@pytest.mark.parametrize("env", [[[1], [2, 3], [1]], [[1, 2, 3], [1, 2], [3]]])
def test_scan_of_dense_and_sparse_centres(ctx, oracle, targets, env):
    """The per-centre scan with counts, RDF and kNN at once, one list or several,
    for centres in most cells and in few."""
    env = env[: len(targets)]
    spec = synth.cylinder_specimen(n=16000, radius=3.0, height=12.0, fractions=(0.9, 0.07, 0.03), seed=23, nseg=48,
                                   stack=4.0)
    d2 = np.where(np.arange(len(spec.xyz)) % 7 == 0, 0.5, 10.0).astype(np.float32)
    hist, ks, flags = (0.0, 0.02, 1.0), [31, 4, 1], N.PP_RDF | N.PP_MKNN | N.PP_CNTNB
    cid = ctx.upload(spec.xyz, spec.labels)
    ctx.surfdist(cid, d2)
    ctx.tasks(targets, env)
    ctx.hist(*hist)
    try:
        ctx.run(cid, flags, ks)
        bins, counts, st = ctx.fetch(), ctx.fetch_cntnb(), ctx.stats()
        assert ctx.last_kernel() == "k_scan"
    finally:
        ctx.free(cid)
    ref = oracle.spatstat(spec.xyz, spec.labels, d2, *hist, flags, targets, env, ks)
    assert np.array_equal(bins, ref["bins"]) and st["pairs"] == ref["pairs"] and st["centres"] == ref["centres"]
    assert np.array_equal(counts, ref["cntnb"][:, : counts.shape[1]]) and ref["cntnb"][:, counts.shape[1]:].sum() == 0


@pytest.mark.parametrize("nbins", [2500, 6000, 16380])
@pytest.mark.parametrize("symmetric", [1, 0])
@pytest.mark.parametrize("tasks", ["pairs", "matrix only around others", "matrix in no environment"])
def test_rdf_rows_in_shared_memory(ctx, oracle, nbins, symmetric, tasks):
    """Bins of which some rows fit in shared memory, one row or none: those of
    the commonest types there, the others in global memory; more than half of
    the ions are centres, some are not."""
    spec = synth.cone_specimen(n=14000, r_apex=4.0, half_angle_deg=10.0, length=14.0, n_clusters=20, members=40,
                               nspecies=6, seed=31, nseg=48, stack=4.0)
    trg, env = {"pairs": _pairs(range(1, 7)),
                "matrix only around others": ([[2], [3], [4, 5, 6]], [[1], [1, 2], [1]]),
                "matrix in no environment": ([[t] for t in range(1, 7)], [[2, 3], [4], [5], [6], [2], [3]])}[tasks]
    d2 = np.where(np.arange(len(spec.xyz)) % 5 == 0, 0.1, 10.0).astype(np.float32)
    hist = (0.0, 0.9 / nbins, 0.9)
    cid = ctx.upload(spec.xyz, spec.labels)
    ctx.surfdist(cid, d2)
    ctx.tasks(trg, env)
    ctx.hist(*hist)
    ctx.tuning(cid, 4.0, ((3 | 2 << 8 | 2 << 12) << 16) | N.PP_TILE_LANES)
    ctx.set_option("symmetric", symmetric)
    try:
        got = []
        for limit in (-1, 1 if symmetric else 2):  # with the map of the rows, and without it
            ctx.set_option("scratch", limit)
            ctx.run(cid, N.PP_RDF)
            got.append((ctx.fetch(), ctx.stats()))
            assert ctx.last_kernel() == "k_lanes"
    finally:
        ctx.set_option("scratch", -1)
        ctx.set_option("symmetric", 1)
        ctx.free(cid)
    ref = oracle.spatstat(spec.xyz, spec.labels, d2, *hist, N.PP_RDF, trg, env, [])
    for bins, st in got:
        assert st["pairs"] == ref["pairs"] and st["centres"] == ref["centres"]
        assert np.array_equal(bins, ref["bins"])
