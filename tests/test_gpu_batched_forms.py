"""Which kernels a batched run takes: told by the nodes of its captured graph,
with counts equal whichever they are."""
import numpy as np
import pytest

from paraprobe_gb300 import native as N
from paraprobe_gb300 import synth

pytestmark = pytest.mark.gpu


def _pairs(types):
    return [[a] for a in types for b in types], [[b] for a in types for b in types]


def _setup(ctx, fractions, hist, n=6000):
    spec = synth.cylinder_specimen(n=n, radius=2.5, height=9.0, fractions=fractions, seed=19, nseg=32, stack=4.0)
    types = tuple(range(1, len(fractions) + 1))
    trg, env = _pairs(types)
    d2 = np.where(np.arange(len(spec.xyz)) % 9 == 0, 0.1, 10.0).astype(np.float32)
    cid = ctx.upload(spec.xyz, spec.labels)
    ctx.surfdist(cid, d2)
    ctx.tasks(trg, env)
    ctx.hist(*hist)
    return spec, d2, trg, env, cid


def _reset(ctx):
    for name, value in (("batched_minor", 1), ("scratch", -1)):
        ctx.set_option(name, value)


@pytest.mark.parametrize("flags,ks", [(N.PP_RDF, []), (N.PP_MKNN, [5, 1]), (N.PP_RDF | N.PP_1NN | N.PP_MKNN, [5, 1])])
def test_by_common_type_without_its_buffers(ctx, oracle, flags, ks):
    """Where a buffer of the form by the common type is missing, whichever it is,
    the other kernels take the run."""
    hist = (0.0, 0.02, 0.9)
    spec, d2, trg, env, cid = _setup(ctx, (0.9, 0.06, 0.04), hist)
    rng = np.random.default_rng(1)
    sets = np.stack([rng.permutation(spec.labels) for _ in range(33)])

    def run(minor, scratch):
        ctx.set_option("batched_minor", minor)
        ctx.set_option("scratch", scratch)
        ctx.run_batched(cid, flags, ks, include_original=True, label_sets=sets)
        return ctx.batched_graph()["nodes"], [ctx.fetch_batched(r) for r in range(ctx.batched_count())]

    try:
        other, base = run(0, -1)
        form, got = run(2, -1)
        assert form != other
        nodes = []
        for limit in range(5):
            k, bins = run(2, limit)
            nodes.append(k)
            assert np.array_equal(bins, base)
        assert np.array_equal(got, base)
        assert nodes[0] == nodes[1] == other and nodes[-1] == form
    finally:
        _reset(ctx)
        ctx.free(cid)
    for r in (0, 1, 33):
        lab = spec.labels if r == 0 else sets[r - 1]
        ref = oracle.spatstat(spec.xyz, lab, d2, *hist, flags, trg, env, ks)
        assert np.array_equal(base[r], ref["bins"])


def test_knn_by_common_type_holds_no_rdf_sums(native_lib):
    """A run that only counts neighbours by the common type takes no memory for
    the sums of pairs: 288 realisations of 1,500 bins would need 60 MB."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    c = N.Context(0)
    try:
        hist = (0.0, 0.9 / 1500, 0.9)
        spec, d2, trg, env, cid = _setup(c, (0.9,) + (0.0125,) * 8, hist, n=3000)
        rng = np.random.default_rng(2)
        sets = np.stack([rng.permutation(spec.labels) for _ in range(287)])
        used, nodes = [], []
        for minor in (0, 2):
            c.set_option("batched_minor", minor)
            c.run_batched(cid, N.PP_1NN, [], include_original=True, label_sets=sets)
            c.fetch_batched(0)
            used.append(torch.cuda.mem_get_info()[0])
            nodes.append(c.batched_graph()["nodes"])
        assert nodes[0] != nodes[1]
        assert used[0] - used[1] < 24 << 20
    finally:
        c.close()


@pytest.mark.parametrize("flags,ks", [(N.PP_RDF, []), (N.PP_MKNN, [5, 1]), (N.PP_RDF | N.PP_MKNN, [5, 1])])
@pytest.mark.parametrize("share", [0.97, 0.85, 0.77])
def test_groups_by_number_of_realisations(ctx, flags, ks, share):
    """The last, partial group of 32 realisations is counted by the common type
    only where enough of its lanes work, a share of it on either side of the
    line; regions of interest share its groups.  Counts are those of the other
    kernels, one realisation never pays, and a full group always does."""
    hist = (0.0, 0.02, 0.9)
    spec, d2, trg, env, cid = _setup(ctx, (share, 0.6 * (1 - share), 0.4 * (1 - share)), hist, n=3000)
    rng = np.random.default_rng(3)
    sets = np.stack([rng.permutation(spec.labels) for _ in range(65)])
    roi = np.array([[0.1 * q, 0.0, 4.5, 2.3] for q in range(5)], dtype=np.float32)

    def run(minor, nsets, rois):
        ctx.set_option("batched_minor", minor)
        ctx.run_batched(cid, flags, ks, include_original=False, label_sets=sets[:nsets] if nsets else None,
                        rois=roi[:rois] if rois else None)
        count = ctx.batched_count()
        return (ctx.batched_graph()["nodes"], [ctx.fetch_batched(r) for r in range(count)],
                [ctx.batched_stats(r) for r in range(count)])

    try:
        for nsets, rois in [(1, 0), (2, 0), (3, 0), (5, 0), (8, 0), (9, 2), (20, 0), (29, 5), (31, 1), (32, 0), (33, 0),
                            (37, 0), (40, 3), (64, 0), (65, 2), (0, 5)]:
            nodes = {}
            nodes[0], base, stats = run(0, nsets, rois)
            for minor in (1, 2):
                nodes[minor], got, st = run(minor, nsets, rois)
                assert st == stats and np.array_equal(got, base), (nsets, rois, minor)
            if (nsets, rois) == (1, 0) or (nsets == 0 and flags == N.PP_RDF):
                assert nodes[1] == nodes[0]
            if nsets >= 32:
                assert nodes[1] != nodes[0] and nodes[2] != nodes[0]
    finally:
        _reset(ctx)
        ctx.free(cid)
