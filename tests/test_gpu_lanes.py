"""Forms of the centre-per-lane RDF pass against the oracle: where its bins live
(by kind of pair or in the cores' layout in shared memory, or in global memory,
by their number), how categories are found (approximate root or table), which
ions are centres, and blocks cut by the grid's edges.  Counts are whole numbers
and must be equal."""
import numpy as np
import pytest

from paraprobe_gb300 import native as N
from paraprobe_gb300 import synth

pytestmark = pytest.mark.gpu

# 4 centre and 5 environment slots: 4 * (4 + 5 + 1) rows of bins by kind fit
# 224 KB up to about 1,100 bins, the cores' 20 rows up to about 2,200
HISTS = [(0.0, 0.01, 1.2), (0.0, 0.0011, 1.2), (0.0, 0.0008, 1.2), (0.0, 0.0003, 1.2),
         (0.3, 0.01, 1.2), (0.3, 0.0008, 1.2), (0.0, 0.4, 1.2), (0.0, 0.037, 1.25)]


@pytest.mark.parametrize("hist", HISTS)
@pytest.mark.parametrize("symmetric", [1, 0])
def test_lanes_rdf_bin_forms(ctx, oracle, hist, symmetric):
    spec = synth.cone_specimen(n=20000, r_apex=5.0, half_angle_deg=10.0, length=14.0, n_clusters=20, members=40,
                               nspecies=6, seed=97, nseg=48, stack=4.0)
    trg = [[1], [2, 3], [3], [1, 4]]
    env = [[1, 2], [3, 6], [1, 2, 3, 5], [5]]  # type 4: a centre in no environment; 5, 6: never centres
    cid = ctx.upload(spec.xyz, spec.labels)
    ctx.hull(cid, spec.hull, 0.5)
    ctx.tuning(cid, 4.0, ((3 | 2 << 8 | 2 << 12) << 16) | N.PP_TILE_LANES)
    ctx.tasks(trg, env)
    ctx.hist(*hist)
    ctx.set_option("symmetric", symmetric)
    try:
        ctx.run(cid, N.PP_RDF | N.PP_RIPK)
        bins, st = ctx.fetch(), ctx.stats()
        assert ctx.last_kernel() == "k_lanes"
    finally:
        ctx.set_option("symmetric", 1)
        ctx.free(cid)
    surf = oracle.surface_distance(spec.xyz, spec.hull, np.float32(hist[2]))
    ref = oracle.spatstat(spec.xyz, spec.labels, surf, *hist, N.PP_RDF | N.PP_RIPK, trg, env, [])
    assert st["pairs"] == ref["pairs"] and st["centres"] == ref["centres"]
    assert np.array_equal(bins, ref["bins"])


def test_lanes_pairs_on_bin_edges(ctx, oracle):
    """Ions on a lattice of 2^-4 nm: most distances lie exactly on bin edges or
    on R, and coincident ions give d = 0."""
    g = np.arange(24, dtype=np.float32) / 16
    xyz = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    xyz = np.concatenate([xyz, xyz[:500]]).astype(np.float32)
    labels = (1 + np.arange(len(xyz)) % 3).astype(np.uint8)
    types = [1, 2, 3]
    trg, env = [[a] for a in types for b in types], [[b] for a in types for b in types]
    hist = (0.0, 0.0625, 0.5)
    cid = ctx.upload(xyz, labels)
    ctx.surfdist(cid, np.full(len(xyz), 10.0, dtype=np.float32))
    ctx.tuning(cid, 4.0, ((4 | 2 << 8 | 2 << 12) << 16) | N.PP_TILE_LANES)
    ctx.tasks(trg, env)
    ctx.hist(*hist)
    ctx.run(cid, N.PP_RDF)
    rdf, st = ctx.fetch(), ctx.stats()
    assert ctx.last_kernel() == "k_lanes"
    ctx.run(cid, N.PP_MKNN, [7, 3, 1])
    knn, st2 = ctx.fetch(), ctx.stats()
    assert ctx.last_kernel() == "k_lanes_knn"
    ctx.free(cid)
    surf = np.full(len(xyz), 10.0, dtype=np.float32)
    for got, s, flags, ks in ((rdf, st, N.PP_RDF, []), (knn, st2, N.PP_MKNN, [7, 3, 1])):
        ref = oracle.spatstat(xyz, labels, surf, *hist, flags, trg, env, ks)
        assert s["pairs"] == ref["pairs"] and np.array_equal(got, ref["bins"])


@pytest.mark.parametrize("ks", [[1], [8, 3], [9, 1], [10, 5, 1], [16, 2], [20, 19, 1]])
@pytest.mark.parametrize("fractions", [(0.97, 0.02, 0.01), (0.5, 0.45, 0.05), (0.999, 0.001, 0.0)])
@pytest.mark.parametrize("lists,rmin", [(0, 0.0), (2, 0.0), (0, 0.05)])
def test_knn_in_two_walks(ctx, oracle, ks, fractions, lists, rmin):
    """Dense sets within a first radius, sparse sets from their own list: every
    list size class, one or two dense sets, sets without ions, both list forms,
    table categories; clusters and a hole make centres that need more than the
    first radius; coincident ions and masked centres."""
    spec = synth.cylinder_specimen(n=24000, radius=3.0, height=18.0, fractions=fractions, seed=7 + len(ks), nseg=48,
                                   stack=4.0)
    xyz = spec.xyz.copy()
    inside = np.linalg.norm(xyz - np.array([0, 0, 9.0], dtype=np.float32), axis=1) < 1.1
    keep = ~inside | (np.arange(len(xyz)) % 40 == 0)  # a nearly empty ball: few neighbours within the first radius
    xyz, labels = xyz[keep], spec.labels[keep]
    xyz[:200] = xyz[200:400]
    types = [1, 2, 3]
    trg, env = [[a] for a in types for b in types], [[b] for a in types for b in types]
    hist = (rmin, 0.01, 1.5)
    n = len(xyz)
    mask = (np.arange(n) % 7 != 0).astype(np.uint8)
    cid = ctx.upload(xyz, labels)
    ctx.surfdist(cid, np.where(np.arange(n) % 11 == 0, 1.0, 10.0).astype(np.float32))
    ctx.tasks(trg, env)
    ctx.hist(*hist)
    ctx.set_option("knn_lists", lists)
    ctx.set_option("knn_walks", 2)
    try:
        ctx.run(cid, N.PP_MKNN, ks)
        got, st, kernel = ctx.fetch(), ctx.stats(), ctx.last_kernel()
        ctx.run(cid, N.PP_MKNN, ks, centre_mask=mask)
        part, stp = ctx.fetch(), ctx.stats()
        ctx.run(cid, N.PP_MKNN, ks, centre_mask=1 - mask)
        rest, str_ = ctx.fetch(), ctx.stats()
    finally:
        ctx.set_option("knn_lists", 0)
        ctx.set_option("knn_walks", 0)
        ctx.free(cid)
    assert kernel == "k_lanes_knn"
    surf = np.where(np.arange(n) % 11 == 0, 1.0, 10.0).astype(np.float32)
    ref = oracle.spatstat(xyz, labels, surf, *hist, N.PP_MKNN, trg, env, ks)
    assert st["pairs"] == ref["pairs"] and st["centres"] == ref["centres"]
    assert np.array_equal(got, ref["bins"])
    assert np.array_equal(part + rest, got) and stp["pairs"] + str_["pairs"] == st["pairs"]


TASKS = {
    "pairs": ([[a] for a in (1, 2, 3) for b in (1, 2, 3)], [[b] for a in (1, 2, 3) for b in (1, 2, 3)]),
    "common type in a wider set": ([[2], [1]], [[1, 2, 3], [1, 4]]),
    "common type never a centre": ([[2], [3]], [[1], [1, 2]]),
    "common type in no set": ([[1], [2, 3]], [[2], [2, 3, 4]]),
    "overlapping sets": ([[1], [1]], [[1, 2], [2, 3]]),
}


@pytest.mark.parametrize("form", [0, 1, 2])
@pytest.mark.parametrize("tasks", sorted(TASKS))
@pytest.mark.parametrize("nsets,rois,cap", [(3, 2, 0), (34, 0, 0), (40, 3, 60000)])
def test_batched_by_common_type(ctx, oracle, form, tasks, nsets, rois, cap):
    """Batched realisations counted by what is not of the common type, for sets
    that hold it, hold it with others or leave it out, types without a slot,
    label sets that are no shuffles, groups of 32 and their remainders, regions
    of interest and pair lists in chunks."""
    spec = synth.cylinder_specimen(n=9000, radius=2.5, height=11.0, fractions=(0.9, 0.05, 0.04, 0.01), seed=17, nseg=32,
                                   stack=4.0)
    n = len(spec.xyz)
    rng = np.random.default_rng(nsets)
    sets = np.stack([rng.permutation(spec.labels) for _ in range(nsets)])
    sets[1] = rng.integers(0, 5, n)                 # no common type, and type 0
    sets[2] = 2                                     # one type only
    roi = np.stack([[0.3, -0.2, 5.5, 2.2 + 0.4 * q] for q in range(rois)]).astype(np.float32) if rois else None
    trg, env = TASKS[tasks]
    hist, ks, flags = (0.0, 0.02, 0.9), [12, 5, 1], N.PP_RDF | N.PP_1NN | N.PP_MKNN
    d2 = np.where(np.arange(n) % 9 == 0, 0.1, 10.0).astype(np.float32)
    cid = ctx.upload(spec.xyz, spec.labels)
    ctx.surfdist(cid, d2)
    ctx.tasks(trg, env)
    ctx.hist(*hist)
    ctx.set_option("batched_minor", form)
    ctx.set_option("batched_pair_cap", cap)
    try:
        ctx.run_batched(cid, flags, ks, include_original=True, label_sets=sets, rois=roi)
        got = [ctx.fetch_batched(r) for r in range(ctx.batched_count())]
        stats = [ctx.batched_stats(r) for r in range(ctx.batched_count())]
    finally:
        ctx.set_option("batched_minor", 1)
        ctx.set_option("batched_pair_cap", 0)
        ctx.free(cid)
    assert len(got) == 1 + nsets + rois
    for r in [0, 1, 2, 3, nsets] + list(range(1 + nsets, 1 + nsets + rois)):
        lab = spec.labels if r == 0 or r > nsets else sets[r - 1]
        surf = d2
        if r > nsets:
            c = roi[r - 1 - nsets]
            far = c[3] - np.sqrt(((spec.xyz - c[:3]) ** 2).sum(1, dtype=np.float64)) < hist[2]
            surf = np.where(far, 0.0, d2).astype(np.float32)
        ref = oracle.spatstat(spec.xyz, lab.astype(np.uint8), surf, *hist, flags, trg, env, ks)
        assert stats[r]["centres"] == ref["centres"] and stats[r]["pairs"] == ref["pairs"], r
        assert np.array_equal(got[r], ref["bins"]), r


def test_inside_repeats(ctx):
    """The occupancy grid's clusters are joined concurrently: the counts of a
    porous cloud are the same every time."""
    rng = np.random.default_rng(5)
    xyz = rng.uniform(0, 30, (9000, 3)).astype(np.float32)
    cid = ctx.upload(xyz, np.ones(len(xyz), dtype=np.uint8))
    got = {tuple(sorted(ctx.inside(cid, 1.0, 1.0).items())) for _ in range(40)}
    ctx.free(cid)
    assert len(got) == 1


@pytest.mark.parametrize("dense", [0, 500, 1500])
def test_batched_lists_of_uneven_length(ctx, oracle, dense):
    """Pair lists some of which are far longer than the mean: balls that the
    first walk keeps and balls that are walked again, more than 1024 ions too."""
    rng = np.random.default_rng(dense)
    xyz = np.concatenate([rng.uniform(0, 11, (3000, 3)), rng.uniform(5, 5.4, (dense, 3))]).astype(np.float32)
    n = len(xyz)
    labels = rng.choice(np.array([1, 2], dtype=np.uint8), n, p=[0.9, 0.1])
    sets = np.stack([rng.permutation(labels) for _ in range(2)])
    d2, hist, ks, flags = np.full(n, 10.0, dtype=np.float32), (0.0, 0.02, 1.0), [6, 1], N.PP_RDF | N.PP_MKNN
    trg, env = [[1], [2]], [[2], [1]]
    cid = ctx.upload(xyz, labels)
    ctx.surfdist(cid, d2)
    ctx.tasks(trg, env)
    ctx.hist(*hist)
    ctx.run_batched(cid, flags, ks, include_original=True, label_sets=sets)
    got = [ctx.fetch_batched(r) for r in range(ctx.batched_count())]
    ctx.free(cid)
    for r, lab in enumerate([labels, sets[0], sets[1]]):
        ref = oracle.spatstat(xyz, lab, d2, *hist, flags, trg, env, ks)
        assert np.array_equal(got[r], ref["bins"]), r


@pytest.mark.parametrize("nbins", [8000, 16380])
def test_knn_of_many_bins(ctx, oracle, nbins):
    """Bins whose tables leave the kNN walks little shared memory, up to the most
    that are taken."""
    spec = synth.cylinder_specimen(n=12000, radius=2.5, height=14.0, fractions=(0.95, 0.04, 0.01), seed=3, nseg=32,
                                   stack=4.0)
    types = [1, 2, 3]
    trg, env = [[a] for a in types for b in types], [[b] for a in types for b in types]
    d2, hist, ks = np.full(len(spec.xyz), 10.0, dtype=np.float32), (0.0, 1.0 / nbins, 1.0), [20, 1]
    cid = ctx.upload(spec.xyz, spec.labels)
    ctx.surfdist(cid, d2)
    ctx.tasks(trg, env)
    ctx.hist(*hist)
    ctx.set_option("knn_walks", 2)
    try:
        ctx.run(cid, N.PP_MKNN, ks)
        got, st = ctx.fetch(), ctx.stats()
    finally:
        ctx.set_option("knn_walks", 0)
        ctx.free(cid)
    ref = oracle.spatstat(spec.xyz, spec.labels, d2, *hist, N.PP_MKNN, trg, env, ks)
    assert st["pairs"] == ref["pairs"] and np.array_equal(got, ref["bins"])
