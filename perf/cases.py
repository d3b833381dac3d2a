"""What is measured when this framework is made faster: the calls a user of the spatial statistics makes.

Every case is a dict of plain values.  listed() gives the fixed ones, draw() more of the same ranges; prepare()
makes a seeded specimen on the GPU and holds what a program has in hand before the call (a resident cloud with its
hull, label sets, host buffers), run() is one call through paraprobe_gb300.native and returns all it computes,
work() what the call cannot do without, and exact() the distances in 64 bits where a call returns distances.

Specimens are the two geometries of paraprobe_gb300.synth (cylinder, truncated cone with solute clusters), with the
densities and species fractions bench.py uses, drawn with torch so that a 20M-ion cloud takes milliseconds.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from paraprobe_gb300 import native as N
from paraprobe_gb300 import synth

TIP_RHO = 13.42      # ions per nm^3 of the 20M-ion tip (apex radius 30 nm, 10 degrees, 200 nm long)
CYL_RHO = 50.0       # ions per nm^3 of the 1M-ion cylinder (radius 10 nm, 63.66 nm high)
CARVE = 2.0          # SurfaceCellsCarvingRadius
TIP_IID = (0.02, 0.01, 0.005, 0.005, 0.002)   # iid minority species of the tips
CYL_FRACTIONS = (0.90, 0.08, 0.02)

_context = None


def context():
    """One context per program, as the interface asks for."""
    global _context
    if _context is None:
        _context = N.Context(0)
    return _context


# ------------------------------------------------------------------ cases
def _pass(name, **kw):
    c = dict(kind="pass", name=name, n=1_000_000, shape="tip", species=6, tasks="pairs", R=2.0, incr=0.01, rdf=True,
             nn1=False, ripk=False, k=0, orders="all", hull=True, shuffled=False)
    c.update(kw)
    return c


def listed():
    return [
        # the neighbours of one ion of a resident cloud: an interactive look-up, the smallest call there is
        dict(kind="neighbours", name="neighbours_1m", n=1_000_000, R=2.0),
        # a small specimen, minority centres against everything, all analyses in one pass: launches and latency
        _pass("cyl50k_all", n=50_000, shape="cylinder", species=3, tasks="solute", R=1.0, nn1=True, k=10, orders="few"),
        # the 1M-ion cylinder of the benchmark's first configuration: sparse centres, RDF and kNN in one pass
        _pass("cyl1m_solute", n=1_000_000, shape="cylinder", species=3, tasks="solute", R=1.0, k=10, orders="few"),
        # the benchmark's 20M-ion tip: all 36 pair RDFs ...
        _pass("tip20m_rdf", n=20_000_000),
        # ... and all 36 kNN distributions, k = 1..10, in finer bins
        _pass("tip20m_knn", n=20_000_000, incr=0.005, rdf=False, k=10),
        # RDF, first neighbour and kNN of an ordinary tip asked for together, as one settings file does
        _pass("tip5m_all", n=5_000_000, R=1.5, nn1=True, k=8),
        # the largest kind of workload (8 species, 64 pairs, k = 1..20 within 2.5 nm), at a size one pass can repeat
        _pass("tip8sp_both", n=12_000_000, species=8, R=2.5, k=20),
        # a whole job from a POS image on the host: ranging, header values, hull, an RDF and a kNN pass, results back
        dict(kind="job", name="job_tip4m", n=4_000_000, species=6, R=2.0, incr=0.01, k=10),
        # null model and regions of interest: many label shuffles and spheres over one geometry
        dict(kind="batched", name="batched_tip2m", n=2_000_000, species=6, R=1.5, incr=0.01, k=8, shuffles=64, rois=16),
        # many small queries on resident clouds at once (radii 0.5 .. 3 nm, one species pair each)
        dict(kind="served", name="served_tip1m", n=1_000_000, species=6, queries=24, slots=4),
        # distances to the hull alone, on the caller's own device buffers
        dict(kind="surface", name="surface_1m", n=1_000_000, R=2.0, stack=4.0, nseg=128),
        # neighbour counts and n-point correlations of the solutes
        dict(kind="counts", name="counts_tip1m", n=1_000_000, species=6, R=2.0, incr=0.1, order=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("pass",) * 8 + ("job", "batched", "served", "surface", "neighbours", "counts"))
    R = round(rng.uniform(0.7, 2.5), 3)
    if kind == "pass":
        shape = rng.choice(("tip", "tip", "tip", "cylinder"))
        rho = TIP_RHO if shape == "tip" else CYL_RHO
        what = rng.choice(("rdf", "knn", "both", "both"))
        tasks = rng.choice(("pairs", "pairs", "solute", "overlapping"))
        if shape == "cylinder":
            R = round(rng.uniform(0.5, 1.5), 3)
        # no more neighbour pairs than a quarter of the largest listed pass: overlapping sets and shuffles cost more a pair
        most = 2.4e9 / (rho * 4.19 * R ** 3)
        n = _log(rng, 20_000, min(20_000_000, max(40_000, int(most))))
        return dict(kind="pass", n=n, shape=shape, species=3 if shape == "cylinder" else rng.randint(4, 8), tasks=tasks,
                    R=R, incr=rng.choice((0.005, 0.01, 0.02, 0.037)), rdf=what != "knn", nn1=rng.random() < 0.4,
                    ripk=what != "knn" and rng.random() < 0.3, k=0 if what == "rdf" else rng.randint(1, 20),
                    orders=rng.choice(("all", "few")), hull=rng.random() < 0.8, shuffled=rng.random() < 0.2)
    if kind == "job":
        return dict(kind=kind, n=_log(rng, 100_000, 4_000_000), species=rng.randint(4, 8), R=R, incr=rng.choice((0.005, 0.01, 0.02)),
                    k=rng.randint(1, 16))
    if kind == "batched":
        return dict(kind=kind, n=_log(rng, 50_000, 1_500_000), species=rng.randint(4, 8), R=round(rng.uniform(0.7, 1.6), 3), incr=0.01,
                    k=rng.randint(1, 10), shuffles=rng.randint(3, 70), rois=rng.randint(0, 20))
    if kind == "served":
        return dict(kind=kind, n=_log(rng, 100_000, 1_500_000), species=rng.randint(4, 8), queries=rng.randint(8, 32), slots=rng.randint(1, 4))
    if kind == "surface":
        return dict(kind=kind, n=_log(rng, 20_000, 2_000_000), R=R, stack=round(rng.uniform(2.0, 6.0), 2), nseg=rng.randint(48, 200))
    if kind == "neighbours":
        return dict(kind=kind, n=_log(rng, 20_000, 4_000_000), R=round(rng.uniform(0.3, 3.0), 3))
    return dict(kind=kind, n=_log(rng, 50_000, 1_500_000), species=rng.randint(4, 8), R=R, incr=rng.choice((0.05, 0.1, 0.2)),
                order=rng.randint(0, 9))


# -------------------------------------------------------------- specimens
def _tip_length(n):
    return synth.cone_length_for(n, TIP_RHO, 30.0, 10.0) if n > 200_000 else synth.cone_length_for(n, TIP_RHO, 8.0, 10.0)


def _tip_apex(n):
    return 30.0 if n > 200_000 else 8.0


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(n, g):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _tip(n, species, seed):
    """Truncated cone: uniform matrix (type 1), Gaussian solute clusters (types 2 and 3) and iid minority species."""
    g = _generator(seed)
    r0, tan, length = _tip_apex(n), math.tan(math.radians(10.0)), _tip_length(n)
    r1 = r0 + length * tan

    def inside(m):
        z = ((r0 ** 3 + _uniform(m, g) * (r1 ** 3 - r0 ** 3)) ** (1.0 / 3.0) - r0) / tan
        r = (r0 + z * tan) * _uniform(m, g).sqrt()
        phi = 2.0 * math.pi * _uniform(m, g)
        return torch.stack((r * phi.cos(), r * phi.sin(), z), 1)

    p = inside(n)
    m = max(1, n // 200)                                       # 0.5 % of the ions, 50 to a cluster
    centres = inside(max(1, m // 50))
    at = torch.randint(n, (m,), generator=g, device="cuda")
    q = centres[torch.randint(centres.shape[0], (m,), generator=g, device="cuda")]
    q = q + 1.5 * torch.randn((m, 3), generator=g, device="cuda", dtype=torch.float64)
    ok = (q[:, 2] >= 0) & (q[:, 2] <= length) & (q[:, 0] ** 2 + q[:, 1] ** 2 <= (r0 + q[:, 2] * tan) ** 2)
    u = _uniform(n, g)
    lab = torch.ones(n, dtype=torch.uint8, device="cuda")
    edge = 0.0
    for s, f in enumerate(TIP_IID[: max(0, species - 3)]):
        lab[(u >= edge) & (u < edge + f)] = 4 + s
        edge += f
    sol = torch.where(_uniform(m, g) < 0.7, 2, 3).to(torch.uint8)
    keep, inv = torch.unique(at[ok], return_inverse=True)      # an ion named twice takes one place, the same every time
    first = torch.full((keep.numel(),), m, dtype=torch.int64, device="cuda")
    first.scatter_reduce_(0, inv, torch.arange(m, device="cuda")[ok], "amin")
    p[keep], lab[keep] = q[first], sol[first]
    return p.float().contiguous(), lab


def _cylinder(n, seed):
    """Uniform ions, iid species, radius 10 nm (4 nm below 200,000 ions)."""
    g = _generator(seed)
    radius = 10.0 if n > 200_000 else 4.0
    r, phi, z = radius * _uniform(n, g).sqrt(), 2.0 * math.pi * _uniform(n, g), _cyl_height(n) * _uniform(n, g)
    u = _uniform(n, g)
    lab = 1 + (u >= CYL_FRACTIONS[0]).to(torch.uint8) + (u >= CYL_FRACTIONS[0] + CYL_FRACTIONS[1]).to(torch.uint8)
    return torch.stack((r * phi.cos(), r * phi.sin(), z), 1).float().contiguous(), lab.to(torch.uint8)


def _cyl_height(n):
    radius = 10.0 if n > 200_000 else 4.0
    return n / (CYL_RHO * math.pi * radius * radius)


def _specimen(shape, n, species, seed):
    return _tip(n, species, seed) if shape == "tip" else _cylinder(n, seed)


def _hull(shape, n, nseg=512, stack=2.0):
    if n <= 200_000:
        nseg = min(nseg, 96)
    if shape == "tip":
        return synth.cone_hull(_tip_apex(n), 10.0, _tip_length(n), nseg=nseg, stack=stack)
    return synth.cylinder_hull(10.0 if n > 200_000 else 4.0, _cyl_height(n), nseg=nseg, stack=stack)


def _tasks(tasks, species):
    types = list(range(1, species + 1))
    if tasks == "pairs":
        return [[a] for a in types for b in types], [[b] for a in types for b in types]
    if tasks == "solute":                                       # one minority species against every ion
        return [[2]], [types]
    return [[2], [2, 3], types], [types, [1, 2], [3]]           # environments that share types


class _Cloud:
    """A resident cloud of the program's context."""

    def __init__(self, ctx, xyz, lab, hull):
        self.ctx = ctx
        self.id = ctx.upload_device(xyz.data_ptr(), lab.data_ptr(), lab.numel())
        torch.cuda.synchronize()
        if hull is not None:
            ctx.hull(self.id, hull, CARVE)

    def __del__(self):
        try:
            if self.ctx.h:
                self.ctx.free(self.id)
        except Exception:
            pass


def _orders(case):
    k = case["k"]
    return list(range(k, 0, -1)) if case.get("orders", "all") == "all" else sorted({1, (k + 1) // 2, k} if k else (), reverse=True)


def _room(case):
    """Places for one ion's neighbours: three times the mean, and more for small balls (clusters are denser)."""
    return int(3.0 * TIP_RHO * 4.19 * case["R"] ** 3) + 256


# ---------------------------------------------------------------- prepare
def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    shape, species = case.get("shape", "tip"), case.get("species", 6)
    s = {"case": case, "kind": kind, "n": n}
    if kind == "surface":
        xyz, _ = _tip(n, 4, seed)
        s["xyz"], s["tri"] = xyz, torch.from_numpy(_hull("tip", n, case["nseg"], case["stack"])).cuda()
        s["out"] = torch.empty(n, dtype=torch.float32, device="cuda")
        return s
    ctx = s["ctx"] = context()
    if kind == "job":
        xyz, lab = _tip(n, species, seed)
        g = _generator(seed + 1)
        u = _uniform(n, g)
        mq = 10.0 + 5.0 * (lab.double() - 1.0) + 0.1 + 0.8 * u
        mq = torch.where(_uniform(n, g) < 0.02, torch.full_like(mq, 3.0), mq)    # 2 % of the ions are in no range
        rec = torch.cat((xyz, mq.float()[:, None]), 1).contiguous().view(torch.uint8).reshape(-1, 4).flip(1).contiguous()
        host = torch.empty(rec.shape, dtype=torch.uint8, pin_memory=True)
        host.copy_(rec)
        s["pos"], s["ranges"] = host.numpy().reshape(-1), [(lo, hi, t + 1) for t, (lo, hi) in enumerate(synth.species_windows(species))]
        s["hull"] = _hull("tip", n)
        s["trg"], s["env"] = _tasks("pairs", species)
        return s
    xyz, lab = _specimen(shape, n, species, seed)
    if kind == "neighbours":
        s["cloud"] = _Cloud(ctx, xyz, lab, None)
        s["ion"] = int(torch.randint(n, (1,), generator=_generator(seed + 1), device="cuda").item())
        s["xyz"], s["room"] = xyz, _room(case)
        return s
    if kind == "served":
        # three resident clouds and a server over them; radii cover 0.5 .. 3 nm evenly in a seeded order
        s["own"] = own = N.Context(0)
        s["clouds"] = []
        for i, m in enumerate((n, max(1000, n // 4), max(1000, n // 10))):
            x, l = (xyz, lab) if i == 0 else _tip(m, species, seed + 17 * i)
            c = own.upload_device(x.data_ptr(), l.data_ptr(), m)
            torch.cuda.synchronize()
            own.hull(c, _hull("tip", m, 128, 4.0), CARVE)
            own.prepare(c, 0.5, 3.0)
            s["clouds"].append(c)
        rng = np.random.default_rng(seed)
        q = case["queries"]
        radii = (0.5 + 2.5 * (rng.permutation(q) + 0.5) / q).round(3)
        s["queries"] = [(s["clouds"][i % 3], float(radii[i]), 1 + i % species, int(rng.integers(1, species + 1)), int(rng.integers(1, 21)))
                        for i in range(q)]
        s["server"] = N.Server(own, slots=case["slots"], budget_bytes=16 << 30)
        return s
    s["cloud"] = _Cloud(ctx, xyz, lab, _hull(shape, n) if case.get("hull", True) else None)
    s["trg"], s["env"] = _tasks(case.get("tasks", "pairs"), species)
    if kind == "pass":
        s["k"] = _orders(case)
        s["flags"] = (N.PP_RDF if case["rdf"] else 0) | (N.PP_1NN if case["nn1"] else 0) | (N.PP_RIPK if case["ripk"] else 0) | \
            (N.PP_MKNN if case["k"] else 0)
        s["perm"] = torch.randperm(n, generator=_generator(seed + 1), device="cuda").cpu().numpy().astype(np.uint32) if case["shuffled"] else None
    elif kind == "batched":
        g = _generator(seed + 1)
        s["k"] = _orders(case)
        s["sets"] = torch.stack([lab[torch.randperm(n, generator=g, device="cuda")] for _ in range(case["shuffles"])])
        length, r0 = _tip_length(n), _tip_apex(n)
        rng = np.random.default_rng(seed)
        z, r, phi = rng.uniform(0, length, case["rois"]), r0 * np.sqrt(rng.random(case["rois"])), rng.uniform(0, 2 * np.pi, case["rois"])
        rad = np.exp(rng.uniform(np.log(5.0), np.log(40.0), case["rois"]))
        s["rois"] = np.stack((r * np.cos(phi), r * np.sin(phi), z, rad), 1).astype(np.float32) if case["rois"] else None
    elif kind == "counts":
        ctx.set_option("npcorr_order", 0)
        s["trg"], s["env"] = [[2], [3]], [list(range(1, species + 1)), [2, 3]]
    return s


# -------------------------------------------------------------------- run
def _result(ctx):
    st = ctx.stats()
    return {"bins": ctx.fetch(), "centres": st["centres"], "discarded": st["discarded"], "pairs": st["pairs"]}


def run(s):
    case, kind = s["case"], s["kind"]
    if kind == "surface":
        err = ctypes.create_string_buffer(256)
        rc = N.load().pp_surfdist_noalloc(s["xyz"].data_ptr(), s["n"], s["tri"].data_ptr(), s["tri"].shape[0],
                                          max(case["R"], CARVE), s["out"].data_ptr(), None, err, 256)
        if rc:
            raise N.PPError(rc, err.value.decode())
        return s["out"]
    if kind == "served":
        srv = s["server"]
        tickets = [srv.submit(c, N.PP_RDF | N.PP_MKNN, (0.0, 0.01, R), [[a]], [[b]], [k]) for c, R, a, b, k in s["queries"]]
        got = [srv.wait(t, cap=1 << 14) for t in tickets]
        return {"bins": np.concatenate([g[0] for g in got]), "pairs": np.array([g[1] for g in got], dtype=np.uint64)}
    ctx = s["ctx"]
    if kind == "job":
        cid = ctx.upload_pos(s["pos"], s["ranges"])
        ctx.hull(cid, s["hull"], CARVE)
        inside = ctx.inside(cid, 1.0, 1.0)
        ctx.tasks(s["trg"], s["env"])
        ctx.hist(0.0, case["incr"], case["R"])
        ctx.run(cid, N.PP_RDF)
        rdf = _result(ctx)
        ctx.run(cid, N.PP_1NN | N.PP_MKNN, list(range(case["k"], 0, -1)))
        knn = _result(ctx)
        ctx.free(cid)
        return {"rdf": rdf, "knn": knn, "inside": [inside["nions_inside"], float(inside["volume_inside"])]}
    cid = s["cloud"].id
    if kind == "neighbours":
        ids, d2 = ctx.neighbors(cid, s["ion"], case["R"])
        m = min(ids.size, s["room"])                          # a program's own arrays, as long for every ion
        out = {"ids": np.zeros(s["room"], dtype=np.uint64), "d2": np.zeros(s["room"], dtype=np.float32)}
        out["ids"][:m], out["d2"][:m] = ids[:m], d2[:m]
        return out
    ctx.tasks(s["trg"], s["env"])
    ctx.hist(0.0, case["incr"], case["R"])
    if kind == "pass":
        ctx.run(cid, s["flags"], s["k"], label_perm=s["perm"])
        return _result(ctx)
    if kind == "batched":
        ctx.run_batched(cid, N.PP_RDF | N.PP_MKNN, s["k"], include_original=True, label_sets=s["sets"].data_ptr(),
                        nsets=s["sets"].shape[0], rois=s["rois"])
        count = ctx.batched_count()
        return {"bins": np.stack([ctx.fetch_batched(r) for r in range(count)]).view(np.int64),
                "pairs": np.array([ctx.batched_stats(r)["pairs"] for r in range(count)], dtype=np.uint64)}
    ctx.set_option("npcorr_order", case["order"])
    ctx.run(cid, N.PP_CNTNB | N.PP_NPCORR)
    ctx.set_option("npcorr_order", 0)
    counts = np.zeros((2, 4096), dtype=np.uint64)             # as long as a count may be
    got = ctx.fetch_cntnb()
    counts[:, : got.shape[1]] = got
    return {"counts": counts, "npcorr": ctx.fetch_npcorr()}


# ------------------------------------------------------------------- work
def _bins(case):
    return int(case["R"] / case["incr"]) + 2


def _fractions(shape, species):
    if shape == "cylinder":
        return list(CYL_FRACTIONS)
    minor = list(TIP_IID[: max(0, species - 3)])
    return [1.0 - 0.005 - sum(minor), 0.0035, 0.0015] + minor


def work(case):
    """Bytes: every input read and every result written once.  Flops: three differences, three squares and two sums
    per in-ball pair, a pair of two centres once."""
    kind, n = case["kind"], case["n"]
    shape, species = case.get("shape", "tip"), case.get("species", 6)
    rho = TIP_RHO if shape == "tip" else CYL_RHO
    if kind == "surface":
        tri = len(_hull("tip", n, case["nseg"], case["stack"]))
        shell = min(1.0, 2.0 * max(case["R"], CARVE) / _tip_apex(n))       # ions within R' of the side
        return {"bytes": 12.0 * n + 36.0 * tri + 4.0 * n, "flops": 60.0 * n * shell}
    if kind == "neighbours":
        ball = rho * 4.19 * case["R"] ** 3
        return {"bytes": 28.0 * ball, "flops": 8.0 * ball}
    ball = lambda R: rho * 4.19 * R ** 3  # noqa: E731
    if kind == "served":
        f = _fractions(shape, species)
        pairs = 0.0
        for i in range(case["queries"]):
            m = (n, max(1000, n // 4), max(1000, n // 10))[i % 3]
            pairs += m * f[i % species] * ball(0.5 + 2.5 * (i + 0.5) / case["queries"])
        return {"bytes": 16.0 * n * 1.35 + 8.0 * 350 * case["queries"], "flops": 8.0 * pairs}
    f = _fractions(shape, species)
    H = _bins(case)
    if kind == "counts":
        edge = 3 + 2 * math.ceil(case["R"] / case["incr"])
        return {"bytes": 13.0 * n + 2 * (8.0 * 4096 + 4.0 * edge ** 3), "flops": 8.0 * n * 0.005 * ball(case["R"])}
    if kind == "batched":
        real = 1 + case["shuffles"]
        hists = species * species * (1 + case["k"])
        return {"bytes": 13.0 * n + 1.0 * n * case["shuffles"] + 8.0 * H * hists * (real + case["rois"]), "flops": 4.0 * n * ball(case["R"])}
    if kind == "job":
        hists = species * species * (2 + case["k"])
        return {"bytes": 16.0 * n + 8.0 * H * hists, "flops": 4.0 * n * ball(case["R"])}
    ntask = {"pairs": species * species, "solute": 1, "overlapping": 3}[case["tasks"]]
    hists = ntask * (int(case["rdf"]) + int(case["nn1"]) + int(case["ripk"]) + len(_orders(case)))
    sparse = case["tasks"] == "solute"
    flops = 8.0 * n * f[1] * ball(case["R"]) if sparse else 4.0 * n * ball(case["R"])
    return {"bytes": (17.0 if case["shuffled"] else 13.0) * n + 8.0 * H * hists, "flops": flops}


# ------------------------------------------------------------------ exact
def exact(case, seed):
    """Distances in 64 bits.  Everything else this framework returns is whole numbers."""
    if case["kind"] == "neighbours":
        s = prepare(case, seed)
        p = s["xyz"]
        d = p - p[s["ion"]]
        sq = d * d
        near = ((sq[:, 0] + sq[:, 1]) + sq[:, 2]) <= torch.tensor(case["R"], dtype=torch.float32, device="cuda") ** 2
        near[s["ion"]] = False                                # the members: single-precision distances, as documented
        e = p[near].double() - p[s["ion"]].double()
        d2 = np.zeros(s["room"], dtype=np.float64)
        e = (e * e).sum(1).sort().values.cpu().numpy()[: s["room"]]
        d2[: e.size] = e
        return {"ids": None, "d2": d2}
    if case["kind"] != "surface":
        return None
    s = prepare(case, seed)
    p, tri = s["xyz"].double(), s["tri"].double()
    if p.shape[0] * tri.shape[0] > 6e10:
        return None
    rp = max(float(np.float32(case["R"])), CARVE)
    out = torch.full((p.shape[0],), float(np.float32(rp) * np.float32(rp)), dtype=torch.float64, device="cuda")
    order = torch.argsort(p[:, 2])
    tlo, thi = tri[:, 2::3].min(1).values - rp - 1e-3, tri[:, 2::3].max(1).values + rp + 1e-3
    step = 20_000
    for a in range(0, p.shape[0], step):
        at = order[a: a + step]
        q = p[at]
        t = tri[(thi >= q[0, 2]) & (tlo <= q[-1, 2])]
        for b in range(0, t.shape[0], 1000):
            out[at] = torch.minimum(out[at], _closest2(q, t[b: b + 1000]))
    return out


def _closest2(q, t):
    """Smallest squared distance of each point to the triangles: inside the face, or to one of the three edges."""
    a, b, c = t[None, :, 0:3], t[None, :, 3:6], t[None, :, 6:9]
    p = q[:, None, :]
    ab, ac, ap = b - a, c - a, p - a
    n = torch.linalg.cross(ab, ac)
    nn = (n * n).sum(-1)
    height = (ap * n).sum(-1) / nn
    v = (torch.linalg.cross(ap, ac.expand_as(ap)) * n).sum(-1) / nn
    w = (torch.linalg.cross(ab.expand_as(ap), ap) * n).sum(-1) / nn
    best = torch.where((v >= 0) & (w >= 0) & (v + w <= 1), height * height * nn, torch.full_like(v, math.inf))
    for o, e in ((a, b - a), (a, c - a), (b, c - b)):
        f = p - o
        x = ((f * e).sum(-1) / (e * e).sum(-1)).clamp(0, 1)
        d = f - x[..., None] * e
        best = torch.minimum(best, (d * d).sum(-1))
    return best.min(1).values
