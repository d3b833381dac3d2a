"""Hull distances where triangles are skipped by their boxes, and look-ups whose
neighbours come in two downloads."""
import ctypes as C

import numpy as np
import pytest

from paraprobe_gb300 import native as N

pytestmark = pytest.mark.gpu


def _triangles(rng, n, side):
    """Triangles of every shape around a cube: fat ones, slivers on both sides of
    sin^2 = 1e-5 between two edges, lines and points, from 0.2 to 1.5 sides long."""
    a = rng.uniform(-0.2, 1.2, (n, 3)) * side
    e0 = rng.normal(size=(n, 3))
    e0 *= (side * rng.uniform(0.2, 1.5, n) / np.linalg.norm(e0, axis=1))[:, None]
    w = np.cross(e0, rng.normal(size=(n, 3)))
    w /= np.linalg.norm(w, axis=1)[:, None]
    sin = np.choose(np.arange(n) % 6, [1.0, 0.05, 10 ** rng.uniform(-2.7, -2.3, n), 10 ** rng.uniform(-5, -3, n), 0.0, 0.0])
    e1 = rng.uniform(-1.0, 1.0, n)[:, None] * e0 + (sin * np.linalg.norm(e0, axis=1))[:, None] * w
    tri = np.stack([a, a + e0, a + e1], 1)
    tri[5::12] = tri[5::12, :1]                    # points
    tri[11::12, 2] = tri[11::12, 1]                # two vertices in one place
    return tri


@pytest.mark.parametrize("shift", [0.0, 4096.0, -300.0])
@pytest.mark.parametrize("R", [0.4, 2.0, 5.0])
def test_hull_of_slivers(ctx, oracle, shift, R):
    """A box farther than the nearest triangle so far skips its triangle, whatever
    the triangle's shape and wherever the cloud lies: the distances of both entry
    points are the oracle's, bit for bit."""
    import torch
    rng = np.random.default_rng(int(10 * R))
    side = 12.0
    xyz = (rng.uniform(0, side, (15000, 3)) + shift).astype(np.float32)
    tri = (_triangles(rng, 360, side) + shift).astype(np.float32).reshape(-1, 9)
    want = oracle.surface_distance(xyz, tri, np.float32(R))
    cid = ctx.upload(xyz, np.ones(len(xyz), dtype=np.uint8))
    try:
        ctx.hull(cid, tri, min(R, 0.3))
        ctx.tasks([[1]], [[1]])
        ctx.hist(0.0, R / 4, R)
        ctx.run(cid, N.PP_1NN)
        got = ctx.surfdist_fetch(cid, len(xyz))
    finally:
        ctx.free(cid)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    x, t = torch.from_numpy(xyz).cuda(), torch.from_numpy(tri).cuda()
    out, err = torch.empty(len(xyz), dtype=torch.float32, device="cuda"), C.create_string_buffer(256)
    rc = N.load().pp_surfdist_noalloc(C.c_void_p(x.data_ptr()), len(xyz), C.c_void_p(t.data_ptr()), len(tri), R,
                                      C.c_void_p(out.data_ptr()), None, err, 256)
    assert rc == 0, err.value
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("more", [-1, 0, 1, 3000])
def test_neighbours_beyond_the_first_download(ctx, oracle, more):
    """4,095 records come with the count, the others in a second download."""
    rng = np.random.default_rng(9)
    xyz = rng.uniform(0, 10, (9000, 3)).astype(np.float32)
    ids, d2 = oracle.neighbors(xyz, 42, 20.0)
    assert len(ids) == len(xyz) - 1
    d = np.sort(d2)[4095 + more - 1]               # so many of them lie within
    r = float(np.nextafter(np.sqrt(np.float32(d)), np.float32(np.inf)))
    want_ids, want = oracle.neighbors(xyz, 42, r)
    cid = ctx.upload(xyz, np.ones(len(xyz), dtype=np.uint8))
    try:
        got_ids, got = ctx.neighbors(cid, 42, r)
    finally:
        ctx.free(cid)
    assert abs(len(want_ids) - (4095 + more)) <= 1
    assert np.array_equal(got_ids, want_ids) and np.array_equal(got.view(np.uint32), want.view(np.uint32))
