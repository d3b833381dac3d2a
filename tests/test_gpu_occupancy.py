"""The occupancy grid's clusters and classes against the oracle: grids of one
block and of many, porous clouds whose empty voxels form winding clusters, and
grids on either side of the line between the two forms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,side,width", [(1, 1.0, 1.0), (40, 6.0, 2.0), (300, 9.0, 1.0), (900, 12.9, 1.0), (1100, 13.1, 1.0),
                                          (2000, 14.0, 0.7), (6000, 25.0, 1.0), (20000, 40.0, 0.9), (5000, 40.0, 0.8)])
@pytest.mark.parametrize("kind", ["porous", "shell"])
def test_inside_matches_oracle(ctx, oracle, n, side, width, kind):
    rng = np.random.default_rng(n)
    xyz = rng.uniform(0, side, (n, 3))
    if kind == "shell" and n > 1:  # a hollow ball with a hole: vacuum inside and out
        u = rng.normal(size=(n, 3))
        u /= np.linalg.norm(u, axis=1)[:, None]
        u = u[u[:, 0] < 0.9]
        xyz = side / 2 + u * (side / 2 - rng.uniform(0, 1.0, (len(u), 1)))
    xyz = xyz.astype(np.float32)
    cid = ctx.upload(xyz, np.ones(len(xyz), dtype=np.uint8))
    try:
        got = [ctx.inside(cid, width, width) for _ in range(5)]
    finally:
        ctx.free(cid)
    want = oracle.voxelize(xyz, width, width)
    assert all(g == want for g in got)
