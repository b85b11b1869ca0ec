"""Target groups on both sides of the size up to which small ones are listed
last, 2,097,152 bodies.  Leaves of many coincident bodies emit one group per 64
or 128 of them from a single cell, which fills the packed counts most.  (A leaf
of all bodies would fill them to their limit, but the walk that follows takes
every pair of a leaf.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMIT = 2097152


@pytest.mark.parametrize("n", [LIMIT, LIMIT + 1])
@pytest.mark.parametrize("lane_bodies", [2, 4])
@pytest.mark.parametrize("kind", ["spread", "clumps", "large leaf"])
def test_groups_at_the_limit(nbp, n, lane_bodies, kind):
    p = np.random.default_rng(n + lane_bodies).normal(size=(n, 2))
    if kind == "clumps":  # 30 leaves of some 60,000 bodies among the others
        for k in range(30):
            p[k * 69000: k * 69000 + 60000 + 7 * k] = p[k * 69000]
    elif kind == "large leaf":
        p[1000: 301005] = p[1000]
    cfg = nbp.SimConfig(mode=nbp.NB_MODE_SPLIT, bodies_per_lane=lane_bodies, theta=1.0)
    with nbp.NbContext(cfg, np.ones(n), p, np.zeros_like(p)) as ctx:
        ctx.accelerations()
        g = ctx.debug_groups().astype(np.int64)
    size, full = g[:, 1] - g[:, 0] + 1, 32 * lane_bodies
    order = np.argsort(g[:, 0])
    assert size.min() >= 1 and size.max() <= full
    assert g[order[0], 0] == 0 and g[order[-1], 1] == n - 1
    assert np.array_equal(g[order[1:], 0], g[order[:-1], 1] + 1)
    small = size <= full // 2
    mixed = (small[:-1] & ~small[1:]).any()
    assert mixed == (n > LIMIT)  # above, cell by cell
