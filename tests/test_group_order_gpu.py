"""Order of the SPLIT target groups: with 64 or 128 bodies to a group, those of
half the size or less follow all others; with 32, groups keep the order of the
keys.  Every body lies in exactly one group."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 65, 129, 2049, 30_000, 131_072, 300_007])
@pytest.mark.parametrize("lane_bodies", [1, 2, 4])
@pytest.mark.parametrize("kind", ["spread", "clumps", "one leaf"])
def test_small_groups_last(nbp, n, lane_bodies, kind):
    rng = np.random.default_rng(n + lane_bodies)
    p = rng.normal(size=(n, 2))
    if kind == "clumps":  # leaves of many bodies: chunks of whole groups and a rest
        p[n // 4: n // 2] = p[0]
        p[n // 2: n // 2 + n // 10] = p[n - 1]
    elif kind == "one leaf":
        p[:] = p[0]
    cfg = nbp.SimConfig(mode=nbp.NB_MODE_SPLIT, bodies_per_lane=lane_bodies)
    with nbp.NbContext(cfg, np.ones(n), p, np.zeros_like(p)) as ctx:
        ctx.accelerations()
        g = ctx.debug_groups().astype(np.int64)
    size, full = g[:, 1] - g[:, 0] + 1, 32 * lane_bodies
    order = np.argsort(g[:, 0])
    assert size.min() >= 1 and size.max() <= full
    assert g[order[0], 0] == 0 and g[order[-1], 1] == n - 1
    assert np.array_equal(g[order[1:], 0], g[order[:-1], 1] + 1)
    if lane_bodies > 1:
        small = size <= full // 2
        assert not (small[:-1] & ~small[1:]).any()
