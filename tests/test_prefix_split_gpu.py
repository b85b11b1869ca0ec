"""SPLIT monopoles where the prefix sums take another form: up to 256 tiles of
2,048 bodies each block scans the tiles' totals itself (one warp, eight totals
per lane), above a kernel of its own does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE = 2048


@pytest.mark.parametrize("n", [TILE - 1, TILE, TILE + 1, 9 * TILE, 255 * TILE + 1, 256 * TILE - 1,
                               256 * TILE, 256 * TILE + 1, 257 * TILE + 5])
def test_cells_from_prefix_sums(nbp, n):
    rng = np.random.default_rng(n)
    p, m = rng.normal(size=(n, 2)), rng.random(n) + 0.5
    with nbp.NbContext(nbp.SimConfig(mode=nbp.NB_MODE_SPLIT), m, p, np.zeros_like(p)) as ctx:
        ctx.accelerations()
        t = ctx.debug_tree()
        mass, pos, _, _ = ctx.debug_state()
        _, order, box = ctx.debug_morton()
    assert np.array_equal(order, np.arange(n))
    first, last = t["first"], t["last"]
    assert (last == n - 1).any() and (last - first + 1 == n).sum() == 1  # the last total is used
    c = np.array([box[0] + box[1], box[2] + box[3]]) / 2
    terms = np.stack([mass, mass * (pos[:, 0] - c[0]), mass * (pos[:, 1] - c[1])]).astype(np.longdouble)
    total = np.concatenate([np.zeros((3, 1)), np.cumsum(terms, axis=1)], axis=1)
    want = total[:, last + 1] - total[:, first]
    # each prefix sum takes at most 8 rows, 8 warps, 8 tiles, 32 lanes and as many
    # tiles again one after the other: below 64 + tiles / 8 roundings, of sums no
    # larger than the sum of all magnitudes; then a difference and a division
    u = 2.0 ** -53 * (64 + n // (8 * TILE)) * np.abs(terms).sum(axis=1)
    assert (np.abs(t["mass"] - want[0]) <= 2 * u[0]).all()
    for k in (0, 1):
        com = c[k] + want[k + 1] / want[0]
        bound = 4 * (u[k + 1] + np.abs(want[k + 1] / want[0]) * u[0]) / want[0] + 2.0 ** -50 * np.abs(com)
        assert (np.abs(t["com"][:, k] - com) <= bound).all()
