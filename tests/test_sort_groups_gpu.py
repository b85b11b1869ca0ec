"""Digit passes whose tiles take their places from groups of eight tiles: sizes
around whole tiles and groups of 1,024, 2,048 or 3,072 keys to a tile, with more
groups than a look-back has in flight.  Codes and permutation are compared with
the oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE, GROUP = 3072, 8 * 3072


@pytest.mark.parametrize("n", [11 * TILE + 1, 2 * GROUP - 1, 2 * GROUP, 2 * GROUP + 1,
                               2 * GROUP + TILE, 5 * GROUP, 5 * GROUP + 1, 43 * GROUP - 5])
@pytest.mark.parametrize("kind", ["spread", "clustered"])
def test_sort_groups(nbp, orc, n, kind):
    rng = np.random.default_rng(n)
    p = rng.normal(size=(n, 2)) * [4.0, 1.0]
    if kind == "clustered":  # whole groups of tiles with one top digit, and ties
        p[n // 8:] = 1e-7 * rng.normal(size=(n - n // 8, 2))
        p[n // 2:n // 2 + n // 16] = p[n // 2]
    p = np.ascontiguousarray(p)
    codes_o, order_o = orc.stable_sort(orc.morton(p))
    with nbp.NbContext(nbp.SimConfig(), np.ones(n), p, np.zeros((n, 2))) as ctx:
        for passes in (0, 5, 8):
            ctx.debug_sort_passes(passes)
            codes, order, _ = ctx.debug_morton()
            assert np.array_equal(codes, codes_o), passes
            assert np.array_equal(order, order_o), passes
