"""The tree kernels where their splits change: 64 tiles of 2,048 bodies (the
other tiles' tables are read in place up to there) and 148 (1,024 threads per
tile, prefix sums without a scan kernel)."""
import numpy as np
import pytest

from test_parity_gpu import _cells_from_codes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 64 * 2048, 64 * 2048 + 1, 148 * 2048, 148 * 2048 + 1])
def test_cells_and_groups(nbp, n):
    m, p, v = nbp.universes.plummer_disc(n, n)
    if n > 1000:
        p[100:140] = p[100]  # a multi-body leaf
        p[n // 2:n // 2 + 5] = p[n // 2]
    cfg = nbp.SimConfig(mode=nbp.NB_MODE_SPLIT)
    with nbp.NbContext(cfg, m, p, v) as ctx:
        ctx.accelerations()
        t = ctx.debug_tree()
        groups = ctx.debug_groups()
        mass, pos, _, _ = ctx.debug_state()
        codes, order, _ = ctx.debug_morton()
    assert np.array_equal(order, np.arange(n))
    # groups tile the bodies, in slots' order once sorted
    g = groups[np.argsort(groups[:, 0])]
    assert g[0, 0] == 0 and g[-1, 1] == n - 1 and (g[1:, 0] == g[:-1, 1] + 1).all()
    if n < 3:
        return
    got = set(zip(t["first"].tolist(), t["last"].tolist(), t["level"].tolist()))
    assert len(got) == len(t["first"])
    assert got == _cells_from_codes(codes)
    # monopoles from the prefix sums: rounded by 2^-53 of the whole sum's terms
    # (n additions in blocks of 2,048, then of tiles), relative to the box centre
    cm = np.concatenate([[0], np.cumsum(mass.astype(np.longdouble))])
    M = cm[t["last"] + 1] - cm[t["first"]]
    assert (np.abs(t["mass"] - M) <= 64 * 2.0 ** -53 * cm[-1]).all()
