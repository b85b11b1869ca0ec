"""Cell moments at the edges of the blocks that compute them: masses and centres
of mass of every cell equal the direct sums over its bodies, for body counts
around one block, cells that reach over blocks, and multi-body leaves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 5, 1023, 1024, 1025, 2049, 5000])
@pytest.mark.parametrize("quad", [False, True])
def test_cell_moments_equal_direct_sums(nbp, n, quad):
    rng = np.random.default_rng(n)
    p, m = rng.normal(size=(n, 2)), rng.random(n) + 0.5
    if n > 100:
        p[7:60] = p[7]          # a leaf of 53 bodies
        p[n // 2] = p[n // 2 + 1]
    mode = nbp.NB_MODE_SPLIT if quad else nbp.NB_MODE_FP64
    with nbp.NbContext(nbp.SimConfig(mode=mode, quadrupole=quad), m, p, np.zeros((n, 2))) as ctx:
        ctx.accelerations()
        t = ctx.debug_tree()
        mass, pos, _, _ = ctx.debug_state()
    # differences of prefix sums in long double: exact enough to compare with
    cm = np.concatenate([[0], np.cumsum(mass.astype(np.longdouble))])
    cr = np.concatenate([np.zeros((1, 2)), np.cumsum(mass[:, None].astype(np.longdouble) * pos, 0)])
    a, b = t["first"], t["last"] + 1
    M = cm[b] - cm[a]
    R = (cr[b] - cr[a]) / M[:, None]
    # a cell adds at most 4 terms per level and 30 levels, each rounded by 2^-53
    bound = 120 * 2.0 ** -53
    assert (np.abs(t["mass"] - M) <= bound * M + 1e-17 * cm[-1]).all()
    assert (np.abs(t["com"] - R) <= 4 * bound * np.abs(pos).max()).all()
