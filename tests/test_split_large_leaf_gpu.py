"""SPLIT walks that meet a leaf of more than 65,536 coincident bodies, whose
places are counted by a scan of their own, and one just below: at theta = 0
every body is summed directly exactly once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS2 = 1e-4


@pytest.mark.parametrize("clump", [65536, 65537, 70001])
def test_every_pair_once(nbp, orc, clump):
    n = clump + 3001
    rng = np.random.default_rng(clump)
    p, m = rng.normal(size=(n, 2)), rng.random(n) + 0.5
    p[1000:1000 + clump] = p[1000]
    cfg = nbp.SimConfig(theta=0.0, epsilon_squared=EPS2, mode=nbp.NB_MODE_SPLIT)
    with nbp.NbContext(cfg, m, p, np.zeros_like(p)) as ctx:
        a = ctx.accelerations()
        st = ctx.stats()
        box = ctx.debug_morton()[2]
    assert st.cell_interactions == 0
    assert st.body_interactions == n * (n - 1)
    tgt = np.unique(np.linspace(0, n - 1, 300).astype(np.int64))
    center = np.array([0.5 * (box[0] + box[1]), 0.5 * (box[2] + box[3])])
    exact = orc.allpairs_plummer(m, p, tgt, eps2=EPS2)
    bound = orc.allpairs_fp32_bound(m, p, center, targets=tgt, eps2=EPS2)
    assert (np.linalg.norm(a[tgt] - exact, axis=1) <= bound).all()
