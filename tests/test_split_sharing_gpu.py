"""SPLIT walks whose block shares a group (up to 24,576 bodies), and groups whose
bodies have two or four lanes each: at theta = 0 every body is summed directly
by exactly one lane of one warp."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS2 = 1e-4


@pytest.mark.parametrize("n", [1, 2, 7, 9, 17, 33, 40, 1000, 24576, 24577])
@pytest.mark.parametrize("quad", [False, True])
@pytest.mark.parametrize("lane_bodies", [0, 2])
def test_every_pair_once(nbp, orc, n, quad, lane_bodies):
    rng = np.random.default_rng(n)
    p, m = rng.normal(size=(n, 2)), rng.random(n) + 0.5
    cfg = nbp.SimConfig(theta=0.0, epsilon_squared=EPS2, mode=nbp.NB_MODE_SPLIT, quadrupole=quad,
                        bodies_per_lane=lane_bodies)
    with nbp.NbContext(cfg, m, p, np.zeros_like(p)) as ctx:
        a = ctx.accelerations()
        st = ctx.stats()
        box = ctx.debug_morton()[2]
    assert st.cell_interactions == 0
    assert st.body_interactions == n * (n - 1)
    tgt = np.unique(np.linspace(0, n - 1, 500).astype(np.int64))
    center = np.array([0.5 * (box[0] + box[1]), 0.5 * (box[2] + box[3])])
    exact = orc.allpairs_plummer(m, p, tgt, eps2=EPS2)
    bound = orc.allpairs_fp32_bound(m, p, center, targets=tgt, eps2=EPS2)
    assert (np.linalg.norm(a[tgt] - exact, axis=1) <= bound).all()
