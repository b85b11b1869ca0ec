"""Learned corrections on the quadrupole walk: both the second moments and the
features climb the tree with the same arrival counters, so the second climb
must start from zero.  Otherwise cells above the directly summed size keep the
feature records of whatever cell had their number before."""
import pathlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WEIGHTS = pathlib.Path(__file__).resolve().parents[1] / "n-body-2d_b200" / "weights"


def test_corrections_depend_on_the_current_state_only(nbp):
    m, p, v = nbp.universes.colliding_discs(60000, 5)
    cfg = nbp.SimConfig(theta=0.5, epsilon_squared=1e-4, mode=nbp.NB_MODE_SPLIT, quadrupole=True,
                        learned=True, band_theta=0.4)
    w = np.load(WEIGHTS / "correction_quad_theta0.5.npy")
    with nbp.NbContext(cfg, m, p, v) as ctx:
        ctx.set_mlp_weights(w)
        ctx.step(5)
        pos, vel = ctx.download()
        a = ctx.accelerations()
    with nbp.NbContext(cfg, m, pos, vel) as ctx:
        ctx.set_mlp_weights(w)
        assert np.array_equal(ctx.accelerations(), a)


def test_every_sampled_cell_has_its_own_mass_and_shape(nbp):
    """Feature 3 is the heaviest child's mass fraction (between 1/4 and 1) and
    features 4 and 6 are the diagonal second moments over M w^2 (positive)."""
    m, p, v = nbp.universes.colliding_discs(60000, 5)
    cfg = nbp.SimConfig(theta=0.5, epsilon_squared=1e-4, mode=nbp.NB_MODE_SPLIT, quadrupole=True,
                        learned=True, band_theta=0.4)
    with nbp.NbContext(cfg, m, p, v) as ctx:
        ctx.set_mlp_weights(np.load(WEIGHTS / "correction_quad_theta0.5.npy"))
        x, _ = ctx.mlp_samples(200, seed=1)
    assert len(x) > 1000
    # BF16 features: 2^-9 relative
    assert (x[:, 3] > 0.25 * (1 - 2.0 ** -8)).all() and (x[:, 3] <= 1.0).all()
    assert (x[:, 4] + x[:, 6] > 0).all()
