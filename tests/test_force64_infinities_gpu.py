"""FP64 walk, no softening, bodies so close that m / r^3 overflows although r^2
is a normal number: the infinities (and the NaN of opposite ones) of the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def both(nbp, orc, m, p):
    with nbp.NbContext(nbp.SimConfig(theta=0.5, epsilon_squared=0.0), m, p, np.zeros_like(p)) as ctx:
        acc = ctx.accelerations()
    ref = orc.RefState(m, p, np.zeros_like(p))
    r = ref.step(theta=0.5, eps2=0.0, integrate=False, want_acc=True)
    return acc, ref.in_original_order(r["acc"])


# 40 bodies one per warp, 20,000 with entries that act on some of a group's
# bodies, 70,000 and 140,000 with a list of their own for these
@pytest.mark.parametrize("n", [2, 40, 20000, 70000, 140000])
@pytest.mark.parametrize("scale", [2.0 ** -400, 1e-110, 1e-130])
def test_every_term_overflows(nbp, orc, n, scale):
    acc, want = both(nbp, orc, np.ones(n), np.random.default_rng(n).normal(size=(n, 2)) * scale)
    assert np.isinf(want).any()
    assert np.array_equal(acc, want, equal_nan=True)


@pytest.mark.parametrize("n", [2000, 20000, 70000, 140000])
def test_some_terms_overflow(nbp, orc, n):
    """Only neighbours closer than 8e-103 overflow."""
    p = np.random.default_rng(n).normal(size=(n, 2)) * 1e-102 * np.sqrt(n)
    acc, want = both(nbp, orc, np.ones(n), p)
    assert np.isinf(want).sum() > 10 and np.isfinite(want).sum() > n // 4
    ok = np.isfinite(want)
    assert np.array_equal(acc[~ok], want[~ok], equal_nan=True)
    # sums of a few hundred to thousands of terms in another order
    assert np.abs(acc[ok] - want[ok]).max() <= 1e-11 * np.abs(want[ok]).max()


@pytest.mark.parametrize("n", [40, 20000, 70000, 140000])
def test_a_close_pair_in_a_leaf(nbp, orc, n):
    p = np.random.default_rng(n).normal(size=(n, 2))
    p[0], p[1] = [0.0, 0.0], [1e-110, 2e-111]
    acc, want = both(nbp, orc, np.ones(n), p)
    assert np.array_equal(acc[:2], want[:2]) and np.isinf(want[:2]).all()
    assert np.abs(acc[2:] - want[2:]).max() <= 1e-11 * np.abs(want[2:]).max()


@pytest.mark.parametrize("x", [2.0 ** -400, 2.0 ** -342, 3e-104, 1e-130])
def test_two_bodies_on_an_axis(nbp, orc, x):
    """One term, exact squares among them (where the series' correction is zero)."""
    acc, want = both(nbp, orc, np.array([1.0, 3.0]), np.array([[0.0, 1e-200], [x, 1e-200]]))
    assert np.isinf(want[:, 0]).all() and np.array_equal(acc, want, equal_nan=True)
