"""The FP64 walk over groups of bodies against the CPU oracle: every group size
at the body counts where the next one takes over, ragged ends, multi-body
leaves, and distances whose squares leave FP64's normal range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS2 = 1e-4


def accelerations(nbp, m, p, theta, eps2):
    cfg = nbp.SimConfig(theta=theta, epsilon_squared=eps2)
    with nbp.NbContext(cfg, m, p, np.zeros_like(p)) as ctx:
        return ctx.accelerations(), ctx.stats()


# group sizes 1, 2, 4, 8, 16, 32 start at 0, 8192, 16384, 32768, 65536, 131072 bodies
@pytest.mark.parametrize("n", [5, 33, 8191, 8193, 16387, 32769, 65537, 131075])
@pytest.mark.parametrize("theta", [0.5, 1.0])
def test_group_walk_matches_oracle(nbp, orc, n, theta):
    m, p, v = nbp.universes.plummer_disc(n, n)
    acc, st = accelerations(nbp, m, p, theta, EPS2)
    ref = orc.RefState(m, p, v)
    r = ref.step(theta=theta, eps2=EPS2, integrate=False, want_acc=True)
    assert st.cell_interactions == r["stats"]["cell_interactions"]
    assert st.body_interactions == r["stats"]["body_interactions"]
    # both sums round at most 2,048 terms, four roundings of 2^-53 each, of
    # terms whose magnitudes add up to little more than the all-pairs sum's
    tgt = np.unique(np.linspace(0, n - 1, 200).astype(np.int64))
    bound = 2 * 4 * 2048 * 2.0 ** -53 * orc.allpairs_plummer_abs(m, p, tgt, eps2=EPS2)
    err = np.abs(acc - ref.in_original_order(r["acc"]))[tgt].max(axis=1)
    assert (err <= bound).all(), (err / bound).max()


@pytest.mark.parametrize("n", [300, 20000])
def test_multi_body_leaves_in_groups(nbp, orc, n):
    """Clumps of coincident bodies: leaves that hold part of a group, all of
    it, and more than a group."""
    rng = np.random.default_rng(n)
    p = rng.normal(size=(n, 2))
    p[10:40] = p[10]
    p[50:57] = p[50]
    p[100:250] = p[100]
    m = rng.random(n) + 0.5
    for theta in (0.5, 1.2):
        acc, st = accelerations(nbp, m, p, theta, EPS2)
        ref = orc.RefState(m, p, np.zeros_like(p))
        r = ref.step(theta=theta, eps2=EPS2, integrate=False, want_acc=True)
        assert st.cell_interactions == r["stats"]["cell_interactions"]
        assert st.body_interactions == r["stats"]["body_interactions"]
        acc_o = ref.in_original_order(r["acc"])
        assert np.abs(acc - acc_o).max() <= 1e-11 * np.abs(acc_o).max()


@pytest.mark.parametrize("n,scale", [(2, 1e-155), (2, 1e-200), (40, 1e160), (20000, 1e160)])
def test_squares_outside_the_normal_range(nbp, orc, n, scale):
    """d^2 subnormal, zero or infinite: the same infinities, NaN and zeros as
    the oracle's 1/sqrt."""
    rng = np.random.default_rng(n)
    p = rng.normal(size=(n, 2)) * scale
    m = np.ones(n)
    acc, _ = accelerations(nbp, m, p, 0.5, 0.0)
    ref = orc.RefState(m, p, np.zeros_like(p))
    r = ref.step(theta=0.5, eps2=0.0, integrate=False, want_acc=True)
    assert np.array_equal(acc, ref.in_original_order(r["acc"]), equal_nan=True)
