"""The all-pairs kernels at the edges of their splits: one target, targets
around a block and around the switch to two per thread, few sources, and
squared distances that are zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS2 = 1e-4


def bounded(acc, exact, p, m, tgt, law):
    """At most n terms are rounded a few times each, by 2^-53 of the sum of
    magnitudes (the terms' own rounding: 8 of 2^-53)."""
    d = p[None, :, :] - p[tgt][:, None, :]
    r2 = (d ** 2).sum(-1)
    w = m / (np.sqrt(r2) * (r2 + EPS2) + 1e-300) if law == "cpu" else m * (r2 + EPS2) ** -1.5
    w[r2 == 0.0] = 0.0
    size = (w * np.sqrt(r2)).sum(1)
    return (np.abs(acc - exact).max(axis=1) <= (len(m) + 8) * 2.0 ** -53 * size).all()


@pytest.mark.parametrize("n,k", [(1, 1), (2, 2), (31, 31), (1000, 1), (1000, 127), (1000, 129),
                                 (40000, 1), (20000, 16383), (20000, 16385)])
def test_exact_forces_of_any_number_of_targets(nbp, orc, n, k):
    rng = np.random.default_rng(n + k)
    p, m = rng.normal(size=(n, 2)), rng.random(n) + 0.5
    tgt = rng.permutation(n)[:k].astype(np.int64)
    acc = nbp.allpairs_accelerations(m, p, tgt, EPS2)
    some = np.unique(np.linspace(0, k - 1, 40).astype(np.int64))
    exact = orc.allpairs_plummer(m, p, tgt[some], eps2=EPS2)
    assert bounded(acc[some], exact, p, m, tgt[some], "plummer")


@pytest.mark.parametrize("n", [1, 2, 33, 300, 16383, 16385])
@pytest.mark.parametrize("law", ["plummer", "cpu"])
def test_all_pairs_mode_sizes(nbp, orc, n, law):
    rng = np.random.default_rng(n)
    p, m = rng.normal(size=(n, 2)), rng.random(n) + 0.5
    cfg = nbp.SimConfig(mode=nbp.NB_MODE_ALLPAIRS, epsilon_squared=EPS2, cpu_law=law == "cpu")
    with nbp.NbContext(cfg, m, p, np.zeros_like(p)) as ctx:
        acc = ctx.accelerations()
    some = np.unique(np.linspace(0, n - 1, 40).astype(np.int64))
    exact = (orc.allpairs_cpulaw if law == "cpu" else orc.allpairs_plummer)(m, p, some, eps2=EPS2)
    assert bounded(acc[some], exact, p, m, some, law)


@pytest.mark.parametrize("law", ["plummer", "cpu"])
@pytest.mark.parametrize("n", [40, 17000])
def test_zero_distances_without_softening(nbp, n, law):
    """Two coincident bodies: their own forces are undefined (0 * inf), every
    other body's is finite."""
    rng = np.random.default_rng(n)
    p, m = rng.normal(size=(n, 2)), np.ones(n)
    p[n - 3] = p[5]
    cfg = nbp.SimConfig(mode=nbp.NB_MODE_ALLPAIRS, epsilon_squared=0.0, cpu_law=law == "cpu")
    with nbp.NbContext(cfg, m, p, np.zeros_like(p)) as ctx:
        acc = ctx.accelerations()
    bad = ~np.isfinite(acc).all(axis=1)
    assert set(np.nonzero(bad)[0]) == {5, n - 3}
    acc = nbp.allpairs_accelerations(m, p, np.arange(n), 0.0)
    assert set(np.nonzero(~np.isfinite(acc).all(axis=1))[0]) == {5, n - 3}
