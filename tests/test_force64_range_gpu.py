"""FP64 walk at the ends of r^-3's range.  The reference forms 1 / r^3 and then
multiplies by the mass (BarnesHutCuda.cu:427-431): close to a light body 1 / r^3
overflows although m / r^3 would not, far from a heavy one it underflows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def both(nbp, orc, m, p, eps2=0.0, theta=0.5):
    with nbp.NbContext(nbp.SimConfig(theta=theta, epsilon_squared=eps2), m, p, np.zeros_like(p)) as ctx:
        acc = ctx.accelerations()
    ref = orc.RefState(m, p, np.zeros_like(p))
    r = ref.step(theta=theta, eps2=eps2, integrate=False, want_acc=True)
    return acc, ref.in_original_order(r["acc"])


@pytest.mark.parametrize("n", [2, 40, 9000, 20000, 70000, 140000])
@pytest.mark.parametrize("scale,mass", [(3e-125, 1e-92), (1e-110, 1e-20), (1e115, 1e150), (1e140, 1e120)])
def test_outside_the_range(nbp, orc, n, scale, mass):
    """Every 1 / r^3 is infinite or zero."""
    p = np.random.default_rng(n).normal(size=(n, 2)) * scale
    if scale > 1.0 and n > 2:  # no pair closer than 1e109
        s = int(np.ceil(np.sqrt(n)))
        p = (np.stack(np.divmod(np.arange(n), s), 1) + 0.25) * scale
    acc, want = both(nbp, orc, np.full(n, mass), p)
    assert np.isinf(want).any() if scale < 1.0 else not want.any()
    assert np.array_equal(acc, want, equal_nan=True)


@pytest.mark.parametrize("r", [1e105, 3e106, 1e107, 2.5e107, 4e107])
@pytest.mark.parametrize("mass", [1.0, 1e200])
def test_two_bodies_where_it_goes_subnormal(nbp, orc, r, mass):
    acc, want = both(nbp, orc, np.array([mass, mass]), np.array([[0.0, 0.0], [r, 0.0]]))
    # three roundings of r^-3 to the subnormal grid on one side, two on the other
    assert np.abs(acc[:, 0] - want[:, 0]).max() <= 5 * 2.0 ** -1074 * mass * r + 1e-15 * np.abs(want).max()
