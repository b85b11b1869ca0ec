"""FP64 walk where a cell's moments overflow: its centre of mass is infinite on
one axis and undefined on the other.  A body's own test compares with NaN and
opens such a cell; the test against a group's box has to say the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 9000, 20000, 70000, 140000])
def test_undefined_centres_are_opened(nbp, orc, n):
    rng = np.random.default_rng(n)
    p = rng.normal(size=(n, 2)) * 1e150
    p[:, 1] = np.abs(p[:, 1])
    m = np.full(n, 1e200)
    with nbp.NbContext(nbp.SimConfig(theta=0.5), m, p, np.zeros_like(p)) as ctx:
        ctx.accelerations()
        st = ctx.stats()
    ref = orc.RefState(m, p, np.zeros_like(p))
    r = ref.step(theta=0.5, eps2=1e-4, integrate=False, want_acc=True)
    assert st.cell_interactions == r["stats"]["cell_interactions"]
    assert st.body_interactions == r["stats"]["body_interactions"]
