"""Digit passes with 4, 8 and 12 keys per thread: contexts one body around the
sizes where the tile changes (one tile of 1,024 keys per SM; four tiles of 2,048
per SM) and around whole tiles.  Codes and permutation are compared with the
oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles, keys, off", [
    (33, 1024, -1), (33, 1024, 0), (33, 1024, 1), ("sms", 1024, 0), ("sms", 1024, 1),
    (200, 2048, -3), (200, 2048, 0), (200, 2048, 2), ("4 sms", 2048, 0), ("4 sms", 2048, 1)])
@pytest.mark.parametrize("kind", ["spread", "clustered"])
def test_tile_sizes(nbp, orc, tiles, keys, off, kind):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = {"sms": sms, "4 sms": 4 * sms}.get(tiles, tiles) * keys + off
    rng = np.random.default_rng(n)
    p = rng.normal(size=(n, 2)) * [4.0, 1.0]
    if kind == "clustered":  # most keys share their top bytes; ties of every size
        p[n // 8:] = 1e-7 * rng.normal(size=(n - n // 8, 2))
        p[n // 2:n // 2 + n // 16] = p[n // 2]
    p = np.ascontiguousarray(p)
    codes_o, order_o = orc.stable_sort(orc.morton(p))
    with nbp.NbContext(nbp.SimConfig(), np.ones(n), p, np.zeros((n, 2))) as ctx:
        for passes in (0, 4, 8):
            ctx.debug_sort_passes(passes)
            codes, order, _ = ctx.debug_morton()
            assert np.array_equal(codes, codes_o), passes
            assert np.array_equal(order, order_o), passes
