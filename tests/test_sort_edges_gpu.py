"""Sort stage at the edges of its kernels: one cluster of 1 to 16 blocks with
one or two keys per thread, and above it onesweep (contexts) or counting passes
(the zero-allocation entry point).  Codes, permutation and box are compared
with the oracle bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bodies(n, kind):
    rng = np.random.default_rng(n)
    p = rng.normal(size=(n, 2)) * [4.0, 1.0]
    if kind == "clustered":  # most keys share their top bytes; ties of every size
        p[n // 8:] = 1e-7 * rng.normal(size=(n - n // 8, 2))
        p[n // 2:n // 2 + n // 16] = p[n // 2]
    return np.ascontiguousarray(p)


SIZES = [1, 33, 1023, 1025, 2049, 8193, 16384, 16385, 32767, 32768, 32769]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind", ["spread", "clustered"])
def test_context_sort(nbp, orc, n, kind):
    p = bodies(n, kind)
    codes_o, order_o = orc.stable_sort(orc.morton(p))
    with nbp.NbContext(nbp.SimConfig(), np.ones(n), p, np.zeros((n, 2))) as ctx:
        for passes in (0, 2, 5, 8):
            ctx.debug_sort_passes(passes)
            codes, order, box = ctx.debug_morton()
            assert np.array_equal(box, orc.bbox_squared(p))
            assert np.array_equal(codes, codes_o), passes
            assert np.array_equal(order, order_o), passes


@pytest.mark.parametrize("n", SIZES + [40960, 40961, 200_003, 262_144])
@pytest.mark.parametrize("kind", ["spread", "clustered"])
def test_static_sort(nbp, orc, n, kind):
    torch = pytest.importorskip("torch")
    p = bodies(n, kind)
    pos = torch.from_numpy(p).cuda()
    codes = torch.empty(n + 1, dtype=torch.int64, device="cuda")
    order = torch.empty(n + 1, dtype=torch.int32, device="cuda")
    box = torch.empty(4, dtype=torch.float64, device="cuda")
    codes_o, order_o = orc.stable_sort(orc.morton(p))
    for off in (0, 1):  # outputs at any element offset
        rc = nbp.load().nb_morton_sort_static(
            pos.data_ptr(), n, codes[off:].data_ptr(), order[off:].data_ptr(), box.data_ptr(),
            torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        torch.cuda.synchronize()
        assert np.array_equal(box.cpu().numpy(), orc.bbox_squared(p))
        assert np.array_equal(codes[off:off + n].cpu().numpy().view(np.uint64), codes_o)
        assert np.array_equal(order[off:off + n].cpu().numpy(), order_o)
