"""nb_morton_sort_static takes device positions that nothing has checked.  An
axis without a finite value leaves the box at the reduction's seeds, +-DBL_MAX,
whichever way the call sorts (a cluster up to 32,768 bodies, counting passes
above): the same box, codes and order as from the host's arithmetic."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BIG = np.finfo(np.float64).max


def squared_box(p):
    x0, x1 = np.fmin.reduce(p[:, 0], initial=BIG), np.fmax.reduce(p[:, 0], initial=-BIG)
    y0, y1 = np.fmin.reduce(p[:, 1], initial=BIG), np.fmax.reduce(p[:, 1], initial=-BIG)
    xr, yr = x1 - x0, y1 - y0
    if xr > yr:
        mid = (y0 + y1) * 0.5
        y0, y1 = mid - xr * 0.5, mid + xr * 0.5
    else:
        mid = (x0 + x1) * 0.5
        x0, x1 = mid - yr * 0.5, mid + yr * 0.5
    return np.array([x0, x1, y0, y1])


def spread(v):
    x = v.astype(np.uint64)
    for s, k in ((16, 0x0000FFFF0000FFFF), (8, 0x00FF00FF00FF00FF), (4, 0x0F0F0F0F0F0F0F0F),
                 (2, 0x3333333333333333), (1, 0x5555555555555555)):
        x = (x | (x << np.uint64(s))) & np.uint64(k)
    return x


def codes_of(p, box):
    def grid(v, lo, hi):
        return np.fmin(np.fmax((v - lo) * (1.0 / (hi - lo)) * 4294967296.0, 0.0), 4294967295.0)
    ix, iy = (np.floor(grid(p[:, k], box[2 * k], box[2 * k + 1])).astype(np.uint32) for k in (0, 1))
    return (spread(ix) << np.uint64(1)) | spread(iy)


@pytest.mark.parametrize("n", [1, 1000, 20000, 32768, 32769, 100000])
@pytest.mark.parametrize("kind", ["finite", "x nan", "x inf", "x -inf", "y inf", "all nan", "some inf",
                                  "some nan"])
def test_box_and_codes(nbp, n, kind):
    torch = pytest.importorskip("torch")
    p = np.random.default_rng(n).normal(size=(n, 2))
    axis = {"x": [0], "y": [1], "a": [0, 1], "s": [0, 1], "f": []}[kind[0]]
    value = {"nan": np.nan, "inf": np.inf, "-inf": -np.inf, "finite": 0.0}[kind.split()[-1]]
    rows = slice(0, n, 3) if kind.startswith("some") else slice(None)
    for k in axis:
        p[rows, k] = value
    dpos = torch.from_numpy(p).cuda()
    codes = torch.empty(n, dtype=torch.int64, device="cuda")
    order = torch.empty(n, dtype=torch.int32, device="cuda")
    dbox = torch.empty(4, dtype=torch.float64, device="cuda")
    assert nbp.load().nb_morton_sort_static(dpos.data_ptr(), n, codes.data_ptr(), order.data_ptr(),
                                            dbox.data_ptr(),
                                            torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    with np.errstate(all="ignore"):
        box = squared_box(p)
        want = codes_of(p, box)
    assert np.array_equal(dbox.cpu().numpy(), box, equal_nan=True)
    perm = np.argsort(want, kind="stable")
    assert np.array_equal(order.cpu().numpy(), perm)
    assert np.array_equal(codes.cpu().numpy().view(np.uint64), want[perm])
