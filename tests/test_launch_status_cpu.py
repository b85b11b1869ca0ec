"""Failed launches are reported: the library's host side on a fake CUDA runtime
(fake_cudart.c) that runs no kernel and fails the calls it is told to."""
import ctypes as C
import importlib
import pathlib
import subprocess

import numpy as np
import pytest

HERE = pathlib.Path(__file__).resolve().parent
LAUNCH, ATTRIBUTE, CLUSTERS, HOST_ALLOC, SYNC = range(5)
NB_ERR_CUDA = 2


@pytest.fixture(scope="module")
def fake(nbp, tmp_path_factory):
    """libnbody_b200's own objects, linked with the fake runtime."""
    build = importlib.import_module(nbp.__name__ + ".build")
    build.build()
    objects = sorted(build.OBJ / (s.stem + ".o") for s in build.CSRC.glob("*.cu"))
    so = tmp_path_factory.mktemp("fake") / "libnbody_fake.so"
    cuda = pathlib.Path(build.nvcc()).resolve().parents[1]
    fake_o = so.with_suffix(".o")
    subprocess.run(["gcc", "-c", "-O1", "-fPIC", "-fvisibility=hidden", "-I", str(cuda / "include"),
                    str(HERE / "fake_cudart.c"), "-o", str(fake_o)], check=True)
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-Wl,--no-undefined", "-o", str(so),
                    *map(str, objects), str(fake_o)], check=True)
    lib = C.CDLL(str(so))
    lib.nb_last_error.restype = C.c_char_p
    lib.nb_last_error.argtypes = [C.c_void_p]
    lib.fake_calls.restype = C.c_long
    lib.fake_fail.argtypes = [C.c_int, C.c_long]
    lib.fake_launched.restype = C.c_void_p
    return lib


# (mode, flags, bodies, universes): one context per chain of kernels
KINDS = {
    "fp64 cluster": (0, 0, 1000, 0), "fp64 onesweep": (0, 0, 40000, 0),
    "fp64 wide": (0, 0, 400000, 0),
    "split cluster": (1, 0, 1000, 0), "split onesweep": (1, 0, 140000, 0),
    "split scanned tiles": (1, 0, 600000, 0),
    "quad": (1, 1, 1000, 0), "learned": (1, 2, 1000, 0), "learned quad": (1, 3, 40000, 0),
    "batch cluster": (1, 0, 1000, 4), "batch onesweep": (1, 0, 40000, 4),
    "allpairs": (2, 0, 1000, 0), "allpairs cpu law": (2, 4, 1000, 0),
}


class Context:
    def __init__(self, nbp, lib, kind, fail=None):
        mode, flags, n, universes = KINDS[kind]
        p = nbp.NbParams()
        lib.nb_params_default(C.byref(p))
        p.mode, p.flags = mode, flags
        self.lib, self.h, self.n = lib, C.c_void_p(), n
        m, x = np.ones(n), np.zeros((n, 2))
        lib.fake_reset()
        lib.fake_forget_probes()
        if fail:
            lib.fake_fail(*fail)
        args = (m.ctypes.data_as(C.c_void_p), x.ctypes.data_as(C.c_void_p),
                x.ctypes.data_as(C.c_void_p), C.byref(self.h))
        if universes:
            counts = (C.c_uint64 * universes)(*[n // universes] * universes)
            rc = lib.nb_batch_create(C.byref(p), universes, counts, *args)
        else:
            rc = lib.nb_create(C.byref(p), C.c_uint64(n), *args)
        assert rc == 0
        self.host_allocs = lib.fake_calls(HOST_ALLOC)
        if flags & 2:
            w = np.zeros(5123, np.float32)
            assert lib.nb_set_mlp_weights(self.h, w.ctypes.data_as(C.c_void_p)) == 0
        assert lib.fake_last_error() == 0  # nothing left for the next call to trip over
        lib.fake_reset()

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        assert self.lib.nb_destroy(self.h) == 0

    def step(self, n=1):
        return self.lib.nb_step(self.h, n)


@pytest.mark.parametrize("kind", KINDS)
def test_a_failed_launch_fails_the_step(nbp, fake, kind):
    with Context(nbp, fake, kind) as ctx:
        assert ctx.step() == 0
        calls = [fake.fake_calls(LAUNCH), fake.fake_calls(ATTRIBUTE)]
    assert calls[0] >= 6
    for what in (LAUNCH, ATTRIBUTE):
        for k in range(calls[what]):
            with Context(nbp, fake, kind) as ctx:
                fake.fake_fail(what, k)
                launched = fake.fake_graph_launches()
                assert ctx.step() == NB_ERR_CUDA, (what, k)
                assert fake.fake_graph_launches() == launched  # nothing ran
                assert b"launch" in fake.nb_last_error(ctx.h)
                assert fake.fake_open_captures() == 0 and fake.fake_live_graphs() == 0
                assert fake.fake_last_error() == 0
                # the next step captures what is missing and runs
                assert ctx.step(3) == 0
                assert fake.fake_graph_launches() == launched + 3


@pytest.mark.parametrize("kind", [k for k in KINDS if KINDS[k][2] <= 32768 and KINDS[k][0] < 2])
def test_without_clusters_the_sort_takes_passes(nbp, fake, kind):
    """A device that cannot run the cluster sort (or an error while asking)."""
    with Context(nbp, fake, kind) as ctx:
        assert ctx.step() == 0
        clustered = fake.fake_calls(LAUNCH)
    for what, k in ((CLUSTERS, 0), (ATTRIBUTE, 0), (ATTRIBUTE, 1)):
        with Context(nbp, fake, kind, fail=(what, k)) as ctx:
            assert ctx.step() == 0
            assert fake.fake_calls(LAUNCH) > clustered


@pytest.mark.parametrize("n", [1025, 16384, 16385, 32768])
@pytest.mark.parametrize("universes", [0, 4])
def test_the_cluster_kernel_that_runs_was_asked_for(nbp, fake, n, universes):
    KINDS["probe"] = (1, 0, n - n % max(1, universes), universes)
    with Context(nbp, fake, "probe") as ctx:
        assert ctx.step() == 0
        assert fake.fake_unprobed_clusters() == 0
    del KINDS["probe"]


@pytest.mark.parametrize("n", [1000, 32768, 32769, 262144])
def test_static_sort_asks_once_where_a_cluster_can_sort(fake, n):
    buf = (C.c_double * (2 * n))()
    out, order = (C.c_uint64 * n)(), (C.c_int32 * n)()
    fake.fake_reset()
    assert fake.nb_morton_sort_static(buf, C.c_uint64(n), out, order, None, None) == 0
    assert fake.fake_calls(CLUSTERS) == (n <= 32768)
    assert fake.fake_calls(ATTRIBUTE) == (2 if n <= 32768 else 0)
    if n <= 32768:  # cannot: the counting passes, and no error left
        for what in (CLUSTERS, ATTRIBUTE):
            fake.fake_reset()
            fake.fake_fail(what, 0)
            assert fake.nb_morton_sort_static(buf, C.c_uint64(n), out, order, None, None) == 0
            assert fake.fake_calls(LAUNCH) == 18 and fake.fake_last_error() == 0
    fake.fake_reset()
    fake.fake_fail(LAUNCH, 0)
    assert fake.nb_morton_sort_static(buf, C.c_uint64(n), out, order, None, None) == NB_ERR_CUDA


@pytest.mark.parametrize("kind", ["fp64 cluster", "split onesweep", "allpairs"])
def test_a_context_pins_no_memory_and_a_download_waits_once(nbp, fake, kind):
    """Pinned memory costs a context some 4 ms to get and to give back."""
    with Context(nbp, fake, kind) as ctx:
        assert ctx.host_allocs == 0
        assert ctx.step() == 0
        out = np.empty((ctx.n, 2))
        fake.fake_reset()
        assert fake.nb_download(ctx.h, out.ctypes.data_as(C.c_void_p), None) == 0
        assert fake.fake_calls(SYNC) == 1
        fake.fake_fail(SYNC, 1)  # what a failed kernel looks like to the host
        assert fake.nb_download(ctx.h, out.ctypes.data_as(C.c_void_p), None) == NB_ERR_CUDA


def launches_on(nbp, fake, sms, mode, n):
    """(kernel, blocks, threads) of a step's launches on a device of so many SMs."""
    KINDS["sms"] = (mode, 0, n, 0)
    fake.fake_set_sms(sms)
    try:
        with Context(nbp, fake, "sms") as ctx:
            assert ctx.step() == 0
            per_step = fake.fake_calls(LAUNCH) // 2  # both parities were captured
            return [(fake.fake_launched(k), fake.fake_grid(k), fake.fake_block(k))
                    for k in range(per_step)]
    finally:
        fake.fake_set_sms(148)
        del KINDS["sms"]


@pytest.mark.parametrize("mode,n", [(0, 9000), (0, 40000), (0, 100000), (0, 250000), (1, 20000),
                                    (1, 250000)])
def test_rules_follow_the_sms(nbp, fake, mode, n):
    """Half the SMs take n bodies as all of them take 2 n: the same walk, bodies
    per warp, and threads per tile of the tree (where the rules end differs)."""
    def rules(sms, n):
        launches = launches_on(nbp, fake, sms, mode, n)
        walk = max(k for k, (_, _, threads) in enumerate(launches) if threads == 128)
        tiles = -(-n // 2048)
        return launches[walk][0], any(launch[1:] == (tiles, 1024) for launch in launches[2:])
    assert rules(74, n) == rules(148, 2 * n)
    assert rules(74, n) != rules(148, n)
