"""The work that a user of this framework has it do, as measurable cases.

Each case goes through the public entry points (``NbContext`` and the functions
beside it in ``simulation.py``, or the C ABI where it takes device pointers).

* ``step``: the simulation loop of ``BarnesHutB200``: ``steps`` steps, then the
  bodies back on the host (``download_every`` = steps).  The bodies stay on the
  GPU from pass to pass, so a pass continues the last one's universe.
* ``pair_acc``: ``allpairs_accelerations``, the exact forces that every
  accuracy figure of a run is stated against.
* ``sort``: ``nb_morton_sort_static``, the per-frame sort of a renderer that
  owns its device memory.

The universes are the repository's own generators; sizes lie between a toy
universe of a thousand bodies and the four-million-body benchmark.
"""
from __future__ import annotations

import importlib.util
import math
import pathlib
import sys

import numpy as np
import torch

_ROOT = pathlib.Path(__file__).resolve().parents[1]


def _package():
    """The package's folder is not an importable name: loaded as the tests do."""
    if "nbody_b200" in sys.modules:
        return sys.modules["nbody_b200"]
    pkg = _ROOT / "n-body-2d_b200"
    spec = importlib.util.spec_from_file_location(
        "nbody_b200", pkg / "__init__.py", submodule_search_locations=[str(pkg)])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["nbody_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


nb = _package()

EPS2 = 1e-4  # softening 0.01, as in every benchmark configuration
DT = 1e-4
# the ensemble's heaviest centres (a thousand disc masses) turn bodies at the
# softening length around in 2e-4: its steps resolve that orbit
DT_ENSEMBLE = 1e-6
BMAX_LEARNED = 0.75  # the guard the shipped weights were trained with


def _step(name, mode, universe, n, steps, theta=0.5):
    case = {"kind": "step", "mode": mode, "universe": universe, "n": n, "steps": steps,
            "theta": theta}
    return dict(case, name=name) if name else case


def listed():
    return [
        # the default mode on a toy universe, shown frame by frame: nothing but
        # launches, latency and the copy back
        _step("fp64_disc_1001", "fp64", "disc", 1001, 1),
        # the default mode on the benchmark's small disc, copied back every fourth step
        _step("fp64_disc_16k", "fp64", "disc", 16384, 4),
        # the default (parity) mode at the size a study of a galaxy pair takes
        _step("fp64_collision_1m", "fp64", "collision", 1 << 20, 2),
        # the fast mode on a small universe, shown frame by frame
        _step("split_plummer_16k", "split", "plummer", 16384, 1),
        # the fast mode at an ordinary, odd size, copied back every fourth step
        _step("split_plummer_300k", "split", "plummer", 300007, 4),
        # the benchmark's galaxy collision
        _step("split_collision_4m", "split", "collision", 1 << 22, 4),
        # the walk that meets a p99 force error of 1e-3: quadrupoles, theta 0.4
        _step("quad_collision_1m", "quad", "collision", 1 << 20, 4, 0.4),
        # the learned far field with the shipped weights
        _step("learned_collision_1m", "learned", "collision", 1 << 20, 4, 1.0),
        # an ensemble of independent universes in one context (1,024 to 262,144
        # bodies each)
        _step("batch_64_universes", "batch", "ensemble", 64, 4),
        # the all-pairs backend on the universe sizes it is for
        _step("allpairs_plummer_20k", "allpairs", "plummer", 20011, 1),
        # exact forces of as many bodies as an accuracy figure samples
        {"name": "pair_acc_64k_of_1m", "kind": "pair_acc", "universe": "collision", "n": 1 << 20,
         "targets": 65536},
        # a renderer's per-frame sort
        {"name": "sort_static_200k", "kind": "sort", "universe": "plummer", "n": 200003},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fp64", "fp64", "split", "split", "split", "quad", "learned", "batch",
                       "allpairs", "pair_acc", "sort"])
    steps = rng.choice([1, 2, 4])
    if kind == "fp64":
        n = _log_int(rng, 1000, 1 << 20)
        universe = rng.choice(["disc", "plummer", "collision"])
        n += n % 2 if universe == "collision" else 0
        return _step(None, "fp64", universe, n, min(steps, 2), rng.choice([0.5, 0.7, 1.0]))
    if kind in ("split", "quad"):
        n = _log_int(rng, 1000, (1 << 22) if kind == "split" else (1 << 20))
        # a collision's centres outweigh everything else in small universes
        universe = "collision" if n >= (1 << 18) and rng.random() < 0.5 else "plummer"
        n -= n % 2 if universe == "collision" else 0
        return _step(None, kind, universe, n, steps,
                     rng.choice([0.5, 0.7] if kind == "split" else [0.4, 0.5, 0.7]))
    if kind == "learned":
        n = 2 * _log_int(rng, 1 << 17, 1 << 19)
        return _step(None, "learned", "collision", n, steps, 1.0)
    if kind == "batch":
        return _step(None, "batch", "ensemble", rng.randint(3, 64), steps)
    if kind == "allpairs":
        return _step(None, rng.choice(["allpairs", "allpairs_cpu_law"]), "plummer",
                     _log_int(rng, 1000, 40000), 1)
    if kind == "pair_acc":
        n = _log_int(rng, 1 << 14, 1 << 20)
        return {"kind": "pair_acc", "universe": "plummer", "n": n,
                "targets": min(n, _log_int(rng, 64, 65536))}
    return {"kind": "sort", "universe": rng.choice(["disc", "plummer"]),
            "n": _log_int(rng, 1000, nb.NB_STATIC_SORT_MAX_BODIES)}


def _universe(case, seed):
    """(mass, pos, vel, universe sizes or None)"""
    u, n, seed = case["universe"], case["n"], seed % (1 << 31)
    if u == "ensemble":
        # sizes, scale lengths and central masses are the ensemble's own, the bodies the seed's
        rng = np.random.default_rng([n, 1])
        sizes = nb.universes.ensemble_sizes(n, n)
        scales, ratios = rng.uniform(0.5, 2.0, n), np.exp(rng.uniform(*np.log([1e3, 1e6]), n))
        discs = [nb.universes.exponential_disc(int(sizes[k]), seed * n + k, scale=scales[k],
                                               central_ratio=ratios[k]) for k in range(n)]
        return (*(np.concatenate(x) for x in zip(*discs)), sizes)
    return (*nb.universes.make(u, n, seed), None)


def _timestep(case):
    return DT_ENSEMBLE if case["universe"] == "ensemble" else DT


def _pinned(n):
    return torch.empty((n, 2), dtype=torch.float64, pin_memory=True).numpy()


def prepare(case, seed):
    if case["kind"] == "step":
        m, p, v, counts = _universe(case, seed)
        mode = case["mode"]
        cfg = nb.SimConfig(
            timestep=_timestep(case), theta=case["theta"], epsilon_squared=EPS2,
            mode=(nb.NB_MODE_FP64 if mode == "fp64" else
                  nb.NB_MODE_ALLPAIRS if mode.startswith("allpairs") else nb.NB_MODE_SPLIT),
            quadrupole=mode == "quad", learned=mode == "learned",
            bmax_ratio=BMAX_LEARNED if mode == "learned" else 0.0,
            cpu_law=mode == "allpairs_cpu_law")
        ctx = nb.NbContext(cfg, m, p, v, counts=counts)
        if mode == "learned":
            ctx.set_mlp_weights(np.load(_ROOT / "n-body-2d_b200" / "weights"
                                        / "correction_theta1.npy"))
        return {"kind": "step", "ctx": ctx, "steps": case["steps"], "pos": _pinned(ctx.n),
                "vel": _pinned(ctx.n)}
    if case["kind"] == "pair_acc":
        m, p, _, _ = _universe(case, seed)
        return {"kind": "pair_acc", "mass": m, "pos": p, "targets": _targets(case, seed)}
    _, p, _, _ = _universe(case, seed)
    n = case["n"]
    return {"kind": "sort", "lib": nb.load(), "n": n, "pos": torch.from_numpy(p).cuda(),
            "codes": torch.empty(n, dtype=torch.int64, device="cuda"),
            "order": torch.empty(n, dtype=torch.int32, device="cuda"),
            "box": torch.empty(4, dtype=torch.float64, device="cuda")}


def _targets(case, seed):
    rng = np.random.default_rng([seed % (1 << 31), 7])
    return np.sort(rng.choice(case["n"], size=case["targets"], replace=False))


def run(state):
    kind = state["kind"]
    if kind == "step":
        state["ctx"].step(state["steps"], sync=False)
        return state["ctx"].download(state["pos"], state["vel"])
    if kind == "pair_acc":
        return nb.allpairs_accelerations(state["mass"], state["pos"], state["targets"], EPS2)
    rc = state["lib"].nb_morton_sort_static(
        state["pos"].data_ptr(), state["n"], state["codes"].data_ptr(),
        state["order"].data_ptr(), state["box"].data_ptr(),
        torch.cuda.current_stream().cuda_stream)
    if rc != nb._lib.NB_OK:
        raise RuntimeError(f"nb_morton_sort_static: status {rc}")
    return state["codes"], state["order"], state["box"]


def _bodies(case):
    if case.get("universe") != "ensemble":
        return case["n"]
    # sizes are log-uniform in [1024, 262144]
    return int(case["n"] * (262144 - 1024) / math.log(256))


def work(case):
    """Bytes: inputs and outputs once.  Flops: the interactions (14 flops each,
    34 with quadrupoles) that the opening angle asks for, about
    8 log2(n) / theta^2 per body (700 at four million bodies and 0.5)."""
    n = _bodies(case)
    if case["kind"] == "step":
        per_universe = n / case["n"] if case["universe"] == "ensemble" else n
        if case["mode"].startswith("allpairs"):
            terms = float(n)
        else:
            terms = min(n, 8.0 * math.log2(per_universe) / case["theta"] ** 2)
        flops = (34 if case["mode"] == "quad" else 14) * terms * n * case["steps"]
        return {"bytes": 72.0 * n, "flops": flops}
    if case["kind"] == "pair_acc":
        return {"bytes": 24.0 * n + 24.0 * case["targets"], "flops": 14.0 * n * case["targets"]}
    return {"bytes": 28.0 * n, "flops": 0.0}


def _pair_sum(pos, mass, targets, law):
    """Exact accelerations of targets[k, 2], in 64 bits, by blocks of targets."""
    x, y = pos[:, 0].contiguous(), pos[:, 1].contiguous()
    out = torch.empty_like(targets)
    block = max(1, (1 << 26) // x.shape[0])
    for a in range(0, targets.shape[0], block):
        t = targets[a:a + block]
        dx, dy = x[None, :] - t[:, 0:1], y[None, :] - t[:, 1:2]
        r2 = dx * dx + dy * dy
        if law == "cpu":
            w = mass / (r2.sqrt() * (r2 + EPS2))
            w[r2 == 0.0] = 0.0
        else:
            w = mass * (r2 + EPS2).pow(-1.5)
        out[a:a + block, 0] = (w * dx).sum(1)
        out[a:a + block, 1] = (w * dy).sum(1)
    return out


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "pair_acc":
        m, p, _, _ = _universe(case, seed)
        pos = torch.from_numpy(p).to(device)
        at = torch.from_numpy(_targets(case, seed)).to(device)
        return _pair_sum(pos, torch.from_numpy(m).to(device), pos[at], "plummer").cpu().numpy()
    if case["kind"] != "step":  # codes and permutation are whole numbers
        return None
    if case["universe"] == "ensemble" or float(case["n"]) ** 2 * case["steps"] > 3e11:
        return None
    m, p, v, _ = _universe(case, seed)
    mass, pos, vel = (torch.from_numpy(a).to(device) for a in (m, p, v))
    dt = _timestep(case)
    pairs = case["mode"].startswith("allpairs")
    law = "cpu" if case["mode"] == "allpairs_cpu_law" else "plummer"
    for _ in range(case["steps"]):
        if pairs:  # AllPairs drifts before the kick
            pos = pos + vel * dt
        vel = vel + _pair_sum(pos, mass, pos, law) * dt
        if not pairs:
            pos = pos + vel * dt
    return pos.cpu().numpy(), vel.cpu().numpy()
