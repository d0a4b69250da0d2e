"""The work that a user of this framework has it do, as timed cases over its public entry points.

A case is a simulation's production loop between two frames: sweeps over a state that stays on the
GPU, then the frame (positions, and orientations of shapes) read back to the host, with the counts
of accepted and rejected trials. One kind measures the estimators that run between such loops.

Kinds: hard spheres and disks, convex polyhedra (cubes), convex polygons, Lennard-Jones sites,
batches of independent replicas of spheres or Lennard-Jones sites, and the estimators (total
energy, g(r)). States start from a jittered lattice and are relaxed for some sweeps, so the sweeps
that are timed meet liquid-like neighbourhoods; a program that is going to run long also has
`autotune` choose the launch variant once before it starts ("autotune").
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from hoomd_rs_b200 import (FP32_RECHECK, FP64, ROTATE, TRANSLATE, Batch, Context, ConvexPolygon, ConvexPolyhedron,
                           HardShape, HardSphere, Isothermal, Isotropic, LennardJones, Microstate, PairwiseCutoff,
                           ParallelSweep, Periodic, Rotate, Shifted, Translate)

CUBE = np.array([[x, y, z] for x in (-0.5, 0.5) for y in (-0.5, 0.5) for z in (-0.5, 0.5)])
SQUARE = np.array([[-0.5, -0.5], [0.5, -0.5], [0.5, 0.5], [-0.5, 0.5]])
JITTER = 0.01

_context = None


def context() -> Context:
    """One device context per process, as a user's program has it."""
    global _context
    if _context is None:
        _context = Context(0)
    return _context


# ---- the cases ---------------------------------------------------------------------------------
def listed():
    return [
        # The smallest call: one ParallelSweep::apply on a box of disks, as a program that looks at
        # its state after every sweep makes it. Launches, the host round trip and latency count.
        dict(name="disks_1024_one_call", kind="spheres", dim=2, n=1024, fill=0.70, move=0.1, precision="fp64",
             sweeps=1, one_call=False, autotune=False, relax=4),
        # The reference's small benchmark system, run for many sweeps in one call.
        dict(name="disks_4096_run", kind="spheres", dim=2, n=4096, fill=0.70, move=0.1, precision="fp64",
             sweeps=100, one_call=True, autotune=True, relax=20),
        # An ordinary box of spheres with a ragged body count, sweep by sweep (a frame every 20).
        dict(name="spheres_50021", kind="spheres", dim=3, n=50021, fill=0.45, move=0.13, precision="fp32",
             sweeps=20, one_call=False, autotune=False, relax=20),
        # The headline box in both precision modes, at the move size its tuner finds.
        dict(name="spheres_2p20_fp32", kind="spheres", dim=3, n=1 << 20, fill=0.50, move=0.234, precision="fp32",
             sweeps=20, one_call=False, autotune=True, relax=20),
        dict(name="spheres_2p20_fp64", kind="spheres", dim=3, n=1 << 20, fill=0.50, move=0.234, precision="fp64",
             sweeps=20, one_call=True, autotune=True, relax=20),
        # Hard cubes: a translation and a rotation sweep per step.
        dict(name="cubes_2p18", kind="cubes", n=1 << 18, fill=0.55, move=0.08, turn=0.1, precision="fp32", sweeps=10,
             autotune=True, relax=10),
        # Hard squares in 2-D, the same loop.
        dict(name="squares_2p18", kind="polygons", sides=4, n=1 << 18, fill=0.60, move=0.1, turn=0.1,
             precision="fp32", sweeps=10, autotune=True, relax=10),
        # The Lennard-Jones liquid, large in FP32 with recheck and small and ragged in FP64.
        dict(name="lj_2p19", kind="lj", dim=3, n=1 << 19, density=0.8, kt=1.0, r_cut=2.5, move=0.1, precision="fp32",
             sweeps=10, autotune=True, relax=10),
        dict(name="lj_20011_fp64", kind="lj", dim=3, n=20011, density=0.7, kt=1.3, r_cut=2.5, move=0.15,
             precision="fp64", sweeps=10, autotune=False, relax=10),
        # Many independent boxes of uneven sizes at once, captured sweeps, all sweeps in one call.
        dict(name="sphere_replicas_256", kind="sphere_replicas", replicas=256, n_min=1024, n_max=65536,
             fill_min=0.40, fill_max=0.54, move=0.15, spread=4, precision="fp32", sweeps=100, autotune=True, relax=10),
        dict(name="lj_replicas_64", kind="lj_replicas", replicas=64, n=8192, density=0.8, kt_min=0.8, kt_max=2.0,
             r_cut=2.5, move=0.1, spread=5, precision="fp32", sweeps=10, autotune=True, relax=4),
        # What runs between the loops: the total energy and the pair distribution of a liquid.
        dict(name="estimators_lj_2p17", kind="estimators", n=1 << 17, density=0.8, r_cut=2.5, r_max=3.0, bins=150),
    ]


def _log_size(rng: random.Random, low: int, high: int) -> int:
    """A size spread over its logarithm; mostly no round number."""
    n = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    return n | 1 if rng.random() < 0.6 else n


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["disks", "spheres", "spheres", "cubes", "polygons", "lj", "lj", "sphere_replicas",
                       "lj_replicas", "estimators"])
    precision = rng.choice(["fp32", "fp64"])
    tune = rng.random() < 0.5
    if kind == "disks":
        n = _log_size(rng, 512, 1 << 18)
        fill = min(round(rng.uniform(0.45, 0.70), 4), _most_fill(n, 2))
        return dict(kind="spheres", dim=2, n=n, fill=fill, move=round(rng.uniform(0.05, 0.25), 4), precision=precision,
                    sweeps=rng.randint(1, 40), one_call=rng.random() < 0.5, autotune=tune, relax=10)
    if kind == "spheres":
        n = _log_size(rng, 1024, 1 << 20)
        fill = min(round(rng.uniform(0.30, 0.54), 4), _most_fill(n, 3))
        return dict(kind="spheres", dim=3, n=n, fill=fill, move=round(rng.uniform(0.05, 0.25), 4), precision=precision,
                    sweeps=rng.randint(1, 20), one_call=rng.random() < 0.5, autotune=tune, relax=10)
    if kind == "cubes":
        n = _log_size(rng, 1000, 1 << 18)
        return dict(kind="cubes", n=n, fill=round(rng.uniform(0.30, 0.55), 4), move=round(rng.uniform(0.04, 0.15), 4),
                    turn=round(rng.uniform(0.05, 0.2), 4), precision=precision, sweeps=rng.randint(1, 6),
                    autotune=tune, relax=6)
    if kind == "polygons":
        n = _log_size(rng, 1000, 1 << 18)
        sides = rng.choice([3, 4, 5, 6, 8])
        # (triangles of one orientation on a square lattice touch above 0.30)
        return dict(kind="polygons", sides=sides, n=n, fill=round(rng.uniform(0.20, 0.30 if sides == 3 else 0.50), 4),
                    move=round(rng.uniform(0.05, 0.15), 4), turn=round(rng.uniform(0.05, 0.3), 4), precision=precision,
                    sweeps=rng.randint(1, 10), autotune=tune, relax=6)
    if kind == "lj":
        dim = rng.choice([3, 3, 2])
        n = _log_size(rng, 1000, 1 << 19)
        return dict(kind="lj", dim=dim, n=n, density=round(rng.uniform(0.3, 0.85) if dim == 3 else rng.uniform(0.3, 0.7), 4),
                    kt=round(rng.uniform(0.8, 2.0), 4), r_cut=2.5, move=round(rng.uniform(0.05, 0.25), 4),
                    precision=precision, sweeps=rng.randint(1, 10), autotune=tune, relax=4)
    if kind == "sphere_replicas":
        return dict(kind="sphere_replicas", replicas=rng.randint(8, 256), n_min=1024, n_max=_log_size(rng, 4096, 65536),
                    fill_min=0.40, fill_max=round(rng.uniform(0.45, 0.54), 4), move=round(rng.uniform(0.1, 0.2), 4),
                    spread=rng.randrange(1 << 20), precision=precision, sweeps=rng.randint(10, 40), autotune=tune, relax=6)
    if kind == "lj_replicas":
        return dict(kind="lj_replicas", replicas=rng.randint(8, 64), n=_log_size(rng, 1024, 8192), density=0.8,
                    kt_min=0.8, kt_max=2.0, r_cut=2.5, move=round(rng.uniform(0.08, 0.15), 4),
                    spread=rng.randrange(1 << 20), precision=precision, sweeps=rng.randint(2, 10), autotune=tune, relax=4)
    return dict(kind="estimators", n=_log_size(rng, 1 << 12, 1 << 17), density=round(rng.uniform(0.5, 0.85), 4),
                r_cut=2.5, r_max=round(rng.uniform(2.0, 3.5), 3), bins=rng.randint(60, 300))


# ---- states ------------------------------------------------------------------------------------
def _lattice(n: int, L: float, dim: int, fcc: bool, rng: np.random.Generator, jitter: float) -> np.ndarray:
    """The first n sites of a square, simple-cubic or FCC lattice in [-L/2, L/2)^dim, jittered."""
    if fcc:
        m = int(math.ceil((n / 4.0) ** (1.0 / 3.0) - 1e-9))
        basis = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
        cells = np.indices([m, m, m]).reshape(3, -1).T.astype(np.float64)
        sites = (cells[:, None, :] + basis[None, :, :]).reshape(-1, 3)[:n] + 0.25
    else:
        m = int(math.ceil(n ** (1.0 / dim) - 1e-9))
        sites = np.indices([m] * dim).reshape(dim, -1).T[:n].astype(np.float64) + 0.5
    pos = -L / 2.0 + sites * (L / m)
    return pos + rng.uniform(-jitter, jitter, pos.shape) if jitter > 0 else pos


def _box(n: int, density: float, dim: int) -> float:
    return (n / density) ** (1.0 / dim)


def _sphere_density(fill: float, dim: int) -> float:
    return fill / (math.pi / 4.0 if dim == 2 else math.pi / 6.0)


def _most_fill(n: int, dim: int) -> float:
    """The largest packing fraction (at most 0.70 and 0.54) at which the jittered lattice of n
    spheres has no overlap."""
    near = 1.0 + 2.0 * math.sqrt(dim) * JITTER + 1e-6
    m = int(math.ceil((n / 4.0) ** (1.0 / 3.0) - 1e-9)) if dim == 3 else int(math.ceil(math.sqrt(n) - 1e-9))
    L = near * m * (math.sqrt(2.0) if dim == 3 else 1.0)
    most = n * (math.pi / 6.0 if dim == 3 else math.pi / 4.0) / L ** dim
    return min(most, 0.54 if dim == 3 else 0.70)


def _precision(case) -> int:
    return FP32_RECHECK if case["precision"] == "fp32" else FP64


def _polygon(sides: int) -> np.ndarray:
    return SQUARE if sides == 4 else ConvexPolygon.regular(sides).vertices


def _area(v: np.ndarray) -> float:
    x, y = v[:, 0], v[:, 1]
    return 0.5 * abs(float(np.dot(x, np.roll(y, -1)) - np.dot(y, np.roll(x, -1))))


def _pinned(n: int, dim: int) -> np.ndarray:
    return torch.empty((n, dim), dtype=torch.float64, pin_memory=True).numpy()


def _replica_specs(case):
    """Body counts (log-uniform) and packing fractions of a batch's boxes."""
    rng = random.Random(case["spread"])
    out = []
    while len(out) < case["replicas"]:
        n = int(round(math.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"])))))
        fill = rng.uniform(case["fill_min"], case["fill_max"])
        if fill <= _most_fill(n, 3):
            out.append((n, fill))
    return out


def _lj(case) -> PairwiseCutoff:
    return PairwiseCutoff(Isotropic(Shifted(LennardJones(1.0, 1.0), case["r_cut"]), case["r_cut"]))


def prepare(case, seed):
    kind, rng, ctx = case["kind"], np.random.default_rng(seed), context()
    state = {"case": dict(case)}
    if kind in ("sphere_replicas", "lj_replicas"):
        replicas, kts = [], 1.0
        if kind == "sphere_replicas":
            for n, fill in _replica_specs(case):
                L = _box(n, _sphere_density(fill, 3), 3)
                replicas.append(dict(boundary=Periodic(1.0, [L] * 3), positions=_lattice(n, L, 3, True, rng, JITTER),
                                     seed=int(rng.integers(1 << 31))))
        else:
            h = _lj(case)
            n, L = case["n"], _box(case["n"], case["density"], 3)
            temperatures = random.Random(case["spread"])
            kts = np.array([temperatures.uniform(case["kt_min"], case["kt_max"]) for _ in range(case["replicas"])])
            for _ in range(case["replicas"]):
                replicas.append(dict(boundary=Periodic(case["r_cut"], [L] * 3), hamiltonian=h,
                                     positions=_lattice(n, L, 3, True, rng, JITTER), seed=int(rng.integers(1 << 31))))
        batch = Batch(ctx, replicas)
        maxima = np.full(len(replicas), case["move"])
        batch.set_captured_sweeps(True)
        batch.sweep(maxima, _precision(case), n_sweeps=case["relax"], increment_step=True, temperatures=kts)
        if case["autotune"]:
            batch.autotune(maxima, _precision(case), sweeps=2, temperatures=kts)
        total = sum(len(r["positions"]) for r in replicas)
        return dict(state, batch=batch, maxima=maxima, kts=kts, frame=np.empty((total, 3)))
    orientations = None
    if kind == "spheres":
        dim, n = case["dim"], case["n"]
        L = _box(n, _sphere_density(case["fill"], dim), dim)
        pos, h, reach = _lattice(n, L, dim, dim == 3, rng, JITTER), PairwiseCutoff(HardSphere(1.0)), 1.0
        moves = [Translate.with_maximum_distance(case["move"])]
    elif kind == "cubes":
        dim, n = 3, case["n"]
        L = _box(n, case["fill"], 3)
        pos, reach = _lattice(n, L, 3, False, rng, 0.0), math.sqrt(3.0)
        h = PairwiseCutoff(HardShape(ConvexPolyhedron.with_vertices(CUBE)))
        moves = [Translate.with_maximum_distance(case["move"]), Rotate.with_maximum_rotation(case["turn"])]
    elif kind == "polygons":
        dim, n, v = 2, case["n"], _polygon(case["sides"])
        L = _box(n, case["fill"] / _area(v), 2)
        shape = ConvexPolygon.with_vertices(v)
        pos, reach = _lattice(n, L, 2, False, rng, 0.0), 2.0 * shape.bounding_radius
        h, orientations = PairwiseCutoff(HardShape(shape)), np.zeros(n)
        moves = [Translate.with_maximum_distance(case["move"]), Rotate.with_maximum_rotation(case["turn"])]
    elif kind == "lj":
        dim, n = case["dim"], case["n"]
        L = _box(n, case["density"], dim)
        pos, h, reach = _lattice(n, L, dim, dim == 3, rng, JITTER), _lj(case), case["r_cut"]
        moves = [Translate.with_maximum_distance(case["move"])]
    else:
        # the estimators read a frame that is already there: a thermally disordered lattice
        dim, n = 3, case["n"]
        L = _box(n, case["density"], 3)
        pos, h, reach = _wrapped(_lattice(n, L, 3, True, rng, 0.12), L), _lj(case), case["r_cut"]
        return dict(state, microstate=Microstate(ctx, Periodic(reach, [L] * 3), pos, h, seed=seed & 0x7FFFFFFF))
    macro = Isothermal(case.get("kt", 1.0))
    m = Microstate(ctx, Periodic(reach, [L] * dim), pos, h, seed=seed & 0x7FFFFFFF, orientations=orientations)
    precision = _precision(case)
    for move in moves:
        code, size = _move(move)
        m.sweep(code, size, macro.temperature, precision, n_sweeps=case["relax"], increment_step=True)
    if case["autotune"]:
        code, size = _move(moves[0])
        m.autotune(code, size, macro.temperature, precision, sweeps=2)
    sweeps = [ParallelSweep(reach, move, precision) for move in moves]
    return dict(state, microstate=m, hamiltonian=h, macro=macro, sweeps=sweeps, frame=_pinned(n, dim))


def _move(local_trial):
    if isinstance(local_trial, Translate):
        return TRANSLATE, local_trial.maximum_distance
    return ROTATE, local_trial.maximum_rotation


def _wrapped(pos: np.ndarray, L: float) -> np.ndarray:
    x = pos / L
    return (x - np.floor(x + 0.5)) * L


# ---- one pass ----------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("sphere_replicas", "lj_replicas"):
        batch, frame, at = state["batch"], state["frame"], 0
        counts, _ = batch.sweep(state["maxima"], _precision(case), n_sweeps=case["sweeps"], increment_step=True,
                                temperatures=state["kts"])
        for k, n in enumerate(batch.sizes):
            frame[at:at + n] = batch.positions(k)
            at += n
        return {"counts": np.array([(c.accepted, c.rejected) for c in counts], dtype=np.int64), "frame": frame}
    m = state["microstate"]
    if kind == "estimators":
        return {"energy": m.total_energy(), "gr": m.gr_counts(case["r_max"], case["bins"]).astype(np.int64)}
    accepted = rejected = 0
    if kind in ("cubes", "polygons", "lj") or not case["one_call"]:
        for _ in range(case["sweeps"]):
            for sweep in state["sweeps"]:
                c = sweep.apply(m, state["hamiltonian"], state["macro"])
                accepted, rejected = accepted + c.accepted, rejected + c.rejected
            m.increment_step()
    else:
        code, size = _move(state["sweeps"][0].local_trial)
        c = m.sweep(code, size, state["macro"].temperature, _precision(case), n_sweeps=case["sweeps"],
                    increment_step=True)
        accepted, rejected = c.accepted, c.rejected
    m.state(state["frame"])
    out = {"accepted": accepted, "rejected": rejected, "positions": state["frame"]}
    if kind in ("cubes", "polygons"):
        out["orientations"] = m.orientations()
    return out


# ---- what a pass cannot do without --------------------------------------------------------------
def _trial_flops(case) -> float:
    """Arithmetic of one trial: its proposal, the distances to the bodies of its stencil (spaces one
    range wide) and the pair terms of those in range."""
    kind, proposal = case["kind"], 150.0
    if kind in ("spheres", "sphere_replicas"):
        dim = case.get("dim", 3)
        fill = case.get("fill") or 0.5 * (case["fill_min"] + case["fill_max"])
        return proposal + 3.0 ** dim * _sphere_density(fill, dim) * 3.0 * dim
    if kind == "cubes":
        rho, r = case["fill"], math.sqrt(3.0)
        return proposal + 27.0 * rho * r ** 3 * 9.0 + 4.19 * rho * r ** 3 * 300.0
    if kind == "polygons":
        v = _polygon(case["sides"])
        rho, r = case["fill"] / _area(v), 2.0 * float(np.sqrt((v ** 2).sum(axis=1).max()))
        return proposal + 9.0 * rho * r ** 2 * 6.0 + 3.14 * rho * r ** 2 * 100.0
    dim, rho, r = case.get("dim", 3), case["density"], case["r_cut"]
    ball = 4.19 * r ** 3 if dim == 3 else 3.14 * r ** 2
    return proposal + 2.0 * (3.0 ** dim * rho * r ** dim * 3.0 * dim + ball * rho * 12.0)


def work(case):
    kind = case["kind"]
    if kind == "estimators":
        n, rho = case["n"], case["density"]
        pairs = 0.5 * n * rho * 4.19
        return {"bytes": 2.0 * 24.0 * n + 8.0 * case["bins"] + 8.0,
                "flops": pairs * (case["r_cut"] ** 3 * 21.0 + case["r_max"] ** 3 * 11.0)}
    if kind == "sphere_replicas":
        n, sweeps = sum(n for n, _ in _replica_specs(case)), case["sweeps"]
    elif kind == "lj_replicas":
        n, sweeps = case["replicas"] * case["n"], case["sweeps"]
    else:
        n, sweeps = case["n"], case["sweeps"] * (2 if kind in ("cubes", "polygons") else 1)
    body = 8.0 * case.get("dim", 2 if kind == "polygons" else 3)
    turn = {"cubes": 32.0, "polygons": 8.0}.get(kind, 0.0)
    # the state read and written once, and the frame
    return {"bytes": n * (body + turn) * 3.0, "flops": n * sweeps * _trial_flops(case)}


# ---- values in 64 bits ----------------------------------------------------------------------------
def exact(case, seed):
    """The estimators' energy. A Markov chain's trajectory has no value apart from the chain (its
    decisions have to be the same), so the sweeps have none."""
    if case["kind"] != "estimators":
        return None
    rng = np.random.default_rng(seed)
    n, L, r_cut = case["n"], _box(case["n"], case["density"], 3), case["r_cut"]
    x = torch.from_numpy(_wrapped(_lattice(n, L, 3, True, rng, 0.12), L)).cuda()
    shift = 4.0 * ((1.0 / r_cut) ** 12 - (1.0 / r_cut) ** 6)
    total = torch.zeros((), dtype=torch.float64, device="cuda")
    for i in range(0, n, 1024):
        r2 = torch.zeros((min(1024, n - i), n), dtype=torch.float64, device="cuda")
        for a in range(3):
            d = x[i:i + 1024, a, None] - x[None, :, a]
            d -= L * torch.round(d / L)
            r2 += d * d
        r2 = r2[(r2 < r_cut * r_cut) & (r2 > 0.0)]
        s6 = (1.0 / r2) ** 3
        total += (4.0 * (s6 * s6 - s6) - shift).sum()
    return {"energy": 0.5 * float(total), "gr": None}
