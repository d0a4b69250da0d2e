"""Sweeps whose colour passes run in one launch in dataflow order (hmc_flow.cuh).

Trajectories against the oracle's ParallelSweep at the sizes where the scheme's parts can go wrong:
two, four and six spaces per axis (images of the same space, the straddling first space, the
interior form), stencils of one candidate less, equal and more than a staging buffer and of two of
them, more teams than trials, every team size, and one colour set per launch (the form that runs
where the draw buffers do not fit).
"""
import numpy as np
import pytest

import oracle
from hoomd_rs_b200 import (FP32_RECHECK, FP64, ROTATE, TRANSLATE, Context, ConvexPolyhedron, HardShape, HardSphere,
                           Isotropic, LennardJones, Microstate, PairwiseCutoff, Periodic, Shifted, lattice)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return Context(0)


def lj(ctx, dim, n, rho, r_cut, seed=0x5EED0071):
    pos, L = lattice.lennard_jones_box(n, rho, dim, seed, jitter=0.02)
    h = PairwiseCutoff(Isotropic(Shifted(LennardJones(1.0, 1.0), r_cut), r_cut))
    g = Microstate(ctx, Periodic(r_cut, [L] * dim), pos, h, seed=seed)
    o = oracle.System(dim, [L] * dim, pos, seed=seed, interaction=oracle.LENNARD_JONES, lj_epsilon=1.0, lj_sigma=1.0,
                      lj_r_cut=r_cut, lj_r_shift=r_cut)
    return g, o


SIZES = [(3, 383, 1.1, 3.5), (3, 384, 1.1, 3.5), (3, 385, 1.1, 3.5), (3, 770, 1.1, 4.4), (3, 1500, 1.1, 2.7),
         (3, 4001, 1.1, 2.5), (2, 301, 0.7, 2.5), (2, 77, 0.6, 5.0)]


def check(g, o, precision, r_cut, sweeps=2, one_call=False):
    want = np.zeros(2, dtype=np.int64)
    for _ in range(sweeps):
        want += o.parallel_sweep(oracle.TRANSLATE, 0.12, 1.3, r_cut)
        o.increment_step()
    if one_call:
        c = g.sweep(TRANSLATE, 0.12, 1.3, precision, n_sweeps=sweeps, increment_step=True)
        got = np.array([c.accepted, c.rejected])
    else:
        cs = [g.sweep(TRANSLATE, 0.12, 1.3, precision, n_sweeps=1, increment_step=True) for _ in range(sweeps)]
        got = np.array([sum(c.accepted for c in cs), sum(c.rejected for c in cs)])
    assert np.array_equal(got, want)
    assert np.array_equal(g.positions(), o.state()[0])


@pytest.mark.parametrize("precision", [FP64, FP32_RECHECK])
@pytest.mark.parametrize("dim,n,rho,r_cut", SIZES)
def test_lj_sizes(ctx, dim, n, rho, r_cut, precision):
    for variant in range(5):
        g, o = lj(ctx, dim, n, rho, r_cut)
        g.set_launch_variant(precision, variant)
        check(g, o, precision, r_cut)
        g.close()


@pytest.mark.parametrize("one_call", [False, True])
@pytest.mark.parametrize("precision", [FP64, FP32_RECHECK])
def test_lj_one_colour_set_per_launch(ctx, precision, one_call, monkeypatch):
    monkeypatch.setenv("HMC_B200_FLOW_SETS", "1")
    g, o = lj(ctx, 3, 1500, 1.1, 2.7)
    check(g, o, precision, 2.7, sweeps=3, one_call=one_call)


BOX = np.array([[x, y, z] for x in (-1.0, 1.0) for y in (-1.0, 1.0) for z in (-1.0, 1.0)])
TETRAHEDRON = np.array([[1.0, 1.0, 1.0], [1.0, -1.0, -1.0], [-1.0, 1.0, -1.0], [-1.0, -1.0, 1.0]]) * 0.5
ROUND = np.random.default_rng(11).normal(size=(32, 3))
ROUND *= 0.55 / np.linalg.norm(ROUND, axis=1)[:, None]
# shape, sites per axis, spacing per axis: units of one to sixteen trials with remainders, two spaces
# per axis, 4 and 32 vertices, and thin rods, whose circumspheres hold more pairs than a warp's list
# and whose rows hold more candidates than one pass over a stencil takes
SHAPES = {"cubes_two_spaces": (BOX * 0.5, (3, 3, 3), (1.25, 1.25, 1.25)),
          "cubes": (BOX * 0.5, (9, 8, 7), (1.2, 1.25, 1.3)),
          "tetrahedra": (TETRAHEDRON, (7, 7, 7), (1.25, 1.25, 1.25)),
          "round_32": (ROUND, (8, 7, 6), (1.2, 1.2, 1.2)),
          "rods": (BOX * [0.1, 0.1, 1.0], (18, 18, 4), (0.5, 0.5, 2.2))}


@pytest.mark.parametrize("precision", [FP64, FP32_RECHECK])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_polyhedra(ctx, name, precision):
    verts, sites, spacing = SHAPES[name]
    L = [n * a for n, a in zip(sites, spacing)]
    rng = np.random.default_rng(5)
    pos = (np.stack(np.meshgrid(*[np.arange(n) for n in sites], indexing="ij"), -1).reshape(-1, 3) + 0.5) * spacing
    pos = pos - np.array(L) / 2 + rng.uniform(-0.01, 0.01, pos.shape)
    reach = 2.0 * float(np.sqrt((verts ** 2).sum(axis=1).max()))
    h = PairwiseCutoff(HardShape(ConvexPolyhedron.with_vertices(verts)))
    o = oracle.System(3, L, pos, seed=77, interaction=oracle.HARD_CONVEX_POLYHEDRON, vertices=verts)
    gs = [Microstate(ctx, Periodic(reach, L), pos, h, seed=77) for _ in range(2)]
    for v, g in enumerate(gs):
        g.set_launch_variant(precision, v)
    for sweep in range(6):
        move, maximum = ((TRANSLATE, 0.1), (ROTATE, 0.15))[sweep % 2]
        want = o.parallel_sweep(oracle.TRANSLATE if move == TRANSLATE else oracle.ROTATE, maximum, 1.0, reach)
        o.increment_step()
        for g in gs:
            c = g.sweep(move, maximum, 1.0, precision, n_sweeps=1, increment_step=True)
            assert (c.accepted, c.rejected) == tuple(want), sweep
    for g in gs:
        assert np.array_equal(g.positions(), o.state()[0])
        assert np.array_equal(g.orientations(), o.state()[1])


def test_polyhedra_one_colour_set_per_launch(ctx, monkeypatch):
    monkeypatch.setenv("HMC_B200_FLOW_SETS", "1")
    test_polyhedra(ctx, "cubes", FP32_RECHECK)


@pytest.mark.parametrize("scales", [(1.6,), (0.9, 1.4)])
def test_box_grows_between_sweeps(ctx, scales):
    """Estimators rebuild the cell list of the grown box before the next sweep does."""
    g, o = lj(ctx, 3, 1500, 0.6, 2.5)
    check(g, o, FP32_RECHECK, 2.5, sweeps=1)
    L = g.edge_lengths[0]
    for scale in scales:
        L *= scale
        g.set_box([L] * 3)
        assert np.isfinite(g.total_energy())
    fresh = Microstate(ctx, Periodic(2.5, [L] * 3), g.positions(),
                       PairwiseCutoff(Isotropic(Shifted(LennardJones(1.0, 1.0), 2.5), 2.5)), seed=0x5EED0071, step=1)
    assert fresh.total_energy() == pytest.approx(g.total_energy(), rel=1e-12)
    for s in (g, fresh):
        s.sweep(TRANSLATE, 0.12, 1.3, FP32_RECHECK, n_sweeps=2, increment_step=True)
    assert np.array_equal(g.positions(), fresh.positions())

# spaces per axis (of width 1.02 .. 1.3), sites per axis: two spaces on an axis (images of one space),
# units of one to three trials, spaces with one and several bodies, empty spaces
SPHERES = [(3, (2, 2, 2), (2, 2, 2)), (3, (2, 4, 6), (2, 4, 6)), (3, (4, 4, 4), (2, 2, 2)), (3, (6, 6, 6), (6, 6, 6)),
           (3, (8, 10, 12), (7, 9, 10)), (2, (2, 2), (2, 2)), (2, (2, 6), (2, 6)), (2, (12, 14), (12, 13))]


def spheres(ctx, dim, spaces, sites, seed=0x5EED0081):
    L = [1.02 * n + 0.05 for n in spaces]
    rng = np.random.default_rng(3)
    grid = np.stack(np.meshgrid(*[np.arange(n) for n in sites], indexing="ij"), -1).reshape(-1, dim)
    pos = (grid + 0.5) * np.array(L) / np.array(sites) - np.array(L) / 2 + rng.uniform(-0.005, 0.005, grid.shape)
    g = Microstate(ctx, Periodic(1.0, L), pos, PairwiseCutoff(HardSphere(1.0)), seed=seed)
    return g, oracle.System(dim, L, pos, diameter=1.0, seed=seed)


def check_spheres(g, o, precision, one_call=False, sweeps=4):
    want = np.zeros(2, dtype=np.int64)
    for _ in range(sweeps):
        want += o.parallel_sweep(oracle.TRANSLATE, 0.2, 1.0, 1.0)
        o.increment_step()
    if one_call:
        c = g.sweep(TRANSLATE, 0.2, 1.0, precision, n_sweeps=sweeps, increment_step=True)
        got = (c.accepted, c.rejected)
    else:
        cs = [g.sweep(TRANSLATE, 0.2, 1.0, precision, n_sweeps=1, increment_step=True) for _ in range(sweeps)]
        got = (sum(c.accepted for c in cs), sum(c.rejected for c in cs))
    assert got == tuple(want)
    assert np.array_equal(g.positions(), o.state()[0])


@pytest.mark.parametrize("precision", [FP64, FP32_RECHECK])
@pytest.mark.parametrize("dim,spaces,sites", SPHERES)
def test_spheres(ctx, dim, spaces, sites, precision):
    for variant in range(2):
        g, o = spheres(ctx, dim, spaces, sites)
        assert g.launch_variant(precision)["trials_per_warp"] == 3  # the dataflow family
        g.set_launch_variant(precision, variant)
        check_spheres(g, o, precision)
        g.close()


@pytest.mark.parametrize("one_call", [False, True])
@pytest.mark.parametrize("precision", [FP64, FP32_RECHECK])
def test_spheres_one_colour_set_per_launch(ctx, precision, one_call, monkeypatch):
    monkeypatch.setenv("HMC_B200_FLOW_SETS", "1")
    g, o = spheres(ctx, 3, (8, 10, 12), (7, 9, 10))
    check_spheres(g, o, precision, one_call)


@pytest.mark.parametrize("precision,n", [(FP64, 262144), (FP32_RECHECK, 114688)])
def test_spheres_beside_the_line(ctx, precision, n):
    """The largest box in dataflow order and the smallest in colour passes, each against the other form."""
    for bodies in (n + 7, n + 8):
        pos, L = lattice.hard_sphere_box(bodies, 0.45, 3, 5)
        runs = []
        for forced in (False, True):
            g = Microstate(ctx, Periodic(1.0, [L] * 3), pos, PairwiseCutoff(HardSphere(1.0)), seed=9)
            if forced:
                g.set_cooperative_pass(precision, False)
            flow = g.launch_variant(precision)["trials_per_warp"] == 3
            assert flow == (not forced and bodies == n + 7)
            c = g.sweep(TRANSLATE, 0.15, 1.0, precision, n_sweeps=2, increment_step=True)
            runs.append((c.accepted, c.rejected, g.positions()))
            g.close()
        assert runs[0][:2] == runs[1][:2]
        assert np.array_equal(runs[0][2], runs[1][2])
