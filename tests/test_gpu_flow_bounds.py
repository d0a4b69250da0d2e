"""The polyhedron sweep with its FP32 bounds widened, so that its FP64 branches decide.

The first test of a pair (separated32) and the search for support vertices (pair_support) take FP32 values
that clear a bound; a bound 10^5 times as wide leaves nearly all of them to the FP64 forms behind them.
"""
import numpy as np
import pytest

from hoomd_rs_b200 import (FP32_RECHECK, FP64, ROTATE, TRANSLATE, Context, ConvexPolyhedron, HardShape, Microstate,
                           PairwiseCutoff, Periodic, lattice)

pytestmark = pytest.mark.gpu

BOX = np.array([[x, y, z] for x in (-0.5, 0.5) for y in (-0.5, 0.5) for z in (-0.5, 0.5)])
TETRAHEDRON = np.array([[1.0, 1.0, 1.0], [1.0, -1.0, -1.0], [-1.0, 1.0, -1.0], [-1.0, -1.0, 1.0]]) * 0.5
ROUND = np.random.default_rng(11).normal(size=(32, 3))
ROUND *= 0.55 / np.linalg.norm(ROUND, axis=1)[:, None]


@pytest.fixture(scope="module")
def ctx():
    return Context(0)


@pytest.mark.parametrize("name,verts,spacing", [("cubes", BOX, 1.2), ("tetrahedra", TETRAHEDRON, 1.25),
                                                ("round_32", ROUND, 1.2)])
def test_wide_bounds_leave_the_trajectory(ctx, name, verts, spacing, monkeypatch):
    L = 9 * spacing
    pos = lattice.cubic_lattice(729, L, 3, 17, jitter=0.01)
    reach = 2.0 * float(np.sqrt((verts ** 2).sum(axis=1).max()))
    h = PairwiseCutoff(HardShape(ConvexPolyhedron.with_vertices(verts)))

    def make():
        return Microstate(ctx, Periodic(reach, [L] * 3), pos, h, seed=17)

    monkeypatch.setenv("HMC_B200_FP32_BAND_SCALE", "1e5")
    wide = make()
    monkeypatch.delenv("HMC_B200_FP32_BAND_SCALE")
    runs = [(wide, FP32_RECHECK), (make(), FP32_RECHECK), (make(), FP64)]
    for sweep in range(8):
        move, maximum = ((TRANSLATE, 0.12), (ROTATE, 0.2))[sweep % 2]
        counts = [g.sweep(move, maximum, 1.0, p, n_sweeps=1, increment_step=True) for g, p in runs]
        assert len({(c.accepted, c.rejected) for c in counts}) == 1, sweep
    for g, _ in runs[1:]:
        assert np.array_equal(g.positions(), wide.positions())
        assert np.array_equal(g.orientations(), wide.orientations())


@pytest.mark.parametrize("scale", [0.8, 1.0, 1.25])
def test_versors_of_other_lengths(ctx, scale):
    """Orientations are taken as they are given; the bounds hold for versors that are not of unit length too."""
    n, L = 343, 7 * 1.9
    pos = lattice.cubic_lattice(n, L, 3, 23, jitter=0.05)
    q = np.random.default_rng(3).normal(size=(n, 4))
    q *= scale / np.linalg.norm(q, axis=1)[:, None]
    h = PairwiseCutoff(HardShape(ConvexPolyhedron.with_vertices(BOX)))
    runs = []
    for precision in (FP64, FP32_RECHECK):
        g = Microstate(ctx, Periodic(3.0 ** 0.5, [L] * 3), pos, h, seed=23)
        g.set_state(pos, 0, 0, orientations=q)
        counts = [g.sweep(m, x, 1.0, precision, n_sweeps=3, increment_step=True)
                  for m, x in ((TRANSLATE, 0.4), (ROTATE, 0.5))]
        runs.append(([(c.accepted, c.rejected) for c in counts], g.positions(), g.orientations()))
    assert runs[0][0] == runs[1][0]
    assert np.array_equal(runs[0][1], runs[1][1]) and np.array_equal(runs[0][2], runs[1][2])
