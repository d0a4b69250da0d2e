"""The arrays of a round's trial moves, by space: hard polyhedra keep theirs in the draws of the dataflow sweep."""
import numpy as np
import pytest
import torch

from hoomd_rs_b200 import (FP64, ROTATE, TRANSLATE, Anisotropic, ApproximateShapeOverlap, Context, ConvexPolyhedron,
                           HardShape, Microstate, OverlapPenalty, PairwiseCutoff, Periodic, lattice)

pytestmark = pytest.mark.gpu

CUBE = np.array([[x, y, z] for x in (-0.5, 0.5) for y in (-0.5, 0.5) for z in (-0.5, 0.5)])
REACH = 3.0 ** 0.5


@pytest.fixture(scope="module")
def ctx():
    return Context(0)


def cubes(ctx, L, n=1000):
    return Microstate(ctx, Periodic(REACH, [L] * 3), lattice.cubic_lattice(n, L, 3, 7),
                      PairwiseCutoff(HardShape(ConvexPolyhedron.with_vertices(CUBE))), seed=7)


def test_hard_polyhedra_hold_none(ctx):
    cubes(ctx, 20.0).close()
    before = torch.cuda.mem_get_info(0)[0]
    g = cubes(ctx, 160.0 * REACH * 1.001)  # 160^3 spaces, 84 bytes each in these arrays
    taken = before - torch.cuda.mem_get_info(0)[0]
    assert taken < 40 * 160 ** 3, taken
    g.sweep(TRANSLATE, 0.1, 1.0, FP64, n_sweeps=1, increment_step=True)


def test_the_approximate_overlap_brings_them(ctx):
    """Switched on and off around a box that grows: as a system that starts in the large box."""
    soft = PairwiseCutoff(Anisotropic(ApproximateShapeOverlap(ConvexPolyhedron.with_vertices(CUBE),
                                                              OverlapPenalty(100.0, 0.5, 0.0), resolution=0.02), REACH))
    a = cubes(ctx, 14.0)
    a.set_hamiltonian(soft)
    a.sweep(TRANSLATE, 0.05, 1.0, FP64, n_sweeps=1, increment_step=True)
    a.set_hamiltonian(a.hamiltonian)
    a.set_box([30.0] * 3)
    b = Microstate(ctx, Periodic(REACH, [30.0] * 3), a.positions(),
                   PairwiseCutoff(HardShape(ConvexPolyhedron.with_vertices(CUBE))), seed=7, step=1)
    pos, ori = a.positions(), a.orientations()
    for s in (a, b):
        s.set_state(pos, 1, 0, orientations=ori)
        s.set_hamiltonian(soft)
        for move in (TRANSLATE, ROTATE):
            s.sweep(move, 0.2, 1.0, FP64, n_sweeps=2, increment_step=True)
        s.set_hamiltonian(s.hamiltonian)
        s.sweep(ROTATE, 0.2, 1.0, FP64, n_sweeps=1, increment_step=True)
    assert np.array_equal(a.positions(), b.positions()) and np.array_equal(a.orientations(), b.orientations())
