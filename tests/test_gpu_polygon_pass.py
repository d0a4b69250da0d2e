"""The polygon colour pass where its packing can go wrong: two spaces per axis (the rows across the
fast-axis end, images of one space), a warp's trials incomplete, more pairs than a warp's list (thin
polygons, whose circumcircles hold dozens of candidates) and the fewest and the most vertices,
against the oracle's ParallelSweep.
"""
import math

import numpy as np
import pytest

import oracle
from hoomd_rs_b200 import (FP32_RECHECK, FP64, ROTATE, TRANSLATE, Context, ConvexPolygon, ConvexSurfaceMesh2d,
                           HardShape, Microstate, PairwiseCutoff, Periodic)

pytestmark = pytest.mark.gpu


def ngon(n, r=0.55):
    a = 2 * math.pi * (np.arange(n) + 0.25) / n
    return np.stack([np.cos(a), np.sin(a)], -1) * r


ROD = np.array([[-1.0, -0.05], [1.0, -0.05], [1.0, 0.05], [-1.0, 0.05]])
# vertices, sites per axis, spacing per axis, angles up to
SHAPES = {"triangles_two_spaces": (ngon(3), (2, 2), (1.2, 1.2), 3.0), "triangles": (ngon(3), (9, 7), (1.2, 1.2), 3.0),
          "octagons": (ngon(8), (5, 13), (1.15, 1.15), 3.0), "ngon_32": (ngon(32), (6, 7), (1.13, 1.13), 3.0),
          "rods": (ROD, (4, 60), (2.2, 0.16), 0.02)}


@pytest.mark.parametrize("precision", [FP64, FP32_RECHECK])
@pytest.mark.parametrize("mesh", [False, True])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_polygon_pass(name, mesh, precision):
    verts, sites, spacing, most = SHAPES[name]
    L = [n * a for n, a in zip(sites, spacing)]
    rng = np.random.default_rng(7)
    grid = np.stack(np.meshgrid(*[np.arange(n) for n in sites], indexing="ij"), -1).reshape(-1, 2)
    pos = (grid + 0.5) * spacing - np.array(L) / 2 + rng.uniform(-0.005, 0.005, grid.shape)
    angles = rng.uniform(-most, most, len(pos))
    shape = ConvexSurfaceMesh2d.from_point_set(verts) if mesh else ConvexPolygon.with_vertices(verts)
    reach = 2.0 * shape.bounding_radius
    g = Microstate(Context(0), Periodic(reach, L), pos, PairwiseCutoff(HardShape(shape)), seed=31, orientations=angles)
    o = oracle.System(2, L, pos, angles, seed=31, vertices=shape.vertices,
                      interaction=oracle.HARD_CONVEX_SURFACE_MESH_2D if mesh else oracle.HARD_CONVEX_POLYGON)
    for sweep in range(6):
        move, maximum = ((TRANSLATE, 0.1), (ROTATE, 0.1))[sweep % 2]
        c = g.sweep(move, maximum, 1.0, precision, n_sweeps=1, increment_step=True)
        want = o.parallel_sweep(oracle.TRANSLATE if move == TRANSLATE else oracle.ROTATE, maximum, 1.0, reach)
        o.increment_step()
        assert (c.accepted, c.rejected) == tuple(want), sweep
    assert np.array_equal(g.positions(), o.state()[0])
    assert np.array_equal(g.orientations(), o.state()[1].reshape(-1))
