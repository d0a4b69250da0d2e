"""Lennard-Jones and Isotropic sweeps whose trials have few candidates, so that their lanes load the sites.

Trajectories against the oracle's ParallelSweep on both sides of the rule's lines: few and many spaces
per colour, fewer and more candidates than a warp has lanes, empty stencils, images at the box's ends.
"""
import numpy as np
import pytest

import oracle
from hoomd_rs_b200 import (FP32_RECHECK, FP64, TRANSLATE, Batch, Context, Isotropic, LennardJones, Microstate,
                           OverlapPenalty, PairwiseCutoff, Periodic, Shifted, lattice)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return Context(0)


def compare(g, o, precision, move, kt, r_cut, sweeps=2):
    for _ in range(sweeps):
        want = o.parallel_sweep(oracle.TRANSLATE, move, kt, r_cut)
        o.increment_step()
        c = g.sweep(TRANSLATE, move, kt, precision, n_sweeps=1, increment_step=True)
        assert (c.accepted, c.rejected) == tuple(want)
    assert np.array_equal(g.positions(), o.state()[0])


LJ = PairwiseCutoff(Isotropic(Shifted(LennardJones(1.0, 1.0), 2.5), 2.5))


# dim, sites, density: 4 to 24 candidates in small boxes (two spaces an axis among them), 3 to 90 in boxes of
# 4,600 spaces a colour and more
@pytest.mark.parametrize("precision", [FP64, FP32_RECHECK])
@pytest.mark.parametrize("dim,n,rho", [(2, 12, 0.3), (2, 1500, 0.05), (2, 3000, 0.3), (3, 5, 0.03), (3, 1200, 0.02),
                                       (3, 3000, 0.05), (2, 6200, 0.05), (2, 62000, 0.5), (2, 110000, 0.9),
                                       (3, 19000, 0.03), (3, 62000, 0.1), (3, 100000, 0.16)])
def test_lj(ctx, dim, n, rho, precision):
    pos, L = lattice.lennard_jones_box(n, rho, dim, 11, jitter=0.3 if rho < 0.1 else 0.05)
    g = Microstate(ctx, Periodic(2.5, [L] * dim), pos, LJ, seed=11)
    o = oracle.System(dim, [L] * dim, pos, seed=11, interaction=oracle.LENNARD_JONES, lj_epsilon=1.0, lj_sigma=1.0,
                      lj_r_cut=2.5, lj_r_shift=2.5)
    compare(g, o, precision, 0.3 if rho < 0.1 else 0.12, 1.3, 2.5)


@pytest.mark.parametrize("precision", [FP64, FP32_RECHECK])
def test_lj_one_crowded_corner(ctx, precision):
    """A dilute box with a droplet: single trials with several times 32 candidates."""
    a, _ = lattice.lennard_jones_box(6000, 0.05, 2, 11, jitter=0.3)
    L = (6000 / 0.05) ** 0.5
    drop = lattice.cubic_lattice(196, 15.5, 2, 12, jitter=0.02)
    pos = np.concatenate([a[np.abs(a).max(axis=1) > 10.0], drop])
    g = Microstate(ctx, Periodic(2.5, [L] * 2), pos, LJ, seed=11)
    o = oracle.System(2, [L] * 2, pos, seed=11, interaction=oracle.LENNARD_JONES, lj_epsilon=1.0, lj_sigma=1.0,
                      lj_r_cut=2.5, lj_r_shift=2.5)
    compare(g, o, precision, 0.2, 1.0, 2.5, sweeps=3)


@pytest.mark.parametrize("n,dim,rho", [(400, 2, 0.7), (15000, 2, 0.7), (1000, 3, 0.8), (34000, 3, 0.8)])
def test_penalty(ctx, n, dim, rho):
    pos, L = lattice.lennard_jones_box(n, rho, dim, 5, jitter=0.1)
    g = Microstate(ctx, Periodic(1.0, [L] * dim), pos, PairwiseCutoff(Isotropic(OverlapPenalty(100.0, 0.3, 2.0), 1.0)),
                   seed=5)
    o = oracle.System(dim, [L] * dim, pos, seed=5, interaction=oracle.ISOTROPIC,
                      isotropic={"kind": oracle.UV_OVERLAP_PENALTY, "params": [100.0, 0.3, 2.0], "r_cut": 1.0})
    compare(g, o, FP64, 0.15, 1.0, 1.0)


@pytest.mark.parametrize("precision", [FP64, FP32_RECHECK])
@pytest.mark.parametrize("replicas,n,rho", [(3, 300, 0.02), (4, 9000, 0.08)])
def test_batches_equal_single_systems(ctx, replicas, n, rho, precision):
    reps, singles = [], []
    for k in range(replicas):
        pos, L = lattice.lennard_jones_box(n + 17 * k, rho, 3, 60 + k, jitter=0.2)
        reps.append({"boundary": Periodic(2.5, [L] * 3), "positions": pos, "seed": 60 + k, "hamiltonian": LJ})
        singles.append(Microstate(ctx, Periodic(2.5, [L] * 3), pos, LJ, seed=60 + k))
    b = Batch(ctx, reps)
    b.sweep(0.3, precision, n_sweeps=2, increment_step=True, temperatures=np.full(replicas, 1.2))
    for k, s in enumerate(singles):
        s.sweep(TRANSLATE, 0.3, 1.2, precision, n_sweeps=2, increment_step=True)
        assert np.array_equal(b.positions(k), s.positions()), k
