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
from hoomd_rs_b200 import (FP32_RECHECK, FP64, TRANSLATE, Context, Isotropic, LennardJones, Microstate,
                           PairwiseCutoff, Periodic, Shifted, lattice)

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
