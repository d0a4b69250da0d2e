"""Waits of the dataflow sweeps that run out (hmc_flow.cuh, FlowLimit).

A test switch leaves out the first trial of a launch, so that the trials around it wait for a space that
nothing releases, or lets the staging barriers expect bytes that nobody copies; with a limit of some
milliseconds every such wait ends and the call returns HMC_TIMEOUT. The context stays usable, and
trials whose sites did not arrive are not decided.
"""
import numpy as np
import pytest

from hoomd_rs_b200 import (FP32_RECHECK, FP64, TRANSLATE, Batch, Context, ConvexPolyhedron, HardShape, HardSphere,
                           HmcError, Isotropic, LennardJones, Microstate, PairwiseCutoff, Periodic, Shifted, lattice)

pytestmark = pytest.mark.gpu

TIMEOUT = 7
CUBE = np.array([[x, y, z] for x in (-0.5, 0.5) for y in (-0.5, 0.5) for z in (-0.5, 0.5)])
LJ = PairwiseCutoff(Isotropic(Shifted(LennardJones(1.0, 1.0), 2.5), 2.5))


@pytest.fixture(scope="module")
def ctx():
    return Context(0)


def system(ctx, kind, seed=3):
    if kind == "lj":
        pos, L = lattice.lennard_jones_box(4000, 0.8, 3, seed)
        return Microstate(ctx, Periodic(2.5, [L] * 3), pos, LJ, seed=seed)
    if kind == "cubes":
        pos = lattice.cubic_lattice(1000, 12.5, 3, seed, jitter=0.01)
        return Microstate(ctx, Periodic(3.0 ** 0.5, [12.5] * 3), pos,
                          PairwiseCutoff(HardShape(ConvexPolyhedron.with_vertices(CUBE))), seed=seed)
    dim = 3 if kind == "spheres" else 2
    pos, L = lattice.hard_sphere_box(4096, 0.5, dim, seed)
    return Microstate(ctx, Periodic(1.0, [L] * dim), pos, PairwiseCutoff(HardSphere(1.0)), seed=seed)


def batch(ctx, captured):
    reps = []
    for k in range(4):
        pos, L = lattice.lennard_jones_box(2000, 0.8, 3, 40 + k)
        reps.append({"boundary": Periodic(2.5, [L] * 3), "positions": pos, "seed": 40 + k, "hamiltonian": LJ})
    b = Batch(ctx, reps)
    b.set_captured_sweeps(captured)
    return b


def stalled(make, sweep, monkeypatch, what):
    """The system with the switch on, after the sweep that ran out of time."""
    monkeypatch.setenv("HMC_B200_FLOW_WAIT_MS", "20")
    monkeypatch.setenv("HMC_B200_FLOW_STALL", what)
    g = make()
    monkeypatch.delenv("HMC_B200_FLOW_STALL")
    monkeypatch.delenv("HMC_B200_FLOW_WAIT_MS")
    with pytest.raises(HmcError) as e:
        sweep(g)
    assert e.value.status == TIMEOUT
    return g


@pytest.mark.parametrize("n_sweeps", [1, 3])
@pytest.mark.parametrize("precision", [FP64, FP32_RECHECK])
@pytest.mark.parametrize("kind", ["lj", "cubes", "spheres", "disks"])
def test_a_space_that_is_never_released(ctx, kind, precision, n_sweeps, monkeypatch):
    def sweep(g):
        g.sweep(TRANSLATE, 0.1, 1.0, precision, n_sweeps=n_sweeps, increment_step=True)

    for variant in range(1, 5) if kind == "lj" else (0,):
        def make():
            g = system(ctx, kind)
            g.set_launch_variant(precision, variant)
            return g

        g = stalled(make, sweep, monkeypatch, "trial")
        before, after = system(ctx, kind), g.state()
        assert after[1:] == before.state()[1:]  # the counter has not advanced
        assert np.all(np.isfinite(after[0]))
        # part of the sweep is done: each body is where it was or where the whole sweep puts it after some trial
        assert not np.array_equal(after[0], before.positions())
        sweep(before)  # the context goes on, with the same sweep in a fresh system
        g.close()


@pytest.mark.parametrize("precision", [FP64, FP32_RECHECK])
@pytest.mark.parametrize("variant", [1, 2, 3, 4])
def test_sites_that_do_not_arrive(ctx, variant, precision, monkeypatch):
    def make():
        g = system(ctx, "lj")
        g.set_launch_variant(precision, variant)
        return g

    def sweep(g):
        g.sweep(TRANSLATE, 0.1, 1.0, precision, n_sweeps=1, increment_step=True)

    g = stalled(make, sweep, monkeypatch, "copy")
    fresh = make()
    assert np.array_equal(g.positions(), fresh.positions())  # no trial was decided
    sweep(fresh)


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("what", ["trial", "copy"])
def test_batches(ctx, captured, what, monkeypatch):
    def sweep(b):
        b.sweep(0.1, FP32_RECHECK, n_sweeps=3, increment_step=True, temperatures=np.ones(4))

    b = stalled(lambda: batch(ctx, captured), sweep, monkeypatch, what)
    fresh = batch(ctx, captured)
    if what == "copy":
        assert all(np.array_equal(b.positions(k), fresh.positions(k)) for k in range(4))
    assert b.state(0)[1:] == fresh.state(0)[1:]
    sweep(fresh)


@pytest.mark.parametrize("n_sweeps", [1, 3])
@pytest.mark.parametrize("kind", ["lj", "cubes"])
def test_a_wait_in_the_colour_sets_that_follow_the_count(ctx, kind, n_sweeps, monkeypatch):
    """One colour set per launch: the sets beyond the host's guess are enqueued after a first look at the flags."""
    def sweep(g):
        g.sweep(TRANSLATE, 0.1, 1.0, FP32_RECHECK, n_sweeps=n_sweeps, increment_step=True)

    monkeypatch.setenv("HMC_B200_FLOW_SETS", "1")
    # cubes: 1,000 bodies in 6^3 spaces, five colour sets or more; the first sweep guesses two
    g = stalled(lambda: system(ctx, kind), sweep, monkeypatch, "trial:3")
    assert g.state()[1:] == system(ctx, kind).state()[1:]
