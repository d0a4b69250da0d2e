"""Where a launch choice applies: recorded ones to boxes of their size class, a system's own to its pass."""
import numpy as np
import pytest

from hoomd_rs_b200 import (FP32_RECHECK, FP64, TRANSLATE, Batch, Context, ConvexPolyhedron, GrandCanonical, HardShape,
                           HardSphere, HmcError, IsothermalIsofugacity, Isotropic, LennardJones, Microstate,
                           PairwiseCutoff, Periodic, Shifted, lattice)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return Context(0)


def lj(ctx, n, rho, dim=3, r_cut=2.5):
    pos, L = lattice.lennard_jones_box(n, rho, dim, 7)
    h = PairwiseCutoff(Isotropic(Shifted(LennardJones(1.0, 1.0), r_cut), r_cut))
    return Microstate(ctx, Periodic(r_cut, [L] * dim), pos, h, seed=7)


# (4,096 sites run 8 warps a trial, 200,000 two)
@pytest.mark.parametrize("precision", [FP64, FP32_RECHECK])
@pytest.mark.parametrize("rho", [0.72, 0.77, 0.84, 0.93, 1.02, 1.12])
def test_a_recorded_team_stays_in_its_size_class(ctx, rho, precision):
    small = lj(ctx, 4096, rho)
    chosen, ms = small.autotune(TRANSLATE, 0.1, 1.0, precision, sweeps=2)
    assert len(ms) == chosen["count"] == 5 and ms[chosen["index"]] == ms.min()
    assert ms[0] in ms[1:]  # variant 0 is one of the teams, and not timed twice
    assert lj(ctx, 4096, rho).launch_variant(precision)["index"] == chosen["index"]
    assert lj(ctx, 200000, rho).launch_variant(precision)["index"] == 0
    assert lj(ctx, 200000, rho, r_cut=2.7).launch_variant(precision)["index"] == 0


@pytest.mark.parametrize("rho", [0.72, 0.84, 1.02])
def test_a_recorded_batch_team_stays_in_its_size_class(ctx, rho):
    def batch(n):
        h = PairwiseCutoff(Isotropic(Shifted(LennardJones(1.0, 1.0), 2.5), 2.5))
        pos, L = lattice.lennard_jones_box(n, rho, 3, 7)
        return Batch(ctx, [{"boundary": Periodic(2.5, [L] * 3), "positions": pos, "seed": 7 + k, "hamiltonian": h}
                           for k in range(2)])

    small = batch(4096)
    chosen, ms = small.autotune(0.1, FP32_RECHECK, sweeps=2, temperatures=np.ones(2))
    assert ms[0] in ms[1:]
    large = batch(100000)
    chosen_large, ms = large.autotune(0.1, FP32_RECHECK, sweeps=1, temperatures=np.ones(2))
    assert ms[0] in ms[1:]


def spheres(ctx, n, precision, dim=3, phi=0.45):
    pos, L = lattice.hard_sphere_box(n, phi, dim, 7)
    return Microstate(ctx, Periodic(1.0, [L] * dim), pos, PairwiseCutoff(HardSphere(1.0)), seed=7)


@pytest.mark.parametrize("precision", [FP64, FP32_RECHECK])
def test_an_own_variant_stays_with_its_pass(ctx, precision):
    """A small box's variant is one of the dataflow sweep; the colour passes' tables mean other shapes by it."""
    g = spheres(ctx, 4096, precision)
    flow = g.launch_variant(precision)
    assert flow["trials_per_warp"] == 3
    g.set_launch_variant(precision, 1)
    assert g.launch_variant(precision) == dict(g.launch_variant(precision, 1))
    for coop in (False, True):
        g.set_cooperative_pass(precision, coop)
        v = g.launch_variant(precision)
        assert v["trials_per_warp"] == 1 and v["index"] == 0
        g.set_launch_variant(precision, 2)
        assert g.launch_variant(precision)["index"] == 2
        g.set_cooperative_pass(precision, coop)  # the same pass again keeps it
        assert g.launch_variant(precision)["index"] == 2
    g.set_cooperative_pass(precision, False)
    assert g.launch_variant(precision)["index"] == 0


def test_an_own_variant_stays_with_its_pass_across_the_line(ctx):
    """Removing bodies takes a box of more than 114,695 spheres to the dataflow sweeps."""
    g = spheres(ctx, 114700, FP32_RECHECK)
    assert g.launch_variant(FP32_RECHECK)["trials_per_warp"] == 1
    g.set_launch_variant(FP32_RECHECK, 1)
    GrandCanonical().apply(g, None, IsothermalIsofugacity(1.0, 0.0), 64)
    assert len(g.positions()) < 114696
    v = g.launch_variant(FP32_RECHECK)
    assert v["trials_per_warp"] == 3 and v["index"] == 0
    g.sweep(TRANSLATE, 0.1, 1.0, FP32_RECHECK, n_sweeps=1, increment_step=True)


def cubes(ctx):
    verts = np.array([[x, y, z] for x in (-0.5, 0.5) for y in (-0.5, 0.5) for z in (-0.5, 0.5)])
    return Microstate(ctx, Periodic(3.0 ** 0.5, [12.5] * 3), lattice.cubic_lattice(1000, 12.5, 3, 7),
                      PairwiseCutoff(HardShape(ConvexPolyhedron.with_vertices(verts))), seed=7)


# The indices of the colour passes that these boxes ran before they had dataflow sweeps, or another
# default pass: 3 shapes of polyhedra and of a lane per sphere, 5 of a warp per sphere.
@pytest.mark.parametrize("make,precision,accepted", [
    (cubes, FP32_RECHECK, 3), (cubes, FP64, 3),
    (lambda ctx: spheres(ctx, 4096, FP32_RECHECK), FP32_RECHECK, 3), (lambda ctx: spheres(ctx, 4096, FP64), FP64, 5),
    (lambda ctx: spheres(ctx, 100000, FP64, 2, 0.6), FP64, 5)])
def test_a_kept_index_is_accepted(ctx, make, precision, accepted):
    """An index beyond the table of the pass that runs now stands for variant 0."""
    g = make(ctx)
    count = g.launch_variant(precision)["count"]
    for index in range(accepted):
        g.set_launch_variant(precision, index)
        want = index if index < count else 0
        assert g.launch_variant(precision)["index"] == g.launch_variant(precision, index)["index"] == want
    g.sweep(TRANSLATE, 0.1, 1.0, precision, n_sweeps=1, increment_step=True)
    for refused in (accepted, 1000):
        with pytest.raises(HmcError):
            g.set_launch_variant(precision, refused)
        with pytest.raises(HmcError):
            g.launch_variant(precision, refused)


@pytest.mark.parametrize("precision,coop,accepted", [(FP64, False, 3), (FP64, True, 5), (FP32_RECHECK, False, 3)])
def test_a_pass_that_was_chosen_has_its_own_indices(ctx, precision, coop, accepted):
    g = spheres(ctx, 4096, precision)
    g.set_cooperative_pass(precision, coop)
    g.set_launch_variant(precision, accepted - 1)
    with pytest.raises(HmcError):
        g.set_launch_variant(precision, accepted)


@pytest.mark.parametrize("n,phi,precision", [(250000, 0.02, FP64), (4096, 0.45, FP32_RECHECK), (4096, 0.45, FP64)])
def test_autotune_of_few_spheres_chooses_among_three_forms(ctx, n, phi, precision):
    """Dilute boxes near the dataflow sweeps' line run a colour pass a third faster; small ones do not."""
    g = spheres(ctx, n, precision, phi=phi)
    g.sweep(TRANSLATE, 0.1, 1.0, precision, n_sweeps=2, increment_step=True)
    before = g.state()
    chosen, ms = g.autotune(TRANSLATE, 0.1, 1.0, precision, sweeps=4)
    assert len(ms) == chosen["count"] and ms[chosen["index"]] == ms.min()
    flow = chosen["trials_per_warp"] == 3
    assert flow == (n == 4096)
    after = g.state()
    assert np.array_equal(before[0], after[0]) and before[1:] == after[1:]
    twin, other = spheres(ctx, n, precision, phi=phi), spheres(ctx, 2000, precision, phi=phi)
    assert twin.launch_variant(precision) == g.launch_variant(precision) == chosen
    assert other.launch_variant(precision)["trials_per_warp"] == 3  # another size has its own choice
    for s in (g, twin):
        s.set_state(*before)
    counts = [s.sweep(TRANSLATE, 0.1, 1.0, precision, n_sweeps=2, increment_step=True) for s in (g, twin)]
    assert counts[0].accepted == counts[1].accepted and np.array_equal(g.positions(), twin.positions())
    # tuning again starts from the choice, and a pass that is set by hand is the only one tuned
    again, _ = g.autotune(TRANSLATE, 0.1, 1.0, precision, sweeps=2)
    assert (again["trials_per_warp"] == 3) == flow
    g.set_cooperative_pass(precision, True)
    assert g.autotune(TRANSLATE, 0.1, 1.0, precision, sweeps=1)[0]["count"] == 5


# bodies, packing fraction: on both sides of the dataflow sweeps' line, which falls with the density
@pytest.mark.parametrize("dim,n,phi,precision,flow", [
    (3, 114000, 0.45, FP32_RECHECK, True), (3, 114000, 0.05, FP32_RECHECK, False), (3, 60000, 0.03, FP32_RECHECK, True),
    (3, 250000, 0.45, FP64, True), (3, 260000, 0.30, FP64, True), (3, 250000, 0.11, FP64, False), (3, 60000, 0.03, FP64, True),
    (2, 24000, 0.5, FP64, True), (2, 24000, 0.06, FP64, False), (2, 5000, 0.06, FP64, True)])
def test_the_line_falls_with_the_density(ctx, dim, n, phi, precision, flow):
    g = spheres(ctx, n, precision, dim, phi)
    assert (g.launch_variant(precision)["trials_per_warp"] == 3) == flow
    o = spheres(ctx, n, precision, dim, phi)
    o.set_cooperative_pass(precision, True)  # the other form
    counts = [s.sweep(TRANSLATE, 0.2, 1.0, precision, n_sweeps=2, increment_step=True) for s in (g, o)]
    assert counts[0].accepted == counts[1].accepted and np.array_equal(g.positions(), o.positions())
