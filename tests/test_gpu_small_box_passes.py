"""The hard-sphere colour passes on small boxes.

Few spheres run in dataflow order unless a pass is chosen, so the tests that use small boxes check the dataflow
sweep. Here the same tests run with each colour pass (a lane, a warp per trial) chosen when a system is
created: trajectories against the oracle, adversarial injected trials, two spaces per axis, empty and one-body
boxes, pipelined calls, every launch variant, and the tuner.
"""
import pytest

import test_gpu_autotune as autotune
import test_gpu_colour_pass_trials as trials
import test_gpu_edge_cases as edges
import test_gpu_full_size as full
import test_gpu_launch_choice as choice
import test_gpu_pipelined as pipelined
import test_gpu_sphere as sphere
from hoomd_rs_b200 import FP32_RECHECK, FP64, Context

pytestmark = pytest.mark.gpu

PRECISIONS = pytest.mark.parametrize("precision", [FP64, FP32_RECHECK])


@pytest.fixture(scope="module")
def ctx():
    return Context(0)


@pytest.fixture(params=["direct", "coop"], autouse=True)
def colour_pass(request, monkeypatch):
    monkeypatch.setenv("HMC_B200_SWEEP_KERNEL", request.param)
    return request.param


def test_the_pass_is_chosen(ctx, colour_pass):
    for dim, n in ((3, 1000), (2, 500)):
        for precision in (FP64, FP32_RECHECK):
            g = choice.spheres(ctx, n, precision, dim, 0.4)
            assert g.cooperative_pass(precision) == (colour_pass == "coop")
            assert g.launch_variant(precision)["trials_per_warp"] == 1


@PRECISIONS
@pytest.mark.parametrize("dim,n,phi,d,sweeps", [(3, 4000, 0.50, 0.15, 4), (3, 729, 0.30, 0.3, 4), (2, 4096, 0.70, 0.1, 4),
                                                (2, 777, 0.40, 0.3, 4)])
def test_trajectories(ctx, dim, n, phi, d, sweeps, precision):
    sphere.test_trajectory_bit_identical_to_oracle(ctx, dim, n, phi, d, sweeps, precision)


@pytest.mark.parametrize("dim,n,phi,d", [(3, 4000, 0.50, 0.15), (2, 4096, 0.70, 0.1)])
def test_wide_band(ctx, monkeypatch, dim, n, phi, d):
    sphere.test_wide_fp32_band_rechecks_in_fp64(ctx, monkeypatch, dim, n, phi, d)


@PRECISIONS
def test_several_bodies_in_a_space(ctx, precision):
    sphere.test_large_spaces_choose_among_several_bodies(ctx, precision)


@PRECISIONS
@pytest.mark.parametrize("dim,L,n", [(3, [2.4, 2.6, 4.4], 6), (2, [2.2, 2.9], 3), (2, [4.3, 2.1], 4)])
def test_two_spaces_per_axis(ctx, dim, L, n, precision):
    sphere.test_two_spaces_per_axis(ctx, dim, L, n, precision)


@pytest.mark.parametrize("dim,n,phi", [(3, 32768, 0.50), (2, 4096, 0.70)])
def test_injected_trials(ctx, dim, n, phi):
    trials.test_sphere_trials_through_the_colour_passes(ctx, dim, n, phi, 2_000_000, 400_000)


@PRECISIONS
@pytest.mark.parametrize("dim", [2, 3])
def test_empty_and_one_body(ctx, dim, precision):
    edges.test_empty_system_sweeps(ctx, dim, precision)
    edges.test_one_body_matches_oracle(ctx, dim, precision)


@PRECISIONS
def test_pairs_at_contact(ctx, precision):
    edges.test_pairs_at_contact_distance_match_oracle(ctx, precision)


@PRECISIONS
@pytest.mark.parametrize("kind", ["spheres", "disks"])
def test_pipelined(ctx, kind, precision):
    pipelined.test_pipelined_sweeps_equal_one_call_per_sweep(ctx, kind, precision)


@PRECISIONS
def test_thousand_sweeps(ctx, precision):
    full.test_hard_disks_4096_thousand_sweeps(ctx, precision)


@PRECISIONS
@pytest.mark.parametrize("kind", ["spheres3", "disks"])
def test_variants(ctx, kind, precision, colour_pass):
    make = autotune.spheres(ctx) if kind == "spheres3" else autotune.spheres(ctx, 2, 4096, 0.7)
    assert make().launch_variant(precision)["count"] == (5 if colour_pass == "coop" else 3)
    autotune.test_every_variant_gives_the_same_trajectory(ctx, kind, precision)


@PRECISIONS
def test_autotune(ctx, precision):
    autotune.test_autotune_restores_state_and_records_its_choice(ctx, precision)


def test_autotune_of_a_dilute_box_records_the_pass(ctx, colour_pass, monkeypatch):
    """Without a pass chosen, where a colour pass is the fastest form: both are timed, pass and variant recorded."""
    monkeypatch.delenv("HMC_B200_SWEEP_KERNEL")
    n, phi = 200000 + (1000 if colour_pass == "coop" else 0), 0.02
    g, twin = choice.spheres(ctx, n, FP64, phi=phi), choice.spheres(ctx, n, FP64, phi=phi)
    chosen, ms = g.autotune(0, 0.1, 1.0, FP64, sweeps=3)
    assert len(ms) == chosen["count"] and chosen["trials_per_warp"] == 1
    assert chosen["count"] == (5 if g.cooperative_pass(FP64) else 3)
    assert twin.cooperative_pass(FP64) == g.cooperative_pass(FP64)
    assert twin.launch_variant(FP64) == chosen
