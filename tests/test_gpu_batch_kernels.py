"""The kernels that a batch of Lennard-Jones replicas reports: spaces of four bodies and more are ordered by one more."""
import numpy as np
import pytest

from hoomd_rs_b200 import FP32_RECHECK, Batch, Context, Isotropic, LennardJones, PairwiseCutoff, Periodic, Shifted, lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rho,rebuild", [(0.8, 7), (0.1, 6)])
@pytest.mark.parametrize("captured", [False, True])
def test_lj_batch_counts_its_kernels(rho, rebuild, captured):
    h = PairwiseCutoff(Isotropic(Shifted(LennardJones(1.0, 1.0), 2.5), 2.5))
    pos, L = lattice.lennard_jones_box(2000, rho, 3, 7)
    b = Batch(Context(0), [{"boundary": Periodic(2.5, [L] * 3), "positions": pos, "seed": k, "hamiltonian": h}
                           for k in range(3)])
    b.set_captured_sweeps(captured)
    before = b.kernel_launches()
    b.sweep(0.1, FP32_RECHECK, n_sweeps=4, increment_step=True, temperatures=np.ones(3))
    launched = b.kernel_launches() - before
    # per sweep: captured: origins, rounds, the loop's first test and the end, then draws, sweep and the step to the
    # next sets; else the rounds, then draws and sweep; one launch holds all colour sets of equal replicas, or the host
    # enqueues at most one more than it needs
    if captured:
        assert launched == 4 * (4 + rebuild + 3)
    else:
        assert (launched - 4 * (1 + rebuild)) % 2 == 0 and 8 <= launched - 4 * (1 + rebuild) <= 16
