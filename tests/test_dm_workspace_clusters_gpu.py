"""Density-matrix sweeps whose matrix lies in the workspace (csrc/dm_fact.cuh,
dm_fwd_fact_ws) on the routes that need a large batch or a long circuit: two blocks a
run at windows 10 and 11 (more runs than half the SMs), window 9 once its step tables
do not fit beside the rows in shared memory (from about 6,800 steps on)."""
import numpy as np
import pytest
import torch

from helpers import haar_states
from mentpy_gb300 import circuit as C
from mentpy_gb300.dm import DensityMatrixSweep
from mentpy_gb300.sweep import StatevectorSweep
from oracle import sweep as oracle

pytestmark = pytest.mark.gpu

TOL_RHO_C64 = 2e-5  # as test_dm_gpu.py


def _batch(circ, rows, B, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(0, 2 * np.pi, size=(B, len(circ.trainable_nodes))), haar_states(rng, rows, B)


def test_window_10_in_two_blocks_a_run():
    circ = C.grid_cluster(9, 3)
    ang, psi = _batch(circ, 9, 100, 61)
    sw = DensityMatrixSweep(circ)
    assert sw.plan.window == 10
    rho, outc, st, probs = sw.forward(ang, psi, noise=0.01, want_probs=True)
    assert int((st != 0).sum()) == 0
    ref, ref_out, _ = oracle.run_dm(circ, ang[99], psi[99], noise_p=0.01)
    assert np.abs(rho[99].cpu().numpy() - ref).max() < TOL_RHO_C64
    assert [ref_out[n] for n in sw.plan.schedule_measure] == outc[99].tolist()
    one = sw.forward(ang[:1], psi[:1], noise=0.01, want_probs=True)  # a cluster's shared memory
    assert (rho[0] - one[0][0]).abs().max().item() < 1e-6
    assert (probs[0] - one[3][0]).abs().max().item() < 1e-6


@pytest.mark.parametrize("build,rows,B,tol", [
    (lambda: C.grid_cluster(10, 3), 10, 80, TOL_RHO_C64),
    # four float32 roundings a step on entries of at most ~0.03: 6,872 * 4 * 6e-8 * 0.03
    (lambda: C.many_wires([860] * 8), 8, 2, 5e-5),
])
def test_noise_free_matrix_is_the_statevectors(build, rows, B, tol):
    circ = build()
    ang, psi = _batch(circ, rows, B, 62)
    sw = DensityMatrixSweep(circ)
    assert sw.plan.window == rows + 1
    rho, outc, st, _ = sw.forward(ang, psi)
    assert int((st != 0).sum()) == 0 and int(outc.sum()) == 0
    z = StatevectorSweep(circ, dtype=torch.complex128).forward(ang, psi)[0] if rows < 10 else None
    if z is None:
        z = StatevectorSweep(circ).forward(ang, psi)[0].to(torch.complex128)
    for r in (0, B - 1):
        assert (rho[r] - torch.outer(z[r], z[r].conj())).abs().max().item() < tol
