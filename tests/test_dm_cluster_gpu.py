"""Windows 9 and 10 of the density-matrix sweep on a cluster of blocks: the
steps that need more than prob0 (Z measurements, outcome 1), single-layout and
multi-layout sweeps, and the batch sizes where the route changes."""
import numpy as np
import pytest
import torch

from helpers import haar_states
from mentpy_gb300 import circuit as C
from mentpy_gb300.dm import DensityMatrixSweep
from oracle import sweep as oracle

pytestmark = pytest.mark.gpu

TOL_RHO_C64 = 2e-5  # as test_dm_gpu.py


def _planes(rows, cols):
    c = C.grid_cluster(rows, cols)
    c[0] = C.Ment("XZ")  # outcome 1 at -pi / 2 on an input in |0>
    c[cols] = C.Ment("Z")
    return c


@pytest.mark.parametrize("rows,cols", [(8, 3), (8, 4), (9, 3)])
@pytest.mark.parametrize("mode", ["sample", "expectation"])
def test_planes_and_outcomes_on_a_cluster(rows, cols, mode):
    circ = _planes(rows, cols)
    sw = DensityMatrixSweep(circ)
    assert sw.plan.window == rows + 1
    rng = np.random.default_rng(91)
    ang = rng.uniform(0, 2 * np.pi, size=(2, sw.n_angles))
    ang[:, sw.plan.trainable_nodes.index(0)] = [-np.pi / 2, 0.3]
    psi = haar_states(rng, rows, 2)
    psi[0] = 0.0
    psi[0, 0] = 1.0
    rho, outc, st, _ = sw.forward(ang, psi, noise=0.02, mode=mode, seed=5)
    assert (st.cpu().numpy() == 0).all()
    zk = sw.plan.schedule_measure.index(cols)
    outc = outc.cpu().numpy()
    for r in range(2):
        kw = dict(mode="expectation") if mode == "expectation" else dict(z_outcomes={cols: int(outc[r][zk])})
        ref, ref_out, _ = oracle.run_dm(circ, ang[r], psi[r], noise_p=0.02, **kw)
        assert np.abs(rho[r].cpu().numpy() - ref).max() < TOL_RHO_C64
        for k, node in enumerate(sw.plan.schedule_measure):
            assert k == zk or ref_out[node] == outc[r][k]


@pytest.mark.parametrize("rows,cols,batches", [(8, 5, (1, 39, 60)), (9, 4, (1, 4, 5, 20, 40))])
def test_results_do_not_depend_on_the_batch_route(rows, cols, batches):
    """Clusters in shared memory, clusters over the workspace with 8, 4 or 2
    blocks a run, and clusters looping over runs: the same element-wise
    arithmetic, sums to float-pair accuracy (so equal but for single-ulp
    differences of a scale, ~1e-7 of entries of at most 1)."""
    sw = DensityMatrixSweep(C.grid_cluster(rows, cols))
    rng = np.random.default_rng(92)
    n = max(batches)
    ang = torch.as_tensor(rng.uniform(0, 2 * np.pi, size=(n, sw.n_angles)), device="cuda")
    psi = torch.as_tensor(haar_states(rng, rows, n), dtype=torch.complex64, device="cuda")
    ref = None
    for b in sorted(batches, reverse=True):
        rho, outc, st, probs = sw.forward(ang[:b], psi[:b], noise=0.01, want_probs=True)
        assert int((st != 0).sum()) == 0
        if ref is None:
            ref = (rho, outc, probs)
        assert (rho - ref[0][:b]).abs().max().item() < 1e-6
        assert torch.equal(outc, ref[1][:b])
        assert (probs - ref[2][:b]).abs().max().item() < 1e-6
