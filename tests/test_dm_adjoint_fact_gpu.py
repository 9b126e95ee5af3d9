"""The factored density-matrix adjoint (windows 3..7) where its tiles, slots
and step kinds differ: XZ / YZ steps, outcome-1 steps, fixed angles, windows
wider than the inputs (several shrinking steps, unlinked slots)."""
import numpy as np
import pytest

from helpers import haar_states
from mentpy_gb300 import circuit as C
from mentpy_gb300.dm import DensityMatrixSweep
from oracle import gradients as G

pytestmark = pytest.mark.gpu

TOL_GRAD_C64 = 2e-4  # relative to 1 + max |grad|, as test_dm_adjoint_gpu.py


def _planes(rows, cols):
    c = C.grid_cluster(rows, cols)
    c[0] = C.Ment("XZ")
    c[1] = C.Ment("YZ")
    c[cols] = C.Ment("X")
    c[cols + 1] = C.Ment("XY", 0.4)
    return c


@pytest.mark.parametrize("build,kw", [
    (lambda: _planes(2, 4), {}), (lambda: _planes(3, 4), {}), (lambda: _planes(4, 3), {}), (lambda: _planes(5, 3), {}),
    (lambda: _planes(6, 3), {}), (lambda: C.linear_cluster(9), dict(window_size=5)),
    (lambda: C.linear_cluster(12), dict(window_size=7)), (lambda: C.grid_cluster(2, 6), dict(window_size=6)),
    (lambda: C.muta(2, 1), {})])
def test_factored_adjoint_matches_differences(build, kw):
    circ = build()
    sw = DensityMatrixSweep(circ, **kw)
    assert 3 <= sw.plan.window <= 7
    rng = np.random.default_rng(101)
    ang = rng.uniform(0, 2 * np.pi, size=(2, sw.n_angles))
    psi = haar_states(rng, sw.n_in, 2)
    if 0 in sw.plan.trainable_nodes and circ[0].plane == "XZ":
        ang[0, sw.plan.trainable_nodes.index(0)] = -np.pi / 2 + 1e-3  # outcome 1 on an input in |0>
        psi[0] = 0.0
        psi[0, 0] = 1.0
    d = 2**sw.n_out
    gam = rng.standard_normal((2, d, d)) + 1j * rng.standard_normal((2, d, d))
    gam = gam + gam.conj().transpose(0, 2, 1)
    grad, rho, st = sw.adjoint(ang, psi, gam, noise=0.03)
    assert (st.cpu().numpy() == 0).all()
    fwd = sw.forward(ang, psi, noise=0.03)[0]
    assert (rho - fwd).abs().max().item() < 1e-6
    for r in range(2):
        ref = G.dm_linear_functional_grad(circ, ang[r], psi[r], gam[r], noise_p=0.03, h=1e-6, **kw)
        err = np.abs(grad[r].cpu().numpy() - ref).max() / (1 + np.abs(ref).max())
        assert err < TOL_GRAD_C64, (r, err)
