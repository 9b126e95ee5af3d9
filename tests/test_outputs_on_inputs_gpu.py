"""One buffer for inputs and outputs: the log-probability is relative to the norm of
the input, which has to be read before any output is written."""
import numpy as np
import pytest
import torch

from helpers import haar_states
from mentpy_gb300 import circuit as C
from mentpy_gb300.sweep import StatevectorSweep

pytestmark = pytest.mark.gpu


def _check(circ, B, **kw):
    sw = StatevectorSweep(circ, **kw)
    rng = np.random.default_rng(611)
    ang = rng.uniform(0, 2 * np.pi, size=(B, sw.n_angles))
    psi = torch.as_tensor(3.0 * haar_states(rng, sw.n_in, B), dtype=sw.dtype, device="cuda")
    want, _, wlp = sw.forward(ang, psi, logprob=True)
    got, st, lp = sw.forward(ang, psi, logprob=True, out=psi)
    assert (st == 0).all()
    assert torch.equal(got, want) and torch.equal(lp, wlp)


@pytest.mark.parametrize("rows,B", [(8, 2435), (9, 1219)])
def test_half_window_kernel(rows, B):
    _check(C.grid_cluster(rows, 4), B)


@pytest.mark.parametrize("kw", [{}, dict(dtype=torch.complex128), dict(extended_planes=True)])
@pytest.mark.parametrize("rows,B", [(1, 3), (2, 5000), (4, 700), (7, 300), (8, 20), (9, 20)])
def test_register_kernel(rows, B, kw):
    circ = C.grid_cluster(rows, 4)
    if "extended_planes" in kw:
        circ[1] = C.Ment("XZ")
    _check(circ, B, **kw)


@pytest.mark.parametrize("rows,B", [(10, 20), (17, 2)])  # on chip; streamed
def test_wide_kernels(rows, B):
    _check(C.many_wires([3] * rows), B)
