"""Register sweep with one run a warp (lane variant 5), several warps a block and an
odd number of staged steps: every warp's row staging is 16-byte aligned (its rows are
copied 16 bytes at a time).  Against the kernel with the fewest lanes a run, at the
bound of the other variant comparisons (complex64, another order of the norm's sum)."""
import numpy as np
import pytest
import torch

from helpers import haar_states
from mentpy_gb300 import circuit as C
from mentpy_gb300.sweep import StatevectorSweep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(4, 4), (6, 4), (6, 6), (8, 4), (8, 6), (8, 8)])
def test_one_run_a_warp_odd_steps(rows, cols):
    sw = StatevectorSweep(C.many_wires([cols] * rows))
    rng = np.random.default_rng(rows * 100 + cols)
    B = 1788
    ang = rng.uniform(0, 2 * np.pi, size=(B, sw.n_angles))
    psi = haar_states(rng, sw.n_in, B)
    a, sa, _ = sw.forward(ang, psi, variant=5)
    b, sb, _ = sw.forward(ang, psi, variant=4)
    assert (sa == 0).all() and (sb == 0).all()
    assert (a - b).abs().max().item() < 1e-5
    assert torch.isfinite(a.real).all()
