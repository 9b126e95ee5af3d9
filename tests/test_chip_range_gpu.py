"""The on-chip wide sweep on inputs of a large norm: the scale follows from norms whose
total over a block or a cluster may exceed a float while every warp's part fits.  A
power of two on the input changes no bit of the state; the log-probability is made in
FP64 from logarithms that move by k ln 2 (a few ulps of ~100: 1e-12)."""
import numpy as np
import pytest
import torch

from helpers import haar_states
from mentpy_gb300 import circuit as C
from mentpy_gb300.sweep import StatevectorSweep

pytestmark = pytest.mark.gpu


# squared norm 1.25^2 2^(2 k); after five steps the half window holds 2^6 times that in 2^(w - 11) warps
@pytest.mark.parametrize("rows,B,k", [
    (16, 2, 61), (16, 20, 61),  # w = 17, eight and four blocks: the total beyond a float
    (16, 2, 62), (15, 3, 62), (15, 40, 62), (14, 80, 61), (12, 5, 60), (10, 4, 57),
])
def test_large_norms_keep_the_bits(rows, B, k):
    sw = StatevectorSweep(C.many_wires([5] * rows))
    rng = np.random.default_rng(17)
    ang = rng.uniform(0, 2 * np.pi, size=(B, sw.n_angles))
    psi = torch.as_tensor(1.25 * haar_states(rng, rows, B), dtype=torch.complex64, device="cuda")
    want, st, wlp = sw.forward(ang, psi, logprob=True)
    assert (st == 0).all()
    got, st, lp = sw.forward(ang, psi * 2.0**k, logprob=True)
    assert (st == 0).all()
    assert torch.equal(got, want)
    assert (lp - wlp).abs().max().item() < 1e-12
