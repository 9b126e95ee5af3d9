"""Adjoint of windows 9..17 where its passes change form: two forward steps a
pass against one (an odd or an even number of steps, the run's last), the
measured bit on the pair's own bit (bit 0), inside a block's slice of the
window and on the bits that join two blocks' slices, the slice partly in
shared memory (windows 15 and up, shared by 1, 2 or 4 blocks), wires of uneven
length (steps that no qubit enters).  The gradient along a random direction
against the oracle's complex128 central difference (h = 1e-4).  The complex64
sweep's gradient entries are good to ~1e-6 of the gradient's norm, the
difference itself to h^2 / 6 ~ 2e-9 and 1e-16 / h: 2e-4 is the bound the other
adjoint tests use for the same comparison."""
import numpy as np
import pytest
import torch

from helpers import haar_states
from mentpy_gb300 import circuit as C
from mentpy_gb300.sweep import StatevectorSweep
from oracle import gradients as G

pytestmark = pytest.mark.gpu

CASES = [  # circuit, runs
    (lambda: C.grid_cluster(8, 3), 3),         # w = 9
    (lambda: C.many_wires([3] * 10), 5),       # w = 11
    (lambda: C.many_wires([5, 2, 3] * 4), 5),  # uneven
    (lambda: C.grid_cluster(13, 3), 2),        # w = 14: the widest window in shared memory alone
    (lambda: C.grid_cluster(14, 3), 3),        # w = 15: four blocks a run
    (lambda: C.many_wires([4] * 14), 70),      # w = 15: two, the slice all in shared memory
    (lambda: C.grid_cluster(14, 4), 160),      # w = 15: one block a run
    (lambda: C.many_wires([2, 3] * 8), 3),     # w = 17, uneven
    (lambda: C.grid_cluster(16, 3), 70),       # w = 17: two blocks a run
    (lambda: C.grid_cluster(17, 3), 2),        # w = 18
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_directional_derivative(case):
    circ, B = CASES[case][0](), CASES[case][1]
    sw = StatevectorSweep(circ)
    assert 9 <= sw.plan.window <= 18
    rng = np.random.default_rng(300 + case)
    ang = rng.uniform(0, 2 * np.pi, size=(B, sw.n_angles))
    inp = haar_states(rng, sw.n_in, 2)[np.arange(B) % 2]
    g = rng.standard_normal((2, 2**sw.n_out)) + 1j * rng.standard_normal((2, 2**sw.n_out))
    g = g[np.arange(B) % 2]
    st = torch.empty(B, dtype=torch.int32, device="cuda")
    grad = sw.adjoint(ang, inp, g, status=st).cpu().numpy()
    assert (st.cpu().numpy() == 0).all()
    h = 1e-4
    for r in {0, B - 1}:
        d = rng.standard_normal(sw.n_angles)
        d /= np.linalg.norm(d)
        f = lambda a: float(np.real(np.vdot(g[r], G.canonical_sv(circ, a, inp[r]))))  # noqa: E731
        fd = (f(ang[r] + h * d) - f(ang[r] - h * d)) / (2 * h)
        got = float(grad[r] @ d)
        assert abs(got - fd) < 2e-4 * (1 + np.abs(grad[r]).max()), (r, got, fd)
