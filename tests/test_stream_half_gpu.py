"""Wide sweep, windows 11 and up, where half the window is kept: on chip (the
default up to window 17) and in streamed passes (the bulk-copy staging, XZ / YZ
planes, wider windows).  Steps on the stored half's bits at every offset (short
and long wires, uneven ones with steps that no qubit enters, more steps than the
window), outputs on rotated bits; on chip every number of blocks a run (1, 2, 4
and 8, by window and batch) and every slice size; against the complex128 oracle
at the amplitude bound of the other streamed tests."""
import numpy as np
import pytest
import torch

from helpers import haar_states
from mentpy_gb300 import circuit as C
from mentpy_gb300.sweep import StatevectorSweep
from oracle import sweep as oracle

pytestmark = pytest.mark.gpu

TOL_AMP_C64 = 2e-5


def _planes(circ, rng):
    nodes = list(circ.trainable_nodes)
    for n in rng.choice(nodes, len(nodes) // 3, replace=False):
        circ[int(n)] = C.Ment(str(rng.choice(["XZ", "YZ"])))
    return circ


CASES = [  # circuit, runs, general planes
    (lambda r: C.many_wires([4] * 10), 3, False),               # w = 11: the half is one tile
    (lambda r: C.grid_cluster(11, 3), 2, False),
    (lambda r: C.many_wires([5, 2, 3] * 4), 5, False),          # uneven wires
    (lambda r: C.many_wires([7, 6, 5, 4, 3, 2] * 2), 3, False),
    (lambda r: C.grid_cluster(13, 5), 2, False),
    (lambda r: C.many_wires([2, 3] * 8), 2, False),             # w = 17, eight blocks a run on chip
    (lambda r: C.grid_cluster(16, 3), 20, False),               # w = 17, four
    (lambda r: C.grid_cluster(15, 3), 3, False),                # w = 16, four
    (lambda r: C.many_wires([3] * 15), 40, False),              # w = 16, two
    (lambda r: C.grid_cluster(14, 4), 5, False),                # w = 15, two
    (lambda r: C.many_wires([3] * 14), 80, False),              # w = 15, one
    (lambda r: C.grid_cluster(11, 12), 2, False),               # w = 12, many cycles
    (lambda r: C.many_wires([3] * 17), 1, False),               # w = 18: streamed
    (lambda r: _planes(C.grid_cluster(10, 4), r), 3, True),
    (lambda r: _planes(C.many_wires([4] * 12), r), 2, True),
]


@pytest.mark.parametrize("tma", [False, True])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_half_window_against_oracle(case, tma):
    rng = np.random.default_rng(400 + case)
    build, B, gen = CASES[case]
    circ = build(rng)
    sw = StatevectorSweep(circ, extended_planes=gen)
    assert sw.plan.window >= 11
    ang = rng.uniform(0, 2 * np.pi, size=(B, sw.n_angles))
    psi = haar_states(rng, sw.n_in, B)
    out, st, lp = sw.forward(ang, psi, stream_tma=tma, logprob=True)
    assert (st.cpu().numpy() == 0).all()
    out = out.cpu().numpy()
    r = B - 1
    ref, _, probs = oracle.run_sv(circ, ang[r], psi[r], output_form="sv")
    assert np.abs(out[r] - ref).max() < TOL_AMP_C64
    assert abs(float(lp[r]) - np.log(probs).sum()) < 1e-4


@pytest.mark.parametrize("build", [lambda: C.grid_cluster(10, 3), lambda: C.grid_cluster(15, 3)])
def test_outputs_on_the_inputs(build):
    """One buffer for inputs and outputs: the input (and its norm) is read first."""
    sw = StatevectorSweep(build())
    rng = np.random.default_rng(499)
    B = 20
    ang = rng.uniform(0, 2 * np.pi, size=(B, sw.n_angles))
    psi = torch.as_tensor(3.0 * haar_states(rng, sw.n_in, B), dtype=torch.complex64, device="cuda")
    want, _, wlp = sw.forward(ang, psi, logprob=True)
    got, st, lp = sw.forward(ang, psi, logprob=True, out=psi)
    assert (st == 0).all()
    assert torch.equal(got, want) and torch.equal(lp, wlp)
