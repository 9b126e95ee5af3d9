"""Streamed sweep, windows 11 and up, where the workspace keeps half the window:
steps on the stored half's bits at every offset (short and long wires, uneven
ones with steps that no qubit enters, more steps than the window), outputs on
rotated bits, XZ / YZ planes, both staging paths; against the complex128 oracle
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
    (lambda r: C.many_wires([2, 3] * 8), 2, False),             # w = 17
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
    out, st, _ = sw.forward(ang, psi, stream_tma=tma)
    assert (st.cpu().numpy() == 0).all()
    out = out.cpu().numpy()
    r = B - 1
    ref, _, _ = oracle.run_sv(circ, ang[r], psi[r], output_form="sv")
    assert np.abs(out[r] - ref).max() < TOL_AMP_C64
