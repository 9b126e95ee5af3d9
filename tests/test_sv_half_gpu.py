"""Windows 9 and 10 in large batches (half the window kept, several runs a warp):
ragged batches, uneven wires with steps that no qubit enters, step counts around a
cycle, one broadcast input; against the register kernel's lane variant on the same
batch.  Amplitudes differ by the phase product's order alone (products of up to 72
unit factors in float32: 72 * 1.2e-7 / sqrt(72) ~ 1e-6 at most), log-probabilities
are the same numbers."""
import numpy as np
import pytest
import torch

from helpers import haar_states
from mentpy_gb300 import circuit as C
from mentpy_gb300.sweep import StatevectorSweep

pytestmark = pytest.mark.gpu

CASES = [  # circuit, runs, lane variant of the default kernel
    (lambda: C.grid_cluster(8, 3), 2501, 4),
    (lambda: C.grid_cluster(8, 10), 2433, 4),
    (lambda: C.many_wires([3] + [2] * 7), 2600, 4),     # nine steps: one past a cycle
    (lambda: C.many_wires([5, 2, 3, 4, 2, 3, 2, 6]), 2999, 4),
    (lambda: C.grid_cluster(9, 4), 1301, 5),
    (lambda: C.many_wires([3] * 9), 1500, 5),
    (lambda: C.many_wires([6, 2, 3, 4, 2, 3, 2, 5, 3]), 1217, 5),
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_large_batch_against_register_kernel(case):
    build, B, ll = CASES[case]
    sw = StatevectorSweep(build())
    assert sw.plan.window in (9, 10)
    rng = np.random.default_rng(500 + case)
    ang = rng.uniform(0, 2 * np.pi, size=(B, sw.n_angles))
    psi = haar_states(rng, sw.n_in, 1)[0] if case % 3 == 1 else haar_states(rng, sw.n_in, B)
    a, sa, la = sw.forward(ang, psi, logprob=True)
    b, sb, lb = sw.forward(ang, psi, logprob=True, variant=ll)
    assert (sa == 0).all() and (sb == 0).all()
    assert (a - b).abs().max().item() < 2e-6
    assert torch.equal(la, lb)
    a, _, _ = sw.forward(ang, psi, ref_phase=False)
    b, _, _ = sw.forward(ang, psi, variant=ll, ref_phase=False)
    assert torch.equal(a, b)
