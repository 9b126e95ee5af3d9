"""A Z measurement recorded as prob1 / (prob0 + prob1) on a matrix of trace zero has
no value (0 / 0): NaN, in every kernel (warp and block groups, clusters, the full
matrix), as numpy's division gives."""
import numpy as np
import pytest
import torch

from mentpy_gb300 import circuit as C
from mentpy_gb300.dm import DensityMatrixSweep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,full", [(1, False), (3, False), (6, False), (6, True), (7, False), (8, False),
                                       (9, False), (10, False)])
def test_expectation_of_a_zero_matrix_is_nan(rows, full):
    circ = C.many_wires([3] * rows)
    circ[0] = C.Ment("Z")
    sw = DensityMatrixSweep(circ)
    assert sw.plan.schedule_measure[0] == 0 and sw.plan.window == rows + 1
    psi = np.zeros((2, 2 ** rows))
    psi[1, 0] = 1.0  # run 1: node 0 in |0>
    _, outc, st, probs = sw.forward(np.zeros((2, sw.n_angles)), psi, mode="expectation", want_probs=True,
                                    full_matrix=full)
    probs = probs.cpu().numpy()
    assert (outc[:, 0] == 2).all()
    assert np.isnan(probs[0, 0])
    # run 1: 1 - prob0 / trace, each a float32 sum of at most 2^10 terms in float pairs
    assert abs(probs[1, 0]) < 1e-6 and int(st[1]) == 0
