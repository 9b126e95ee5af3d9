"""Which windows' density-matrix adjoint keeps the factored matrix: 5 to 7 (below, the
full matrix is small and faster).  The workspace tells: a step of a run saves 2 * 4^w
bytes factored, 8 * 4^w as the full matrix."""
import ctypes

import pytest

from mentpy_gb300 import _native
from mentpy_gb300 import circuit as C
from mentpy_gb300.dm import DensityMatrixSweep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,groups,factored", [(2, 8, False), (3, 8, False), (4, 2, True), (5, 1, True),
                                                  (6, 1, True), (7, 1, False)])
def test_route_by_window(rows, groups, factored):
    sw = DensityMatrixSweep(C.grid_cluster(rows, 4))
    w, m, n = sw.plan.window, sw.plan.n_steps, ctypes.c_size_t()
    assert w == rows + 1
    _native.check(_native.lib().mbqc_dm_adjoint_workspace(sw.dplan.handle, 1, w, None, ctypes.byref(n)))
    steps = m + (1 if w > 7 else 0)  # above window 7 the matrix itself is in the workspace
    assert n.value == groups * steps * (2 if factored else 8) * 4 ** w
