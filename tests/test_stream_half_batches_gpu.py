"""Streamed sweeps on half of the window: taken from the batch on whose whole windows
have more than twelve tiles of 2^10 amplitudes an SM (XZ / YZ planes and the bulk-copy
staging at windows 11 to 17, general planes at any), whole windows below.  The
workspace tells the route; results on both sides of the line against the complex128
oracle at the bound of the other streamed tests."""
import ctypes

import numpy as np
import pytest
import torch

from helpers import haar_states
from mentpy_gb300 import _native
from mentpy_gb300 import circuit as C
from mentpy_gb300.sweep import StatevectorSweep
from oracle import sweep as oracle

pytestmark = pytest.mark.gpu

TOL_AMP_C64 = 2e-5


def _planes(circ):
    for i, n in enumerate(list(circ.trainable_nodes)[::3]):
        circ[int(n)] = C.Ment("XZ" if i % 2 else "YZ")
    return circ


def _line(w):
    """The first batch with half windows."""
    return 12 * torch.cuda.get_device_properties(0).multi_processor_count // 2 ** (w - 10) + 1


@pytest.mark.parametrize("build,gen", [
    (lambda: _planes(C.grid_cluster(10, 4)), True),
    (lambda: _planes(C.many_wires([4] * 12)), True),
    (lambda: _planes(C.many_wires([6, 2, 3, 4, 2, 3, 2, 5, 3, 2, 4, 3])), True),
    (lambda: C.many_wires([4] * 10), False),
    (lambda: C.grid_cluster(13, 5), False),
    (lambda: C.grid_cluster(16, 3), False),
])
def test_both_sides_of_the_line(build, gen):
    circ = build()
    sw = StatevectorSweep(circ, extended_planes=gen)
    w = sw.plan.window
    rng = np.random.default_rng(811)
    B = _line(w)
    ang = rng.uniform(0, 2 * np.pi, size=(B, sw.n_angles))
    psi = haar_states(rng, sw.n_in, B)
    for b in (B - 1, B):
        n = ctypes.c_size_t()
        _native.check(_native.lib().mbqc_sv_stream_workspace(sw.dplan.handle, b, ctypes.byref(n)))
        assert (n.value < b * 2 ** w * 8) == (b == B)  # half of the windows, or all of them
        out, st, lp = sw.forward(ang[:b], psi[:b], stream_tma=not gen, logprob=True)
        assert (st == 0).all()
        r = b - 1
        ref, _, probs = oracle.run_sv(circ, ang[r], psi[r], output_form="sv")
        assert np.abs(out[r].cpu().numpy() - ref).max() < TOL_AMP_C64
        assert abs(float(lp[r]) - np.log(probs).sum()) < 1e-4


def test_windows_above_the_chip_keep_half_at_any_batch():
    sw = StatevectorSweep(C.many_wires([3] * 17))
    n = ctypes.c_size_t()
    _native.check(_native.lib().mbqc_sv_stream_workspace(sw.dplan.handle, 1, ctypes.byref(n)))
    assert n.value < 2 ** 18 * 8
