"""``StatevectorSweep.tune`` at windows 9 and 10: the default rule is timed beside the
lane counts, so that a batch whose default kernel has none keeps it."""
import numpy as np
import pytest
import torch

from helpers import haar_states
from mentpy_gb300 import circuit as C
from mentpy_gb300 import sweep
from mentpy_gb300.plan import compile_plan
from mentpy_gb300.sweep import StatevectorSweep


@pytest.mark.parametrize("rows,cost,want", [
    (8, {-1: 70, 4: 5000, 5: 110}, -1),   # an earlier choice (4) must not stand in for the default
    (9, {-1: 80, 5: 70}, 5),
    (3, {0: 30, 1: 20, 2: 25, 3: 40, 4: 50}, 1),
])
def test_the_default_is_a_candidate(monkeypatch, rows, cost, want):
    clock = [0.0]

    class Event:
        def __init__(self, enable_timing=False):
            self.at = 0.0

        def record(self, stream=None):
            self.at = clock[0]

        def elapsed_time(self, other):
            return other.at - self.at

    sw = StatevectorSweep.__new__(StatevectorSweep)
    sw.plan = compile_plan(C.many_wires([4] * rows), "sv")
    sw.dtype, sw.device = torch.complex64, torch.device("cpu")
    sw.n_in, sw.n_out, sw.n_angles = sw.plan.n_in, sw.plan.n_out, sw.plan.n_angles

    def forward(angles, inputs, *, variant, **kw):  # as _entry resolves the variant
        if variant == -1:
            variant = sweep._TUNED.get(sw._tune_key(len(angles)), -1)
        clock[0] += cost[variant]

    sw.forward = forward
    monkeypatch.setattr(sweep, "_TUNED", {sw._tune_key(100): max(cost)})
    monkeypatch.setattr(sweep, "gpu_hold", lambda us=0: None)
    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda device=None: None)
    assert sw.tune(torch.zeros(100, sw.n_angles, dtype=torch.float64)) == want
    assert sweep._TUNED == {sw._tune_key(100): want}


@pytest.mark.gpu
def test_a_tuned_large_batch_keeps_the_half_window_kernel(monkeypatch):
    """At 5,000 runs of grid 8 x 10 the default kernel takes two thirds of the time of
    any lane count."""
    monkeypatch.setattr(sweep, "_TUNED", {})
    sw = StatevectorSweep(C.grid_cluster(8, 10))
    rng = np.random.default_rng(23)
    ang = torch.as_tensor(rng.uniform(0, 6, (5000, sw.n_angles)), device="cuda")
    psi = torch.as_tensor(haar_states(rng, 8, 5000), dtype=torch.complex64, device="cuda")
    assert sw.tune(ang, psi) == -1
