"""``run`` takes one value for every trainable node: arrays of the right length whose
rows hold none or several are refused before anything reaches the bound buffers (no
GPU: the sweep is a stand-in)."""
from types import SimpleNamespace

import numpy as np
import pytest

from mentpy_gb300 import circuit as C
from mentpy_gb300.simulators import CudaSimulatorSV


@pytest.mark.parametrize("shape,ok", [((3, 0), False), ((3, 2), False), ((3, 1), True), ((3,), True)])
def test_angle_arrays(shape, ok):
    sim = CudaSimulatorSV.__new__(CudaSimulatorSV)
    sim._mbqcirc, sim._input_state, sim.current_measurement = C.linear_cluster(4), None, 0
    sim.schedule_measure, sim.plan = [0, 1, 2], SimpleNamespace(outcome_nodes=lambda: [0, 1, 2])
    sim._sweep = SimpleNamespace(n_angles=3)
    seen = []
    sim._run_one = lambda ang: seen.append(ang.reshape(-1).tolist()) or (np.ones(2, complex), 0)
    if ok:
        sim.run(np.ones(shape), output_form="sv")
        assert seen == [[1.0, 1.0, 1.0]]
    else:
        with pytest.raises(ValueError, match="does not match number of trainable nodes"):
            sim.run(np.ones(shape))
        assert not seen
