"""``run`` on the drop-in statevector simulator: the pinned single-run path
gives the batched sweep's bits on every register window, and threads never
share a buffer set."""
import threading
import warnings

import numpy as np
import pytest
import torch

from helpers import haar_states
from mentpy_gb300 import circuit as C
from mentpy_gb300.simulators import CudaSimulatorSV, PatternSimulator
from mentpy_gb300.sweep import StatevectorSweep

pytestmark = pytest.mark.gpu


def _planes():
    c = C.grid_cluster(2, 4)
    c[1] = C.Ment("XZ")
    c[5] = C.Ment("YZ")
    return c


@pytest.mark.parametrize("build,kw", [
    (lambda: C.linear_cluster(9), {}), (lambda: C.grid_cluster(3, 4), {}), (lambda: C.many_wires([5] * 6), {}),
    (lambda: C.grid_cluster(9, 3), {}), (lambda: C.grid_cluster(10, 3), {}), (_planes, dict(extended_planes=True)),
    (lambda: C.linear_cluster(6), dict(dtype="complex128"))])
def test_run_gives_the_sweeps_bits(build, kw):
    circ = build()
    rng = np.random.default_rng(71)
    n = len(circ.input_nodes)
    ps = PatternSimulator(circ, **kw)
    sw = StatevectorSweep(circ, **{k: (torch.complex128 if v == "complex128" else v) for k, v in kw.items()})
    for psi in haar_states(rng, n, 3):
        ang = rng.uniform(-9, 9, len(circ.trainable_nodes))
        ps.reset(input_state=psi)
        got = ps.run(ang, output_form="sv")
        want = sw.forward(ang, psi)[0][0].cpu().numpy().astype(np.complex128)
        assert np.array_equal(got, want)
    with pytest.raises(ValueError, match="input states need"):
        sim = CudaSimulatorSV(circ, np.ones(2 ** n + 1), **kw)
        sim.run(ang)


def test_zero_norm_warns_and_the_next_run_is_clean():
    ps = PatternSimulator(C.linear_cluster(4))
    rng = np.random.default_rng(72)
    psi = haar_states(rng, 1, 1)[0]
    ps.reset(input_state=np.zeros(2))
    with pytest.warns(RuntimeWarning):
        assert np.isnan(ps.run([0.1, 0.2, 0.3], output_form="sv")).all()
    ps.reset(input_state=psi)
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        out = ps.run([0.1, 0.2, 0.3], output_form="sv")
    assert np.isfinite(out).all()


def test_threads_do_not_share_buffers():
    circ = C.many_wires([6] * 3)
    sim = CudaSimulatorSV(circ, haar_states(np.random.default_rng(73), 3, 1)[0])
    angs = np.random.default_rng(74).uniform(0, 6, size=(8, 40, len(circ.trainable_nodes)))
    want = [[sim._run_one(a)[0] for a in rows] for rows in angs]
    bad = []

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for a, w in zip(angs[i], want[i]):
                if not np.array_equal(sim._run_one(a)[0], w):
                    bad.append(i)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(8)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad and len(sim._single) <= sim._SINGLE_POOL
