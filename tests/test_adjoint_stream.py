"""``StatevectorSweep.adjoint`` on a stream of the caller's: what the current stream
does to the operands and to the memory of the results comes before the kernel."""
import ctypes
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from mentpy_gb300 import _native, sweep
from mentpy_gb300 import circuit as C
from mentpy_gb300.plan import compile_plan
from mentpy_gb300.sweep import StatevectorSweep


def _bare_sweep(circ):
    """A sweep on CPU tensors whose C calls are fakes."""
    sw = StatevectorSweep.__new__(StatevectorSweep)
    sw.circuit, sw.plan = circ, compile_plan(circ, "sv")
    sw.dtype, sw.device = torch.complex64, torch.device("cpu")
    sw.dplan = SimpleNamespace(handle=ctypes.c_void_p(0))
    sw.n_in, sw.n_out, sw.n_angles = sw.plan.n_in, sw.plan.n_out, sw.plan.n_angles
    return sw


@pytest.mark.parametrize("rows", [2, 8])  # a register window, a block-per-run one
@pytest.mark.parametrize("inputs", [None, "complex128"])
def test_the_stream_waits_for_the_current_one_before_the_launch(monkeypatch, rows, inputs):
    log = []

    def workspace(handle, runs, f64, n):
        n._obj.value = 64
        return 0

    kept, args = [], []
    monkeypatch.setattr(_native, "lib", lambda: SimpleNamespace(
        mbqc_sv_adjoint_workspace=workspace, mbqc_sv_adjoint=lambda *a: log.append("launch") or args.extend(a) or 0))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: "current")
    for name in ("as_device", "torch.empty", "torch.zeros"):  # work and memory of the current stream
        owner, attr = (torch, name[6:]) if name.startswith("torch.") else (sweep, name)
        real = getattr(owner, attr)
        monkeypatch.setattr(owner, attr, lambda *a, _real=real, **k: log.append("made") or _real(*a, **k))
    monkeypatch.setattr(sweep, "_keep_for", lambda s, *ts: kept.extend(t.data_ptr() for t in ts))
    sw = _bare_sweep(C.many_wires([4] * rows))
    B, d = 3, 2 ** sw.n_in
    psi = None if inputs is None else torch.ones(B, d, dtype=torch.complex128)
    g = torch.ones(B, 2 ** sw.n_out, dtype=torch.complex128)
    side = SimpleNamespace(cuda_stream=7, wait_stream=lambda s: log.append("wait " + s))
    sw.adjoint(torch.zeros(B, sw.n_angles, dtype=torch.float32), psi, g, stream=side)
    assert log[-2:] == ["wait current", "launch"] and log.count("wait current") == 1
    ptrs = [args[i].value for i in (2, 4, 6, 7, 9)]  # angles, inputs, grad_out, gradient, workspace
    assert sorted(kept) == sorted(ptrs)  # the allocator keeps them for the launch's stream


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [2, 8])
def test_operands_made_late_on_the_current_stream(rows):
    sw = StatevectorSweep(C.many_wires([4] * rows))
    rng = np.random.default_rng(31)
    B, d = 50, 2 ** sw.n_out
    ang = torch.as_tensor(rng.uniform(0, 6, (B, sw.n_angles)), dtype=torch.float32, device="cuda")
    g0 = torch.as_tensor(rng.standard_normal((B, d)) + 1j * rng.standard_normal((B, d)), device="cuda")
    want = sw.adjoint(ang, None, 2.0 * g0)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    sweep.gpu_hold(20000.0)  # the conversions, the default input and 2 g0 come after this
    got = sw.adjoint(ang, None, 2.0 * g0, stream=side)
    torch.cuda.current_stream().wait_stream(side)
    assert torch.equal(got, want)
