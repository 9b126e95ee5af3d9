"""Batched GPU sweeps: thousands of runs of one circuit per launch.

``StatevectorSweep(circuit).forward(angles[B, A], inputs[B or 1, 2^n_in])``
runs B independent copies of mentpy's statevector sweep
(np_simulator_sv.py:227-297) in one kernel launch and returns the normalised
output states in the reference's output qubit order.  Buffers live in torch
tensors (device memory and the current stream); the arithmetic is the CUDA
library's.
"""
from __future__ import annotations

import ctypes
from typing import Optional

import numpy as np
import torch

from . import _native
from .plan import PLANE_CODES, WindowPlan, compile_plan


_TUNED = {}  # (window, steps, n_in, n_out, batch bucket) -> fastest register-kernel variant

REGISTER_MAX_WINDOW = 10  # register-resident kernel; wider windows stream through a workspace
STREAMED = 99             # ``variant`` value forcing the streamed kernel (windows >= 8)


def gpu_hold(us: float = 2000.0) -> None:
    """Keep the current stream busy for about ``us`` microseconds so that the
    launches the host enqueues next are queued ahead of the device: CUDA-event
    intervals around them then measure device time only, not host submission
    gaps."""
    torch.cuda._sleep(int(us * 2000))  # ~2 GHz cycles


def _stream_ptr(stream: Optional[torch.cuda.Stream]) -> ctypes.c_void_p:
    if stream is not None:
        return ctypes.c_void_p(stream.cuda_stream)
    # the current stream's handle without building a Stream object (~3 us)
    return ctypes.c_void_p(torch._C._cuda_getCurrentRawStream(torch.cuda.current_device()))


def _ptr(t: Optional[torch.Tensor]) -> ctypes.c_void_p:
    return ctypes.c_void_p(0 if t is None else t.data_ptr())


def mapped_ptr(t: torch.Tensor) -> ctypes.c_void_p:
    """Device address of a pinned (page-locked) CPU tensor, which the kernels
    then read or write in place over the CPU-GPU link (no staging copy).
    Raises for pageable or non-contiguous tensors."""
    if t.device.type != "cpu" or not t.is_pinned():
        raise ValueError("mapped host buffers must be pinned CPU tensors (tensor.pin_memory())")
    if not t.is_contiguous():
        raise ValueError("mapped host buffers must be contiguous")
    out = ctypes.c_void_p()
    _native.check(_native.lib().mbqc_mapped_pointer(ctypes.c_void_p(t.data_ptr()), ctypes.byref(out)))
    return out


def _keep_for(stream, *tensors) -> None:
    """Memory of the current stream that a kernel on ``stream`` uses: not handed
    out again before that kernel is done."""
    for t in tensors:
        if t.is_cuda:
            t.record_stream(stream)


def _mapped_or_device(x, dtype, device, what: str) -> torch.Tensor:
    """``x`` itself when it is a pinned CPU tensor of ``dtype`` (accessed in
    place), else the usual device copy."""
    if isinstance(x, torch.Tensor) and x.device.type == "cpu":
        if x.dtype != dtype or not x.is_pinned() or not x.is_contiguous():
            raise ValueError(f"mapped_host: {what} must be a contiguous pinned CPU tensor of {dtype}")
        return x
    return as_device(x, dtype, device)


def as_device(x, dtype, device) -> torch.Tensor:
    """A contiguous tensor on ``device`` whose memory holds exactly its values
    (lazy conjugate / negative views are materialised: the kernels read raw
    memory)."""
    if isinstance(x, torch.Tensor):
        if (x.dtype == dtype and x.device == device and x.is_contiguous() and not x.is_neg()
                and not (x.is_complex() and x.is_conj())):
            return x  # the usual case: nothing to convert
        t = x.to(device=device, dtype=dtype)
        if t.is_complex():
            t = t.resolve_conj()
        return t.resolve_neg().contiguous()
    return torch.as_tensor(np.asarray(x), dtype=dtype, device=device).contiguous()


class StatevectorSweep:
    """Batched statevector sweep of one circuit.

    ``dtype`` is ``torch.complex64`` (the fast path: complex64 amplitudes,
    FP64 norm reduction) or ``torch.complex128`` (FP64 check mode).
    ``extended_planes=True`` also accepts XZ and YZ measurements (forward
    sweeps; the adjoint and the drawn-outcome mode take XY, X and Y).
    """

    def __init__(self, circuit=None, window_size: int = 1, schedule=None, *,
                 plan: Optional[WindowPlan] = None, dtype=torch.complex64, device=None,
                 extended_planes: bool = False):
        if plan is None:
            plan = compile_plan(circuit, "sv", window_size=window_size, schedule=schedule,
                                extended_planes=extended_planes)
        if plan.kind != "sv":
            raise ValueError("StatevectorSweep needs a statevector plan")
        self.circuit = circuit
        self.plan = plan
        self.dtype = dtype
        self.device = torch.device(device) if device is not None else torch.device("cuda", torch.cuda.current_device())
        self.dplan = _native.DevicePlan(plan)
        self.n_in, self.n_out, self.n_angles = plan.n_in, plan.n_out, plan.n_angles

    def default_input(self) -> torch.Tensor:
        d = 2 ** self.n_in
        return torch.full((1, d), 1.0 / np.sqrt(d), dtype=self.dtype, device=self.device)

    def forward(self, angles, inputs=None, *, ref_phase: bool = True, variant: int = -1,
                out: Optional[torch.Tensor] = None, logprob: Optional[torch.Tensor] = None,
                status: Optional[torch.Tensor] = None, stream=None, mapped_host: bool = False,
                inputs_ready: bool = False, stream_tma: bool = False, _bind: bool = False):
        """Run the batch.  ``angles``: [B, A] (or [A]); ``inputs``: [B, 2^n_in],
        [2^n_in] or None (|+>^n_in).  Returns ``(states, status, logprob)``
        with ``states`` [B, 2^n_out]; ``logprob`` is None unless a buffer is
        passed or ``logprob=True``.

        ``mapped_host=True``: CPU tensors among ``angles``, ``inputs``,
        ``out``, ``status`` and ``logprob`` must be pinned and of the kernel's
        dtype; the kernel reads and writes them in place over the CPU-GPU link
        (no staging copies).  The call is asynchronous on the stream like any
        launch: synchronise before reading ``out`` on the host.

        ``inputs_ready=True`` declares that no earlier work on the stream
        writes ``angles`` or ``inputs`` (filled by the host, or before a
        loop of batches): the launch then reads them and runs its sweep while
        the previous launch finishes, waiting for it only before writing
        (register-resident kernel; ``MBQC_F_INPUTS_READY``).

        ``stream_tma=True`` stages the streamed kernel's tiles with TMA bulk
        copies instead of 16-byte asynchronous copies (same results; the
        default measured faster)."""
        if mapped_host:
            return self._forward_mapped(angles, inputs, ref_phase=ref_phase, variant=variant, out=out,
                                        logprob=logprob, status=status, stream=stream, inputs_ready=inputs_ready,
                                        _bind=_bind)
        ang = as_device(angles, torch.float64, self.device)
        if ang.dim() == 1:
            ang = ang.unsqueeze(0)
        B = ang.shape[0]
        if ang.shape[1] != self.n_angles:
            raise ValueError(
                f"Number of angles ({ang.shape[1]}) does not match number of trainable nodes ({self.n_angles})."
            )
        if inputs is None:
            inp = self.default_input()
        else:
            inp = as_device(inputs, self.dtype, self.device)
            if inp.dim() == 1:
                inp = inp.unsqueeze(0)
        if inp.shape[-1] != 2 ** self.n_in:
            raise ValueError(f"input states need {2 ** self.n_in} amplitudes, got {inp.shape[-1]}")
        if inp.shape[0] not in (1, B):
            raise ValueError("inputs must have one row or one row per angle vector")
        istride = 0 if inp.shape[0] == 1 else inp.shape[1]
        if out is None:
            out = torch.empty((B, 2 ** self.n_out), dtype=self.dtype, device=self.device)
        if status is None:
            status = torch.empty((B,), dtype=torch.int32, device=self.device)
        if logprob is True:
            logprob = torch.empty((B,), dtype=torch.float64, device=self.device)
        elif logprob is False:
            logprob = None
        flags = (_native.MBQC_F_REF_PHASE if ref_phase else 0) | (_native.MBQC_F_INPUTS_READY if inputs_ready else 0)
        if stream_tma:
            flags |= _native.MBQC_F_STREAM_TMA
        fn, args = self._entry(B, _ptr(ang), max(ang.shape[1], 1), _ptr(inp), istride, _ptr(out), flags, variant,
                               _ptr(logprob), _ptr(status))
        if _bind:
            return fn, args
        _native.check(fn(*args, _stream_ptr(stream)))
        return out, status, logprob

    __call__ = forward

    def _entry(self, B, ang, astride, inp, istride, out, flags, variant, logprob, status):
        """The C entry point for this batch and its arguments, all but the
        trailing stream (pointers as ctypes values)."""
        L = _native.lib()
        if variant == -1:
            variant = _TUNED.get(self._tune_key(B), -1)
        if self.dtype == torch.complex64 and (self.plan.window > REGISTER_MAX_WINDOW or variant == STREAMED):
            ws = self._stream_workspace(B)
            return L.mbqc_sv_forward_stream, (self.dplan.handle, B, ang, astride, inp, istride, out, flags, logprob,
                                              status, _ptr(ws), ws.numel())
        if self.dtype == torch.complex64:
            return L.mbqc_sv_forward, (self.dplan.handle, B, ang, astride, inp, istride, out, flags, variant, logprob,
                                       status)
        if self.dtype == torch.complex128:
            return L.mbqc_sv_forward_f64, (self.dplan.handle, B, ang, astride, inp, istride, out, flags, logprob,
                                           status)
        raise TypeError("dtype must be torch.complex64 or torch.complex128")

    def forward_sampled(self, angles, inputs=None, *, seed: Optional[int] = None, circuit=None, stream=None):
        """Runs with drawn outcomes and flow byproduct corrections (mentpy's
        PennyLane-backend semantics; the numpy simulators only force outcome
        0).  ``circuit``: the MBQCircuit of the plan (its flow gives the
        byproducts; defaults to the one this sweep was built from).  ``seed``
        default: a draw from numpy's global generator.  Returns ``(states
        [B, 2^n_out] normalised, global phase unspecified, outcomes [B, M]
        int8, status [B])``."""
        from .sampling import byproduct_tables

        circ = circuit if circuit is not None else self.circuit
        if circ is None:
            raise ValueError("forward_sampled needs the circuit (its flow gives the byproducts)")
        if self.dtype != torch.complex64:
            raise TypeError("sampled outcomes run in complex64")
        key = id(circ)
        tabs = getattr(self, "_byproducts", None)
        if tabs is None or tabs[0] != key:
            xs, zoff, zidx, xo, zo = byproduct_tables(circ, self.plan)
            dev = self.device
            zidx = zidx if zidx.size else np.zeros(1, dtype=np.int32)
            tabs = (key, torch.as_tensor(xs, device=dev), torch.as_tensor(zoff, device=dev),
                    torch.as_tensor(zidx, device=dev), torch.as_tensor(xo.view(np.int32), device=dev),
                    torch.as_tensor(zo.view(np.int32), device=dev))
            self._byproducts = tabs
        ang = as_device(angles, torch.float64, self.device)
        if ang.dim() == 1:
            ang = ang.unsqueeze(0)
        B = ang.shape[0]
        if ang.shape[1] != self.n_angles:
            raise ValueError(f"Number of angles ({ang.shape[1]}) does not match number of trainable nodes "
                             f"({self.n_angles}).")
        inp = self.default_input() if inputs is None else as_device(inputs, self.dtype, self.device)
        if inp.dim() == 1:
            inp = inp.unsqueeze(0)
        istride = 0 if inp.shape[0] == 1 else inp.shape[1]
        if seed is None:
            seed = int(np.random.randint(0, 2**63 - 1, dtype=np.int64))
        M = self.plan.n_steps
        out = torch.empty((B, 2 ** self.n_out), dtype=self.dtype, device=self.device)
        outc = torch.empty((B, max(M, 1)), dtype=torch.int8, device=self.device)
        status = torch.empty((B,), dtype=torch.int32, device=self.device)
        bp = _native.Byproducts(*(t.data_ptr() for t in tabs[1:]))
        L = _native.lib()
        nb = ctypes.c_size_t(0)
        _native.check(L.mbqc_sv_sampled_workspace(self.dplan.handle, B, ctypes.byref(nb)))
        ws = torch.empty((max(nb.value, 1),), dtype=torch.uint8, device=self.device) if nb.value else None
        _native.check(L.mbqc_sv_forward_sampled(
            self.dplan.handle, B, _ptr(ang), max(ang.shape[1], 1), _ptr(inp), istride, _ptr(out),
            int(seed) & (2**64 - 1), ctypes.byref(bp), _ptr(outc), max(M, 1), _ptr(status),
            _ptr(ws) if ws is not None else None, nb.value, _stream_ptr(stream)))
        return out, outc[:, :M], status

    def prepare(self, angles, inputs, out, *, status: Optional[torch.Tensor] = None,
                logprob: Optional[torch.Tensor] = None, mapped_host: bool = False, ref_phase: bool = True,
                variant: int = -1, inputs_ready: bool = False) -> "PreparedSweep":
        """Bind one batch's buffers: every call of the returned object
        launches the batch again on the current stream with no per-call
        argument handling (a pre-resolved C call, or a CUDA graph replay for
        the streamed kernel).  The caller refills ``angles`` / ``inputs``
        between calls and reads ``out`` after synchronising.  With
        ``mapped_host=True`` pinned CPU buffers are read and written in place
        (see ``forward``; also for ``inputs_ready``: a serving loop that
        refills the buffers on the host between calls can set it)."""
        return PreparedSweep(self, angles, inputs, out, status=status, logprob=logprob, mapped_host=mapped_host,
                             ref_phase=ref_phase, variant=variant, inputs_ready=inputs_ready)

    def _forward_mapped(self, angles, inputs, *, ref_phase, variant, out, logprob, status, stream,
                        inputs_ready=False, _bind=False):
        ang = _mapped_or_device(angles, torch.float64, self.device, "angles")
        if ang.dim() != 2 or ang.shape[1] != self.n_angles:
            raise ValueError(f"angles must have shape [B, {self.n_angles}]")
        B = ang.shape[0]
        inp = self.default_input() if inputs is None else _mapped_or_device(inputs, self.dtype, self.device, "inputs")
        if inp.dim() != 2 or inp.shape[1] != 2 ** self.n_in or inp.shape[0] not in (1, B):
            raise ValueError(f"inputs must have shape [B or 1, {2 ** self.n_in}]")
        istride = 0 if inp.shape[0] == 1 else inp.shape[1]
        if out is None:
            raise ValueError("mapped_host: pass ``out`` (a pinned CPU or a device tensor)")
        out = _mapped_or_device(out, self.dtype, self.device, "out")
        if tuple(out.shape) != (B, 2 ** self.n_out):
            raise ValueError(f"out must have shape {(B, 2 ** self.n_out)}")
        if status is None:
            status = torch.empty((B,), dtype=torch.int32, device=self.device)
        status = _mapped_or_device(status, torch.int32, self.device, "status")
        if logprob is not None:
            logprob = _mapped_or_device(logprob, torch.float64, self.device, "logprob")

        def p(t):
            if t is None:
                return ctypes.c_void_p(0)
            return mapped_ptr(t) if t.device.type == "cpu" else ctypes.c_void_p(t.data_ptr())

        flags = (_native.MBQC_F_REF_PHASE if ref_phase else 0) | (_native.MBQC_F_INPUTS_READY if inputs_ready else 0)
        if ang.device.type == "cpu" or inp.device.type == "cpu":
            flags |= _native.MBQC_F_HOST_INPUTS
        fn, args = self._entry(B, p(ang), max(ang.shape[1], 1), p(inp), istride, p(out), flags, variant, p(logprob),
                               p(status))
        if _bind:
            return fn, args
        _native.check(fn(*args, _stream_ptr(stream)))
        return out, status, logprob

    # ------------------------------------------------------------ autotuning
    def variants(self):
        """Register-kernel variants (log2 lanes per run) valid for this window;
        windows above 10 have the wide kernels only."""
        w = self.plan.window
        if w > REGISTER_MAX_WINDOW or self.dtype != torch.complex64:
            return []
        return list(range(max(0, w - 5), min(5, w) + 1))

    def tune(self, angles, inputs=None, reps: int = 5, stream=None, inputs_ready: bool = False) -> int:
        """Time every variant on this batch (CUDA events, back-to-back
        launches after a warm-up) and keep the fastest for batches of this
        size (power-of-two bucket).  At windows 9 and 10 the default (-1) is a
        candidate of its own: large batches take a kernel there that no lane
        count names (csrc/sv_half.cu).  ``inputs_ready`` times the launches in
        that mode (they overlap, which can favour another variant); the
        choice serves both modes, so the declaration never changes results.
        Returns the chosen variant; ``forward(variant=-1)`` uses it."""
        cand = self.variants()
        if not cand:
            return -1
        ang = as_device(angles, torch.float64, self.device)
        if ang.dim() == 1:
            ang = ang.unsqueeze(0)
        B = ang.shape[0]
        if self.plan.window >= 9:
            cand.append(-1)
            _TUNED.pop(self._tune_key(B), None)  # -1 is the default rule, not an earlier choice
        out = torch.empty((B, 2 ** self.n_out), dtype=self.dtype, device=self.device)
        st = torch.empty((B,), dtype=torch.int32, device=self.device)
        best, best_ms = -1, float("inf")
        kw = dict(out=out, status=st, stream=stream, inputs_ready=inputs_ready)
        for v in cand:
            for _ in range(2):
                self.forward(ang, inputs, variant=v, **kw)
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            gpu_hold()  # queue the timed launches ahead of the device: no host gaps in the interval
            e0.record()
            for _ in range(reps):
                self.forward(ang, inputs, variant=v, **kw)
            e1.record()
            torch.cuda.synchronize(self.device)
            ms = e0.elapsed_time(e1) / reps
            if ms < best_ms:
                best, best_ms = v, ms
        _TUNED[self._tune_key(B)] = best
        return best

    def _tune_key(self, batch: int):
        p = self.plan
        return (p.window, p.n_steps, p.n_in, p.n_out, max(int(batch), 1).bit_length())

    def _stream_workspace(self, runs: int) -> torch.Tensor:
        n = ctypes.c_size_t()
        _native.check(_native.lib().mbqc_sv_stream_workspace(self.dplan.handle, runs, ctypes.byref(n)))
        ws = getattr(self, "_sws", None)
        if ws is None or ws.numel() < n.value:
            ws = torch.empty(n.value, dtype=torch.uint8, device=self.device)
            self._sws = ws
        return ws

    # ------------------------------------------------------------ adjoint
    def _workspace(self, runs: int) -> torch.Tensor:
        need = getattr(self, "_ws_need", None)  # (runs, bytes) of the last call
        if need is None or need[0] != runs:
            f64 = 1 if self.dtype == torch.complex128 else 0
            n = ctypes.c_size_t()
            _native.check(_native.lib().mbqc_sv_adjoint_workspace(self.dplan.handle, runs, f64, ctypes.byref(n)))
            need = self._ws_need = (runs, n.value)
        ws = getattr(self, "_ws", None)
        if ws is None or ws.numel() < need[1]:
            ws = torch.empty(max(need[1], 16), dtype=torch.uint8, device=self.device)
            self._ws = ws
        return ws

    def _every_angle_written(self) -> bool:
        """Whether the adjoint writes the gradient of every angle: the register
        kernels (windows up to 8 in XY, X and Y) always do, the block-per-run
        kernels write the angles that some step uses."""
        v = getattr(self, "_all_written", None)
        if v is None:
            p = self.plan
            planes = np.asarray(p.step_plane)
            v = (p.window <= 8 and not (planes > PLANE_CODES["Y"]).any()) or (
                len(set(np.asarray(p.step_angle).tolist()) - {-1}) == self.n_angles)
            self._all_written = v
        return v

    def adjoint(self, angles, inputs, grad_out, *, status: Optional[torch.Tensor] = None, stream=None):
        """dL/dangles [B, A] (float64) for dL = Re sum conj(grad_out) dz, where
        z = forward(angles, inputs, ref_phase=False)."""
        ang = as_device(angles, torch.float64, self.device)
        if ang.dim() == 1:
            ang = ang.unsqueeze(0)
        B = ang.shape[0]
        inp = self.default_input() if inputs is None else as_device(inputs, self.dtype, self.device)
        if inp.dim() == 1:
            inp = inp.unsqueeze(0)
        istride = 0 if inp.shape[0] == 1 else inp.shape[1]
        g = as_device(grad_out, self.dtype, self.device)
        if g.shape != (B, 2 ** self.n_out):
            raise ValueError(f"grad_out must have shape {(B, 2 ** self.n_out)}")
        # an angle no step uses (a trainable node that is never measured) has
        # derivative 0: filled in where the kernel does not write it
        written = self._every_angle_written()
        make = torch.empty if written else torch.zeros
        grad = make((B, self.n_angles), dtype=torch.float64, device=self.device)
        if B == 0:
            return grad
        ws = self._workspace(B)
        if stream is not None:
            # what the current stream still does to the operands (the default
            # input's fill, conversions, the zeros, the caller's own work) and to
            # earlier owners of grad's and the workspace's memory comes before the kernel
            stream.wait_stream(torch.cuda.current_stream(self.device))
            _keep_for(stream, ang, inp, g, grad, ws)
        fn = _native.lib().mbqc_sv_adjoint if self.dtype == torch.complex64 else _native.lib().mbqc_sv_adjoint_f64
        _native.check(fn(self.dplan.handle, B, _ptr(ang), max(ang.shape[1], 1), _ptr(inp), istride, _ptr(g),
                         _ptr(grad), _ptr(status), _ptr(ws), ws.numel(), _stream_ptr(stream)))
        return grad

    def fidelity_grad(self, angles, inputs, targets, *, status: Optional[torch.Tensor] = None, stream=None,
                      loss: Optional[torch.Tensor] = None, grad: Optional[torch.Tensor] = None):
        """Loss 1 - mean_j |<t_j|z(angles_v, psi_j)>|^2 and its gradient for
        every angle vector v, all V x J runs in one launch.  Returns
        ``(loss [V], grad [V, A])`` in float64 (written into ``loss`` /
        ``grad`` when given)."""
        if self.dtype != torch.complex64:
            raise TypeError("fidelity_grad runs in complex64")
        ang = as_device(angles, torch.float64, self.device)
        if ang.dim() == 1:
            ang = ang.unsqueeze(0)
        V = ang.shape[0]
        inp = as_device(inputs, self.dtype, self.device)
        tg = as_device(targets, self.dtype, self.device)
        if inp.dim() == 1:
            inp = inp.unsqueeze(0)
        if tg.dim() == 1:
            tg = tg.unsqueeze(0)
        J = inp.shape[0]
        if tg.shape != (J, 2 ** self.n_out) or inp.shape[1] != 2 ** self.n_in:
            raise ValueError("inputs [J, 2^n_in] and targets [J, 2^n_out] expected")
        if loss is None:
            loss = torch.empty((V,), dtype=torch.float64, device=self.device)
        if grad is None:
            grad = torch.empty((V, self.n_angles), dtype=torch.float64, device=self.device)
        if loss.shape != (V,) or grad.shape != (V, self.n_angles) or not (loss.is_contiguous() and grad.is_contiguous()):
            raise ValueError("loss [V] and grad [V, A] contiguous float64 buffers expected")
        if V == 0:
            return loss, grad
        ws = self._workspace(V * J)
        _native.check(_native.lib().mbqc_sv_fidelity_grad(
            self.dplan.handle, V, _ptr(ang), max(ang.shape[1], 1), J, _ptr(inp), _ptr(tg), _ptr(loss), _ptr(grad),
            _ptr(status), _ptr(ws), ws.numel(), _stream_ptr(stream)))
        return loss, grad


class PreparedSweep:
    """A statevector batch bound to fixed buffers (``StatevectorSweep.prepare``).
    ``__call__`` launches it on the current stream and returns ``out``.

    A register-kernel batch is one launch: its C entry point and arguments
    are resolved once and each call makes only that call (a few microseconds
    of host work; consecutive launches on a stream overlap their prologues).
    A wide batch (one launch on chip, tens when streamed) is recorded into a
    CUDA graph and replayed.  Buffers that the sweep would first convert (another dtype or
    device, lazy conjugate views) are also handled by the graph, which then
    records the conversion too."""

    def __init__(self, sweep: StatevectorSweep, angles, inputs, out, *, status=None, logprob=None,
                 mapped_host=False, ref_phase=True, variant=-1, inputs_ready=False):
        dev = sweep.device
        if status is None:
            n = angles.shape[0] if isinstance(angles, torch.Tensor) and angles.dim() == 2 else 1
            status = torch.empty((n,), dtype=torch.int32, device=dev)
        if inputs is None:
            inputs = sweep.default_input()  # kept alive here: the bound call reads it
        if logprob is True:
            n = angles.shape[0] if isinstance(angles, torch.Tensor) and angles.dim() == 2 else 1
            logprob = torch.empty((n,), dtype=torch.float64, device=dev)
        self.sweep, self.angles, self.inputs, self.out = sweep, angles, inputs, out
        self.status, self.logprob = status, logprob
        kw = dict(out=out, status=status, logprob=logprob, ref_phase=ref_phase, variant=variant,
                  mapped_host=mapped_host, inputs_ready=inputs_ready)
        side = torch.cuda.Stream(device=dev)
        side.wait_stream(torch.cuda.current_stream(dev))
        with torch.cuda.stream(side):
            sweep.forward(angles, inputs, **kw)  # warm-up launch (and argument checks)
        torch.cuda.current_stream(dev).wait_stream(side)
        torch.cuda.synchronize(dev)
        self.graph = None
        self._fn = None

        def direct(t, dtype):
            if not isinstance(t, torch.Tensor) or t.dtype != dtype or not t.is_contiguous():
                return False
            if t.is_complex() and t.is_conj() or t.is_neg():
                return False
            return t.device == dev or (mapped_host and t.device.type == "cpu" and t.is_pinned())

        bound = all(direct(t, dt) for t, dt in ((angles, torch.float64), (inputs, sweep.dtype), (out, sweep.dtype),
                                                  (status, torch.int32)))
        bound = bound and (logprob is None or direct(logprob, torch.float64))
        if bound:
            fn, args = sweep.forward(angles, inputs, _bind=True, **kw)
            if fn.__name__ != "mbqc_sv_forward_stream":
                # the call bound on the C side: each launch passes two arguments
                L = _native.lib()
                f64 = fn.__name__ == "mbqc_sv_forward_f64"
                if f64:  # (plan, B, ang, astride, inp, istride, out, flags, logprob, status)
                    full = args[:8] + (-1,) + args[8:]
                else:
                    full = args
                handle = ctypes.c_void_p()
                _native.check(L.mbqc_sv_call_create(*full, 1 if f64 else 0, ctypes.byref(handle)))
                self._call, self._lib, self._dev = handle, L, dev
                self._fn = L.mbqc_sv_call_launch
                return
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph):
            sweep.forward(angles, inputs, **kw)

    def __del__(self):
        call = getattr(self, "_call", None)
        if call is not None and call.value:
            try:
                self._lib.mbqc_sv_call_destroy(call)
            except Exception:  # interpreter shutdown
                pass
            self._call = None

    def __call__(self, stream: Optional[torch.cuda.Stream] = None):
        """Launch on ``stream`` (default: the current stream).  Passing the
        stream saves the host the current-stream lookup and a stream context
        (together several microseconds a call, more than the launch)."""
        if self._fn is not None:
            s = stream if stream is not None else torch.cuda.current_stream(self._dev)
            rc = self._fn(self._call, s.cuda_stream)
            if rc:
                _native.check(rc)
        elif stream is None:
            self.graph.replay()
        else:
            with torch.cuda.stream(stream):
                self.graph.replay()
        return self.out


def outer(states: torch.Tensor, stream=None) -> torch.Tensor:
    """Density matrices psi psi^dagger of a batch of complex64 states
    (the default output form of np_simulator_sv.py:292-293)."""
    if states.dtype == torch.complex128:
        return torch.einsum("bi,bj->bij", states, states.conj())
    B, d = states.shape
    n = int(round(np.log2(d)))
    rho = torch.empty((B, d, d), dtype=states.dtype, device=states.device)
    _native.check(_native.lib().mbqc_outer(B, n, _ptr(states), _ptr(rho), _stream_ptr(stream)))
    return rho
