"""Drop-in ``PatternSimulator`` with GPU backends ``cuda-sv`` and ``cuda-dm``.

Mirrors mentpy's simulator front-end (mentpy/simulators/pattern_simulator.py:19-88)
and the ``BaseSimulator`` contract (mentpy/simulators/base_simulator.py:13-101):
``PatternSimulator(circuit, input_state=None, backend=..., **kwargs)``, a
stateful simulator with ``run(angles, ...)``, ``reset(input_state=None)`` and
``outcomes``.  The constructor keyword arguments of the numpy simulators
(``window_size``, ``schedule``, ``force0``, ``dev_mode``, ``wires``) keep their
meaning and raise the same errors (np_simulator_sv.py:38-100).

``numpy-sv`` / ``numpy-dm`` delegate to an installed mentpy, so existing code
can switch backends by name.
"""
from __future__ import annotations

import abc
import collections
import ctypes
import warnings
from typing import List, NamedTuple, Optional

import numpy as np
import torch

from . import _native
from .plan import compile_plan
from .sweep import _TUNED, REGISTER_MAX_WINDOW, STREAMED, StatevectorSweep, mapped_ptr, outer


class BaseSimulator(abc.ABC):
    """Holds the circuit, the input state and the outcome record
    (base_simulator.py:13-101)."""

    def __init__(self, mbqcircuit, input_state: np.ndarray = None) -> None:
        self._mbqcirc = mbqcircuit
        self._input_state = input_state
        self._outcomes = {}

    @property
    def mbqcircuit(self):
        return self._mbqcirc

    @property
    def input_state(self):
        return self._input_state

    @input_state.setter
    def input_state(self, value):
        self._input_state = value

    @property
    def outcomes(self) -> dict:
        return self._outcomes

    @outcomes.setter
    def outcomes(self, value: dict):
        self._outcomes = value

    def __call__(self, angles, **kwargs):
        return self.run(angles, **kwargs)

    def __repr__(self) -> str:
        return f"{self.__class__.__name__} for {self.mbqcircuit}"

    @abc.abstractmethod
    def measure(self, angle: float, **kwargs):
        ...

    @abc.abstractmethod
    def run(self, angles: List[float], **kwargs):
        ...

    @abc.abstractmethod
    def reset(self, input_state=None):
        ...


def _pop_kwargs(kwargs):
    return dict(
        window_size=kwargs.pop("window_size", 1),
        schedule=kwargs.pop("schedule", None),
        force0=kwargs.pop("force0", True),
        dev_mode=kwargs.pop("dev_mode", False),
        wires=kwargs.pop("wires", None),
        dtype=kwargs.pop("dtype", "complex64"),
        device=kwargs.pop("device", None),
        extended_planes=kwargs.pop("extended_planes", False),
    )


_DTYPES = {"complex64": torch.complex64, "complex128": torch.complex128,
           torch.complex64: torch.complex64, torch.complex128: torch.complex128}


class BatchResult(NamedTuple):
    """Result of ``run_batch``: ``states`` [B, 2^n_out] (statevector) or
    [B, d, d] (density matrix), ``outcomes`` [B, M] int8 in schedule order
    (the order of ``schedule_measure``), ``status`` [B] int32 (``RUN_OK`` = 0),
    ``logprob`` [B] float64 (statevector: ln of the all-zero branch
    probability) or ``probs`` [B, M] float64 (density matrix: prob0 of every
    step)."""
    states: object
    outcomes: object
    status: object
    logprob: object = None


def _is_tensor_batch(*xs) -> bool:
    return any(isinstance(x, torch.Tensor) for x in xs)


def _pinned(t) -> bool:
    return isinstance(t, torch.Tensor) and t.device.type == "cpu" and t.is_pinned()


def _bind_key(*xs):
    """Identity of a run_batch buffer set: memory, shape, strides and type of
    each tensor (views of the same memory give the same key), other
    arguments as they are."""
    return tuple((x.data_ptr(), tuple(x.shape), tuple(x.stride()), x.dtype, x.device.type)
                 if isinstance(x, torch.Tensor) else x for x in xs)


class _SingleRun:
    """Pinned host buffers of one ``run`` call and the C call bound to them: the
    kernel reads the angles and the input state and writes the output state and
    status in place over the CPU-GPU link, so a run is one launch and one wait
    (a device copy of each operand, the usual way for arrays, is a
    synchronising transfer apiece: 156 us a run of a nine-qubit wire against
    29 us)."""

    def __init__(self, sweep: StatevectorSweep, variant: int):
        def pinned(n, dtype):
            return torch.empty((1, n), dtype=dtype, pin_memory=True)

        self.variant = variant
        self._tensors = (pinned(max(sweep.n_angles, 1), torch.float64), pinned(2 ** sweep.n_in, torch.complex64),
                         pinned(2 ** sweep.n_out, torch.complex64), pinned(1, torch.int32))
        self.angles, self.inputs, self.out, self.status = (t.numpy()[0] for t in self._tensors)
        ang, inp, out, st = (mapped_ptr(t) for t in self._tensors)
        self._lib = _native.lib()
        self._call = ctypes.c_void_p()
        _native.check(self._lib.mbqc_sv_call_create(
            sweep.dplan.handle, 1, ang, self.angles.size, inp, self.inputs.size, out,
            _native.MBQC_F_REF_PHASE | _native.MBQC_F_HOST_INPUTS, variant, ctypes.c_void_p(0), st, 0,
            ctypes.byref(self._call)))
        self._dplan = sweep.dplan  # the call refers to the plan

    def __del__(self):
        call = getattr(self, "_call", None)
        if call is not None and call.value:
            try:
                self._lib.mbqc_sv_call_destroy(call)
            except Exception:  # interpreter shutdown
                pass
            self._call = None

    def __call__(self, angles, inp):
        """One run: the output state (complex128 copy) and the status word."""
        self.angles[: len(angles)] = angles
        self.inputs[:] = inp
        stream = torch.cuda.current_stream()
        rc = self._lib.mbqc_sv_call_launch(self._call, stream.cuda_stream)
        if rc:
            _native.check(rc)
        stream.synchronize()
        return self.out.astype(np.complex128), int(self.status[0])


class CudaSimulatorSV(BaseSimulator):
    """GPU statevector simulator: one kernel launch per ``run``.

    Same contract as ``NumpySimulatorSV`` (np_simulator_sv.py:35-384):
    ``run(angles, output_form="dm"|"sv", input_state=None)``; outcomes are all
    0 (force0); a second ``run`` without ``reset`` raises like the reference.
    Extra keywords ``dtype``: ``"complex64"`` (default) or ``"complex128"``;
    ``extended_planes``: also accept XZ / YZ measurements, which the
    reference statevector simulator rejects (default False: the same
    ValueError as the reference).
    """

    def __init__(self, mbqcircuit, input_state: np.ndarray = None, **kwargs) -> None:
        super().__init__(mbqcircuit, input_state)
        o = _pop_kwargs(kwargs)
        self.force0 = o["force0"]
        self.dev_mode = o["dev_mode"]
        self.wires = o["wires"]
        self.plan = compile_plan(mbqcircuit, "sv", window_size=o["window_size"], schedule=o["schedule"],
                                 force0=o["force0"], dev_mode=o["dev_mode"], extended_planes=o["extended_planes"])
        self.window_size = self.plan.window
        self.schedule = self.plan.schedule
        self.schedule_measure = self.plan.schedule_measure
        self._sweep = StatevectorSweep(plan=self.plan, dtype=_DTYPES[o["dtype"]], device=o["device"])
        self.current_measurement = 0
        self._qstate = None

    @property
    def qstate(self):
        return self._qstate

    def reset(self, input_state: np.ndarray = None):
        self.current_measurement = 0
        if input_state is not None:
            self.input_state = input_state
            self.__dict__.pop("_inp_t", None)
        self.outcomes = {}

    def measure(self, angle: float, **kwargs):
        raise NotImplementedError(
            "the GPU backend executes whole sweeps; call run(angles) instead of measure()"
        )

    _PREPARED_CACHE = 16  # bound buffer sets kept by run_batch

    def run_batch(self, angles, input_states=None, *, output_form: str = "sv", out=None, status=None,
                  logprob=None, stream=None, inputs_ready: bool = False, variant: int = -1) -> BatchResult:
        """B independent runs in one launch: ``angles`` [B, A] (or [A]),
        ``input_states`` [B or 1, 2^n_in], [2^n_in] or None (this
        simulator's input state).  No counterpart in the reference, whose
        ``run`` takes one angle vector (np_simulator_sv.py:227-297); each row
        gives what ``reset(input_state=row)`` + ``run(row angles,
        output_form)`` gives, and the simulator's own state (``reset`` /
        ``run`` cycle, ``outcomes``) is left untouched.

        numpy inputs give numpy results (complex128 states, copied to the
        host).  torch tensors give torch results without host copies: device
        tensors, or page-locked CPU tensors (``tensor.pin_memory()``) that the
        kernel reads and writes in place over the CPU-GPU link.  Passing
        ``out`` and ``status`` buffers (``out`` [B, 2^n_out] complex64,
        ``status`` [B] int32, optional ``logprob`` [B] float64) makes the call
        reusable: the first call with a buffer set binds it, later calls with
        the same tensors only launch (a few microseconds of host time; the
        call is asynchronous on ``stream``, synchronise before reading).  A
        bound set keeps the buffers' addresses: do not ``resize_`` or
        ``set_`` those tensors while they are in use.  Up to 16 bound sets are
        kept (least recently bound dropped first); ``release_buffers()``
        drops them all.
        ``inputs_ready``: the caller guarantees that no earlier work on the
        stream writes this call's angles or inputs (host-filled buffers), so
        consecutive calls overlap (``StatevectorSweep.forward``).  ``variant``:
        lanes per run (log2) of the register kernel, -1 for the tuned or
        default choice.  Outcomes are all 0 (force0,
        np_simulator_sv.py:346-349)."""
        form = output_form if output_form == "sv" else output_form.lower()
        if form not in ("dm", "densitymatrix", "sv", "statevector"):
            raise ValueError(f"Output form {output_form} is not supported.")
        sw = self._sweep
        sv_form = form in ("sv", "statevector")
        if sv_form and out is not None:
            # the same buffer objects as a bound call: a lookup by identity
            # (the entry holds them, so their ids stay theirs), then the launch
            hit = self.__dict__.get("_fast", {}).get((id(angles), id(input_states), id(out), id(status),
                                                      id(logprob), inputs_ready, variant))
            if hit is not None:
                hit[0](stream)
                return hit[2]
        key = None
        if (isinstance(out, torch.Tensor) and isinstance(status, torch.Tensor) and isinstance(angles, torch.Tensor)
                and (input_states is None or isinstance(input_states, torch.Tensor))
                and (logprob is None or isinstance(logprob, torch.Tensor))):
            key = _bind_key(angles, input_states, out, status, logprob, inputs_ready, variant)
        if sv_form and key is not None:
            # a bound buffer set called again through other tensor objects
            # (new views of the same memory): a lookup by memory, then the launch
            prep = self.__dict__.get("_prepared", {}).get(key)
            if prep is not None:
                self._remember(prep, angles, input_states, out, status, logprob, inputs_ready, variant)
                prep(stream)
                return BatchResult(out, self._zero_outcomes(out.shape[0]), status, logprob)
        if not _is_tensor_batch(angles, input_states, out):
            ang = np.asarray(angles, dtype=np.float64)
            ang = ang.reshape(1, -1) if ang.ndim == 1 else ang
            if ang.ndim != 2 or ang.shape[1] != len(self.mbqcircuit.trainable_nodes):
                raise ValueError(
                    f"Number of angles ({ang.shape[-1]}) does not match number of trainable nodes "
                    f"({len(self.mbqcircuit.trainable_nodes)})."
                )
            inp = self.input_state if input_states is None else input_states
            inp = None if inp is None else np.asarray(inp).reshape(-1, 2 ** sw.n_in)
            st, status_t, lp = sw.forward(ang, inp, logprob=True)
            psi = st.cpu().numpy().astype(np.complex128)
            B = ang.shape[0]
            res = (np.einsum("bi,bj->bij", psi, psi.conj()) if form in ("dm", "densitymatrix") else psi)
            return BatchResult(res, np.zeros((B, len(self.schedule_measure)), dtype=np.int8),
                               status_t.cpu().numpy(), lp.cpu().numpy())
        # torch buffers: bound once per buffer set, then one launch per call
        if input_states is None:
            input_states = self._default_input_tensor()
        mapped = _pinned(angles) or _pinned(input_states) or _pinned(out) or _pinned(status) or _pinned(logprob)
        if key is not None:
            cache = self.__dict__.setdefault("_prepared", collections.OrderedDict())
            prep = cache.get(key)
            if prep is None:
                # the bound call keeps references to these tensors, so their
                # memory cannot be handed to other tensors while it is cached
                prep = sw.prepare(angles, input_states, out, status=status, logprob=logprob, mapped_host=mapped,
                                  inputs_ready=inputs_ready, variant=variant)
                cache[key] = prep
                if len(cache) > self._PREPARED_CACHE:
                    cache.popitem(last=False)
            if sv_form:
                self._remember(prep, angles, input_states, out, status, logprob, inputs_ready, variant)
            prep(stream)
            states, status_t, lp = out, status, logprob
        else:
            states, status_t, lp = sw.forward(angles, input_states, out=out, status=status,
                                              logprob=True if logprob is None else logprob, stream=stream,
                                              mapped_host=mapped, inputs_ready=inputs_ready, variant=variant)
        B = states.shape[0]
        outc = self._zero_outcomes(B)
        if form in ("dm", "densitymatrix"):
            states = outer(states.to(sw.device) if states.device.type == "cpu" else states, stream=stream)
        return BatchResult(states, outc, status_t, lp)

    def release_buffers(self) -> None:
        """Drop the buffer sets ``run_batch`` has bound: their C calls and the
        references that keep the tensors (and their memory) alive.  Waits for
        the device first, since a call in flight on another stream may still
        use them; a later call with a buffer set binds it again."""
        if self.__dict__.get("_fast") or self.__dict__.get("_prepared"):
            torch.cuda.synchronize(self._sweep.device)
        self.__dict__.pop("_fast", None)
        self.__dict__.pop("_prepared", None)
        self.__dict__.pop("_single", None)

    def _remember(self, prep, angles, input_states, out, status, logprob, inputs_ready, variant):
        fast = self.__dict__.setdefault("_fast", {})
        if len(fast) >= 4 * self._PREPARED_CACHE:
            fast.clear()
        # the result object too: the same tensors every call
        res = BatchResult(out, self._zero_outcomes(out.shape[0]), status, logprob)
        fast[(id(angles), id(input_states), id(out), id(status), id(logprob), inputs_ready, variant)] = (
            prep, (angles, input_states, out, status, logprob), res)

    def _default_input_tensor(self):
        t = self.__dict__.get("_inp_t")
        if t is None:
            v = np.asarray(self.input_state if self.input_state is not None else
                           np.ones(2 ** self._sweep.n_in) / np.sqrt(2 ** self._sweep.n_in)).reshape(1, -1)
            t = torch.as_tensor(v, dtype=self._sweep.dtype, device=self._sweep.device)
            self._inp_t = t
        return t

    def _zero_outcomes(self, B):
        zb = self.__dict__.get("_zeros_b")
        if zb is not None and zb[0] == B:
            return zb[1]
        z = self.__dict__.get("_zeros")
        if z is None or z.shape[0] < B:
            z = torch.zeros((B, len(self.schedule_measure)), dtype=torch.int8, device=self._sweep.device)
            self._zeros = z
        self._zeros_b = (B, z[:B])
        return self._zeros_b[1]

    _SINGLE_POOL = 4  # idle single-run buffer sets kept (one per thread in ``run`` at a time)

    def _run_one(self, ang):
        """Output state and status of one run with this simulator's input
        state.  Register-kernel windows in complex64 go through pinned host
        buffers (taken from a small pool, so threads never share one); the
        others through device tensors."""
        sw = self._sweep
        inp = None if self.input_state is None else np.asarray(self.input_state).reshape(-1)
        variant = _TUNED.get(sw._tune_key(1), -1)
        if (sw.dtype != torch.complex64 or sw.plan.window > REGISTER_MAX_WINDOW or variant == STREAMED
                or sw.device.index not in (None, torch.cuda.current_device())):
            states, status, _ = sw.forward(ang.reshape(1, -1), None if inp is None else inp.reshape(1, -1))
            return states[0].cpu().numpy().astype(np.complex128), int(status[0].item())
        d = 2 ** sw.n_in
        if inp is None:
            inp = np.full(d, 1.0 / np.sqrt(d))
        elif inp.size != d:
            raise ValueError(f"input states need {d} amplitudes, got {inp.size}")
        pool = self.__dict__.setdefault("_single", [])
        try:
            one = pool.pop()
        except IndexError:
            one = None
        if one is None or one.variant != variant:
            one = _SingleRun(sw, variant)
        try:
            res = one(ang.reshape(-1), inp)
        except BaseException:
            torch.cuda.synchronize(sw.device)  # a launch may still use the buffers
            raise
        if len(pool) < self._SINGLE_POOL:
            pool.append(one)
        return res

    def run(self, angles, output_form: str = "dm", **kwargs):
        if kwargs.get("input_state") is not None:
            self.reset(input_state=kwargs.get("input_state"))
        if len(angles) != len(self.mbqcircuit.trainable_nodes):
            raise ValueError(
                f"Number of angles ({len(angles)}) does not match number of trainable nodes "
                f"({len(self.mbqcircuit.trainable_nodes)})."
            )
        if self.current_measurement >= len(self.schedule_measure):
            raise ValueError("No more measurements to be done.")
        form = output_form.lower()
        if form not in ("dm", "densitymatrix", "sv", "statevector"):
            raise ValueError(f"Output form {output_form} is not supported.")
        ang = np.asarray(angles, dtype=np.float64)
        if ang.size != self._sweep.n_angles:  # one value a node (an [A, 0] or [A, 2] array has none or two)
            raise ValueError(
                f"Number of angles ({ang.size}) does not match number of trainable nodes ({self._sweep.n_angles})."
            )
        psi, status = self._run_one(ang)
        self.current_measurement = len(self.schedule_measure)
        self.outcomes = {node: 0 for node in self.plan.outcome_nodes()}
        if status != _native.RUN_OK:
            warnings.warn("projected state has zero norm: output is NaN, as in the numpy simulator",
                          RuntimeWarning)
        self._qstate = psi
        if form in ("dm", "densitymatrix"):
            return np.outer(psi, psi.conj())
        return psi


class PatternSimulator:
    """Simulator for measuring patterns of MBQC circuits (pattern_simulator.py:19-88).

    Backends: ``"cuda-sv"`` (default), ``"cuda-dm"``, and ``"numpy-sv"`` /
    ``"numpy-dm"`` delegating to an installed mentpy.
    """

    def __init__(self, mbqcircuit, input_state: np.ndarray = None, backend: str = "cuda-sv", *args, **kwargs):
        supported = {"cuda-sv": CudaSimulatorSV, "cuda-dm": _cuda_dm, "numpy-sv": _numpy("NumpySimulatorSV"),
                     "numpy-dm": _numpy("NumpySimulatorDM")}
        backend = backend.lower()
        if backend not in supported:
            raise ValueError(
                f"Backend {backend} not supported. Supported backends are {supported.keys()}"
            )
        if input_state is None:
            input_state = np.ones(1)
            for _ in range(len(mbqcircuit.input_nodes)):
                input_state = np.kron(input_state, np.array([1, 1]) / np.sqrt(2))
        elif not isinstance(input_state, np.ndarray):
            raise TypeError(f"Input state must be a numpy array, not {type(input_state)}")
        self.simulator = supported[backend](mbqcircuit, input_state, *args, **kwargs)
        rb = getattr(self.simulator, "run_batch", None)
        if rb is not None:
            self.run_batch = rb  # the simulator's batched call, without a forwarding frame

    def __getattr__(self, name):
        return getattr(self.simulator, name)

    def __call__(self, angles, **kwargs):
        return self.run(angles, **kwargs)

    def __repr__(self) -> str:
        return f"{self.__class__.__name__} ({self.simulator!r})"

    def measure(self, angle: float, **kwargs):
        return self.simulator.measure(angle, **kwargs)

    def run(self, angles, **kwargs):
        return self.simulator.run(angles, **kwargs)

    def run_batch(self, angles, input_states=None, **kwargs) -> BatchResult:
        """Many angle vectors (and input states) in one call; see
        ``CudaSimulatorSV.run_batch`` / ``CudaSimulatorDM.run_batch``."""
        fn = getattr(self.simulator, "run_batch", None)
        if fn is None:
            raise NotImplementedError(f"{type(self.simulator).__name__} has no batched run")
        return fn(angles, input_states, **kwargs)

    def reset(self, input_state: np.ndarray = None):
        return self.simulator.reset(input_state)


def _cuda_dm(*args, **kwargs):
    from .dm import CudaSimulatorDM

    return CudaSimulatorDM(*args, **kwargs)


def _numpy(name):
    def make(*args, **kwargs):
        try:
            import mentpy.simulators as ms  # noqa: F401
        except Exception as exc:  # pragma: no cover - depends on the environment
            raise ValueError(f"backend numpy-* needs mentpy installed ({exc})")
        return getattr(ms, name)(*args, **kwargs)

    return make
