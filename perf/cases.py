"""Performance cases of the windowed MBQC sweep: what a user's program calls.

``listed()`` names twelve calls through the package's public entry points,
from one drop-in ``run`` of a nine-qubit wire to a training gradient of
262,144 runs; ``draw`` gives further cases of the same ranges.  A case's
circuit is ``rows`` wires of ``cols`` qubits, linked into a grid or not
(window = rows + 1), its runs are independent angle vectors and input states.
Angles are uniform in [0, 2 pi), input states uniform on the unit sphere
(Haar), as in the package's benchmark.

``exact`` restates the sweeps in plain complex128 torch: node by node on the
circuit's graph, column by column, with autograd for the gradients (with a
causal flow the forced-outcome state does not depend on the measurement
order).
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

# ------------------------------------------------------------------ the cases
_LISTED = [
    # One drop-in call, numpy in and out: the reference's own usage
    # (simulator(angles) inside an optimiser's loop), all launch and host time.
    dict(name="run_wire9", kind="run", grid=False, rows=1, cols=9, runs=1),
    # The headline batch: many_wires([8] * 4), 4096 angle vectors and inputs a
    # call on device buffers bound once (a serving loop).
    dict(name="batch_wires4x8", kind="batch", grid=False, rows=4, cols=8, runs=4096),
    # A wide register-resident window (w = 9) with log-probabilities, a batch
    # that is no power of two.
    dict(name="batch_grid8x10", kind="forward", grid=True, rows=8, cols=10, runs=5000),
    # The widest window the benchmark streams (w = 17): 64 runs of 160 qubits.
    dict(name="wide_grid16x10", kind="forward", grid=True, rows=16, cols=10, runs=64),
    # Training through torch.autograd at an ordinary size: states and angle
    # gradients of a ragged batch.
    dict(name="autograd_wires4x8", kind="autograd", grid=False, rows=4, cols=8, runs=333),
    # The fused training gradient: 1024 angle vectors x 256 data pairs.
    dict(name="fidelity_wires6x12", kind="fidelity", grid=False, rows=6, cols=12, runs=1024, pairs=256),
    # Gradients of the widest circuit (w = 17, 144 angles).
    dict(name="autograd_grid16x10", kind="autograd", grid=True, rows=16, cols=10, runs=64),
    # Drawn outcomes with byproduct corrections (the hardware's view of a run).
    dict(name="sampled_wires6x12", kind="sampled", grid=False, rows=6, cols=12, runs=500),
    # Thousands of noisy density-matrix circuits of uneven width and depth.
    dict(name="mixed_dm", kind="dm_mixed", circuits=2048, mix=5, noise=0.01),
    # Their gradients through the noise channel.
    dict(name="mixed_dm_grad", kind="dm_mixed_grad", circuits=2048, mix=5, noise=0.01),
    # One noisy circuit, a batch of runs, at the uneven batch's widest window
    # (w = 7).
    dict(name="dm_wires6x12", kind="dm", grid=False, rows=6, cols=12, runs=500, noise=0.01),
    # A density matrix beyond shared memory (w = 9), a few runs.
    dict(name="dm_grid8x6", kind="dm", grid=True, rows=8, cols=6, runs=24, noise=0.01),
]


def listed():
    return [dict(c) for c in _LISTED]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    """One more case of the listed cases' ranges (no dearer than the dearest
    of its kind)."""
    kind = rng.choice(["run", "batch", "forward", "wide", "autograd", "wide_autograd", "fidelity", "sampled",
                       "dm_mixed", "dm_mixed_grad", "dm", "wide_dm"])
    grid = rng.random() < 0.5
    if kind == "run":
        return dict(kind="run", grid=grid, rows=rng.randint(1, 4), cols=rng.randint(3, 12), runs=1)
    if kind in ("batch", "forward"):
        rows = rng.randint(1, 9)
        return dict(kind=kind, grid=grid, rows=rows, cols=rng.randint(3, 12),
                    runs=_log_int(rng, 16, min(16384, 5000 << max(0, 8 - rows))))
    if kind == "wide":
        rows = rng.randint(10, 16)
        return dict(kind="forward", grid=grid, rows=rows, cols=rng.randint(3, 10),
                    runs=_log_int(rng, 1, min(1024, 64 << (16 - rows))))
    if kind == "autograd":
        return dict(kind="autograd", grid=grid, rows=rng.randint(1, 7), cols=rng.randint(3, 12),
                    runs=_log_int(rng, 16, 4096))
    if kind == "wide_autograd":
        rows = rng.randint(8, 16)
        return dict(kind="autograd", grid=grid, rows=rows, cols=rng.randint(3, 10),
                    runs=_log_int(rng, 1, min(512, 64 << (16 - rows))))
    if kind == "fidelity":
        return dict(kind="fidelity", grid=grid, rows=rng.randint(2, 6), cols=rng.randint(4, 12),
                    runs=_log_int(rng, 1, 1024), pairs=_log_int(rng, 4, 256))
    if kind == "sampled":
        rows = rng.randint(2, 14)
        return dict(kind="sampled", grid=grid, rows=rows, cols=rng.randint(3, 12),
                    runs=_log_int(rng, 4, 500 >> max(0, rows - 9)))
    if kind in ("dm_mixed", "dm_mixed_grad"):
        return dict(kind=kind, circuits=_log_int(rng, 16, 2048), mix=rng.randint(0, 10**6),
                    noise=rng.choice([0.0, 0.01, 0.05]))
    rows = rng.randint(2, 6) if kind == "dm" else rng.randint(7, 9)
    return dict(kind="dm", grid=grid, rows=rows, cols=rng.randint(3, 12 if rows <= 6 else 6),
                runs=_log_int(rng, 8, 500 if rows <= 6 else (96 >> 2 * (rows - 7)) * 4 // 3),
                noise=rng.choice([0.0, 0.01, 0.05]))


# ----------------------------------------------------------------- the inputs
def _device():
    return torch.device("cuda") if torch.cuda.is_available() else torch.device("cpu")


def _generator(seed):
    return np.random.default_rng(seed)


def _angles(g, *shape):
    return g.uniform(0.0, 2.0 * np.pi, size=shape)


def _states(g, count, n):
    z = g.standard_normal((count, 2**n), dtype=np.float32) + 1j * g.standard_normal((count, 2**n), dtype=np.float32)
    return (z / np.linalg.norm(z, axis=1, keepdims=True)).astype(np.complex64)


def _complex(g, *shape):
    return (g.standard_normal(shape, dtype=np.float32) + 1j * g.standard_normal(shape, dtype=np.float32)).astype(
        np.complex64)


def _mix(case):
    """(wires, depth) of every circuit of an uneven batch: 2 to 6 wires of 4
    to 12 qubits."""
    g = np.random.default_rng(case["mix"])
    return [(int(w), int(d)) for w, d in zip(g.integers(2, 7, case["circuits"]), g.integers(4, 13, case["circuits"]))]


def _inputs(case, seed):
    """The numbers a case's call takes, on the host, from the seed alone."""
    g = _generator(seed)
    kind = case["kind"]
    if kind in ("dm_mixed", "dm_mixed_grad"):
        shapes = _mix(case)
        C = len(shapes)
        w = max(s[0] for s in shapes)
        a = max(s[0] * (s[1] - 1) for s in shapes)
        ang, psi = np.zeros((C, a)), np.zeros((C, 2**w), np.complex64)
        gam = np.zeros((C, 4**w), np.complex64)
        all_ang, all_psi, all_gam = _angles(g, C, a), _complex(g, C, 2**w), _complex(g, C, 2**w, 2**w)
        for c, (rows, cols) in enumerate(shapes):
            n, d = rows * (cols - 1), 2**rows
            ang[c, :n] = all_ang[c, :n]
            v = all_psi[c, :d]
            psi[c, :d] = v / np.linalg.norm(v)
            x = all_gam[c, :d, :d]
            gam[c, : d * d] = (0.5 * (x + x.conj().T)).reshape(-1)  # an observable
        return dict(angles=ang, psi=psi, gamma=gam)
    rows, cols, runs = case["rows"], case["cols"], case["runs"]
    d = dict(angles=_angles(g, runs, rows * (cols - 1)), psi=_states(g, case.get("pairs", runs), rows))
    if kind == "fidelity":
        d["targets"] = _states(g, case["pairs"], rows)
    if kind == "autograd":
        d["grad_out"] = _complex(g, runs, 2**rows)
    return d


# -------------------------------------------------------------- prepare / run
def prepare(case, seed):
    """Circuit, simulator and device inputs: what a program holds before the
    call."""
    from mentpy_gb300 import PatternSimulator
    from mentpy_gb300 import circuit as C
    from mentpy_gb300.dm import DensityMatrixSweep, UnevenDensityMatrixBatch
    from mentpy_gb300.native_plan import GraphBatch
    from mentpy_gb300.sweep import StatevectorSweep

    kind = case["kind"]
    x = _inputs(case, seed)
    st = dict(case=case)
    if kind in ("dm_mixed", "dm_mixed_grad"):
        batch = UnevenDensityMatrixBatch.from_graph_batch(GraphBatch.many_wires(_mix(case)))
        buf = batch.allocate()
        buf["angles"].copy_(torch.from_numpy(x["angles"]))
        buf["inputs"].copy_(torch.from_numpy(x["psi"]))
        if kind == "dm_mixed_grad":
            buf["grad_out"] = torch.from_numpy(x["gamma"]).cuda()
        st.update(batch=batch, buf=buf)
        return st
    rows, cols = case["rows"], case["cols"]
    circ = C.grid_cluster(rows, cols) if case["grid"] else C.many_wires([cols] * rows)
    if kind == "run":
        st.update(sim=PatternSimulator(circ, input_state=x["psi"][0].astype(np.complex128), backend="cuda-sv"),
                  angles=x["angles"][0])
        return st
    st["angles"], st["psi"] = torch.from_numpy(x["angles"]).cuda(), torch.from_numpy(x["psi"]).cuda()
    if kind == "batch":
        st.update(sim=PatternSimulator(circ, backend="cuda-sv"),
                  out=torch.empty_like(st["psi"]),
                  status=torch.empty(case["runs"], dtype=torch.int32, device="cuda"))
    elif kind == "dm":
        st["sweep"] = DensityMatrixSweep(circ)
    else:
        st["sweep"] = StatevectorSweep(circ)
    if kind == "fidelity":
        st["targets"] = torch.from_numpy(x["targets"]).cuda()
    elif kind == "autograd":
        st["grad_out"] = torch.from_numpy(x["grad_out"]).cuda()
        st["angles"].requires_grad_(True)
    elif kind == "sampled":
        st["seed"] = int(seed)
    return st


def run(st):
    """One call, as a program makes it."""
    case = st["case"]
    kind = case["kind"]
    if kind == "run":
        st["sim"].reset()
        return st["sim"](st["angles"])
    if kind == "batch":
        r = st["sim"].run_batch(st["angles"], st["psi"], out=st["out"], status=st["status"], inputs_ready=True)
        return r.states, r.outcomes, r.status
    if kind == "forward":
        states, status, logprob = st["sweep"].forward(st["angles"], st["psi"], logprob=True)
        return states, status, logprob
    if kind == "autograd":
        from mentpy_gb300.autograd import sweep_states

        z = sweep_states(st["sweep"], st["angles"], st["psi"])
        (grad,) = torch.autograd.grad(z, st["angles"], st["grad_out"])
        return z.detach(), grad
    if kind == "fidelity":
        return st["sweep"].fidelity_grad(st["angles"], st["psi"], st["targets"])
    if kind == "sampled":
        return st["sweep"].forward_sampled(st["angles"], st["psi"], seed=st["seed"])
    if kind == "dm":
        return st["sweep"].forward(st["angles"], st["psi"], noise=case["noise"], want_probs=True)
    buf = st["buf"]
    if kind == "dm_mixed":
        st["batch"].run(buf, noise=case["noise"])
        return buf["rho"], buf["outcomes"], buf["probs"], buf["status"]
    st["batch"].adjoint(buf, noise=case["noise"])
    return buf["grad"], buf["rho"], buf["outcomes"], buf["status"]


# ----------------------------------------------------------------------- work
def _sv_flops(rows, cols):
    """Complex contraction, expansion, norm and rescale of every step: 12
    flops an amplitude of the 2^(rows + 1) window."""
    return rows * (cols - 1) * 12 * 2 ** (rows + 1)


def _dm_flops(rows, cols):
    """Block contraction of the Hermitian 2^rows x 2^rows matrix a step: 16
    flops an entry of one triangle."""
    return rows * (cols - 1) * 8 * 4**rows


def work(case):
    kind = case["kind"]
    if kind in ("dm_mixed", "dm_mixed_grad"):
        k = 3 if kind == "dm_mixed_grad" else 1
        flops = bytes_ = 0
        for rows, cols in _mix(case):
            m, d = rows * (cols - 1), 2**rows
            flops += k * _dm_flops(rows, cols)
            bytes_ += m * 8 + d * 8 + d * d * 8 + m * 1 + 4
            bytes_ += d * d * 8 + m * 8 if k == 3 else m * 8
        return dict(bytes=bytes_, flops=flops)
    rows, cols, runs = case["rows"], case["cols"], case["runs"]
    m, d = rows * (cols - 1), 2**rows
    if kind == "dm":
        return dict(bytes=runs * (m * 8 + d * 8 + d * d * 8 + m * 9 + 4), flops=runs * _dm_flops(rows, cols))
    if kind == "fidelity":
        return dict(bytes=runs * (m * 16 + 8) + case["pairs"] * d * 16,
                    flops=3 * runs * case["pairs"] * _sv_flops(rows, cols))
    if kind == "autograd":
        return dict(bytes=runs * (m * 16 + d * 24), flops=3 * runs * _sv_flops(rows, cols))
    if kind == "run":
        return dict(bytes=m * 8 + d * 8 + d * d * 16, flops=_sv_flops(rows, cols))
    extra = {"batch": 4, "forward": 12, "sampled": 4 + m}[kind]
    return dict(bytes=runs * (m * 8 + d * 16 + extra), flops=runs * _sv_flops(rows, cols))


# ---------------------------------------------------------------------- exact
def _graph_order(rows, cols):
    """Measured nodes column by column; node (r, j) has label r * cols + j."""
    return [(r, j) for j in range(cols - 1) for r in range(rows)]


def _neighbours(grid, live, r, j):
    return [n for n in live if n == (r, j - 1) or (grid and n[1] == j and abs(n[0] - r) == 1)]


def _cz(s, i, j, n):
    """Sign of a CZ between qubits i < j of the n leading-first qubits of the
    last axis."""
    v = s.reshape(*s.shape[:-1], 2**i, 2, 2 ** (j - i - 1), 2, 2 ** (n - j - 1))
    sign = torch.ones(2, 1, 2, 1, dtype=torch.float64, device=s.device)
    sign[1, 0, 1, 0] = -1.0
    return (v * sign).reshape(s.shape)


def _sv_exact(grid, rows, cols, ang, psi, want_logprob=False):
    """Normalised force-0 states (no global phase) of runs [B] in output-row
    order, and ln of the branch probability."""
    live = [(r, 0) for r in range(rows)]
    s = psi
    if grid:
        for r in range(rows - 1):
            s = _cz(s, r, r + 1, rows)
    ph = torch.exp(-1j * ang.to(torch.complex128))
    lp = torch.zeros(s.shape[0], dtype=torch.float64, device=s.device)
    for r, j in _graph_order(rows, cols):
        s = s.unsqueeze(-1).expand(*s.shape, 2).reshape(s.shape[0], -1) / math.sqrt(2.0)
        new = (r, j + 1)
        live.append(new)
        for nb in _neighbours(grid, live[:-1], *new):
            s = _cz(s, live.index(nb), len(live) - 1, len(live))
        i = live.index((r, j))
        v = s.reshape(s.shape[0], 2**i, 2, -1)
        s = (v[:, :, 0] + ph[:, r * (cols - 1) + j, None, None] * v[:, :, 1]).reshape(s.shape[0], -1) / math.sqrt(2.0)
        live.remove((r, j))
        n2 = (s.real**2 + s.imag**2).sum(1, keepdim=True)
        if want_logprob:
            lp = lp + torch.log(n2[:, 0])
        s = s / torch.sqrt(n2)
    order = sorted(range(rows), key=lambda q: live[q][0])
    s = s.reshape(-1, *([2] * rows)).permute(0, *[1 + q for q in order]).reshape(s.shape[0], -1)
    return s, lp


def _phase(ang):
    """The phase the reference's summing partial trace leaves: e^{i t / 2} per
    step, t the angle reduced to [-pi, pi]."""
    t = torch.remainder(ang + math.pi, 2 * math.pi) - math.pi
    return torch.exp(0.5j * t.sum(1, keepdim=True).to(torch.complex128))


def _dm_exact(grid, rows, cols, ang, psi, noise):
    """rho over the outputs [B, 2^rows, 2^rows] and the outcome-0
    probabilities, each qubit depolarised right before it is measured and the
    outputs at the end."""
    B, dev = psi.shape[0], psi.device
    a, b = 1.0 - 4.0 * noise / 3.0, 2.0 * noise / 3.0
    live = [(r, 0) for r in range(rows)]
    if grid:
        for r in range(rows - 1):
            psi = _cz(psi, r, r + 1, rows)
    s = psi.unsqueeze(2) * psi.conj().unsqueeze(1)
    e = torch.exp(1j * ang.to(torch.complex128))
    probs = []
    for r, j in _graph_order(rows, cols):
        d = s.shape[1]
        s = (s.reshape(B, d, 1, d, 1).expand(B, d, 2, d, 2) / 2.0).reshape(B, 2 * d, 2 * d)
        new = (r, j + 1)
        live.append(new)
        n = len(live)
        for nb in _neighbours(grid, live[:-1], *new):
            q = live.index(nb)
            s = _cz(s, q, n - 1, n)
            s = _cz(s.transpose(1, 2), q, n - 1, n).transpose(1, 2)
        i = live.index((r, j))
        v = s.reshape(B, 2**i, 2, 2 ** (n - 1 - i), 2**i, 2, 2 ** (n - 1 - i))
        x = e[:, r * (cols - 1) + j].reshape(B, 1, 1, 1, 1)
        y = 0.5 * a * (v[:, :, 0, :, :, 0] + v[:, :, 1, :, :, 1] + x * v[:, :, 0, :, :, 1]
                       + x.conj() * v[:, :, 1, :, :, 0]) + b * (v[:, :, 0, :, :, 0] + v[:, :, 1, :, :, 1])
        y = y.reshape(B, d, d)
        p = torch.einsum("bii->b", y).real
        probs.append(p)
        s = y / p.reshape(B, 1, 1)
        live.remove((r, j))
    for q in range(rows):
        v = s.reshape(B, 2**q, 2, 2 ** (rows - 1 - q), 2**q, 2, 2 ** (rows - 1 - q))
        t = b * (v[:, :, 0, :, :, 0] + v[:, :, 1, :, :, 1])
        out = a * v
        diag = torch.zeros_like(out)
        diag[:, :, 0, :, :, 0] = t
        diag[:, :, 1, :, :, 1] = t
        s = (out + diag).reshape(B, 2**rows, 2**rows)
    order = sorted(range(rows), key=lambda q: live[q][0])
    s = s.reshape(B, *([2] * (2 * rows))).permute(
        0, *[1 + q for q in order], *[1 + rows + q for q in order]).reshape(B, 2**rows, 2**rows)
    return s, torch.stack(probs, 1)


def _chunks(n, size):
    return [(i, min(n, i + size)) for i in range(0, n, size)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "sampled":
        return None  # the state's global phase is not specified
    dev = _device()
    x = {k: torch.from_numpy(v).to(dev) for k, v in _inputs(case, seed).items()}
    if kind in ("dm_mixed", "dm_mixed_grad"):
        return _exact_mixed(case, x)
    grid, rows, cols, runs = case["grid"], case["rows"], case["cols"], case["runs"]
    ang, psi = x["angles"], x["psi"].to(torch.complex128)
    if kind in ("run", "batch", "forward"):
        s, lp = _sv_exact(grid, rows, cols, ang, psi, want_logprob=True)
        s = s * _phase(ang)
        if kind == "run":
            return np.outer(s[0].cpu().numpy(), s[0].cpu().numpy().conj())
        return (s, None, None) if kind == "batch" else (s, None, lp)
    if kind == "dm":
        size = max(1, 2**22 >> (2 * rows))
        parts = [_dm_exact(grid, rows, cols, ang[i:j], psi[i:j], case["noise"]) for i, j in _chunks(runs, size)]
        # (in a circuit with causal flow every probability is 1/2, in any
        # measurement order)
        return torch.cat([p[0] for p in parts]), None, None, torch.cat([p[1] for p in parts])
    if kind == "autograd":
        zs, gs = [], []
        for i, j in _chunks(runs, max(1, 2**21 >> rows)):
            t = ang[i:j].clone().requires_grad_(True)
            z, _ = _sv_exact(grid, rows, cols, t, psi[i:j])
            (g,) = torch.autograd.grad(z, t, x["grad_out"][i:j].to(torch.complex128))
            zs.append(z.detach())
            gs.append(g)
        return torch.cat(zs), torch.cat(gs)
    tg, J = x["targets"].to(torch.complex128), case["pairs"]
    losses, grads = [], []
    for i, j in _chunks(runs, max(1, 2**21 // (J << rows))):
        t = ang[i:j].clone().requires_grad_(True)
        z, _ = _sv_exact(grid, rows, cols, t.repeat_interleave(J, 0), psi.repeat(j - i, 1))
        ov = (tg.repeat(j - i, 1).conj() * z).sum(1)
        loss = 1.0 - (ov.real**2 + ov.imag**2).reshape(j - i, J).mean(1)
        (g,) = torch.autograd.grad(loss.sum(), t)
        losses.append(loss.detach())
        grads.append(g)
    return torch.cat(losses), torch.cat(grads)


def _exact_mixed(case, x):
    shapes, noise = _mix(case), case["noise"]
    grad_case = case["kind"] == "dm_mixed_grad"
    dev = x["angles"].device
    C, w = len(shapes), max(s[0] for s in shapes)
    m = max(s[0] * (s[1] - 1) for s in shapes)
    rho = torch.zeros(C, 4**w, dtype=torch.complex128, device=dev)
    probs = torch.zeros(C, m, dtype=torch.float64, device=dev)
    grad = torch.zeros(C, m, dtype=torch.float64, device=dev)
    groups = {}
    for c, sh in enumerate(shapes):
        groups.setdefault(sh, []).append(c)
    for (rows, cols), members in groups.items():
        n, d = rows * (cols - 1), 2**rows
        for i, j in _chunks(len(members), max(1, 2**20 >> (2 * rows))):
            idx = torch.tensor(members[i:j], device=dev)
            t = x["angles"][idx, :n].clone().requires_grad_(grad_case)
            r, p = _dm_exact(False, rows, cols, t, x["psi"][idx, :d].to(torch.complex128), noise)
            if grad_case:
                gam = x["gamma"][idx, : d * d].to(torch.complex128).reshape(-1, d, d)
                (g,) = torch.autograd.grad(r, t, gam)
                grad[idx, :n] = g
            rho[idx, : d * d] = r.detach().reshape(-1, d * d)
            probs[idx, :n] = p.detach()
    if grad_case:
        return grad, rho, None, None
    return rho, None, probs, None
