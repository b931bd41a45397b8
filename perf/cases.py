"""The work that users have the engine do, as cases to be timed.

Each case goes through the package's public entry points on inputs made from a
seed: circuits executed on device states, the reference's GpuExecutionWrapper
on a host state, the batched kernel, the continuous-batching server, and the
read-out of a state.  Circuits, sizes, precisions and depths are those of the
benchmark workloads and of the reference's command-line programs.

    listed()             the cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  inputs, plans and handles a program has before the call
    run(state)           one pass; returns its outputs
    work(case)           the bytes and operations a pass cannot do without
    exact(case, seed)    the same outputs in 64 bits, in plain torch and numpy
"""
import ctypes
import math
import random

import numpy as np
import torch

import simulador_quantico_b200 as sq
from simulador_quantico_b200 import workloads as wl
from simulador_quantico_b200._lib import lib, load_dropin

REAL_BYTES = {"f32": 4, "f64": 8}


def listed():
    return [
        # general.out's Hadamard benchmark at the size of the smallest fixture:
        # one short launch, the latency of a call
        {"name": "hadamard10_f64", "kind": "hadamard", "n": 10, "precision": "f64", "repeats": 3},
        # the serving mix's layered circuits, smallest and largest
        {"name": "layered12_f32", "kind": "layered", "n": 12, "precision": "f32", "layers": 20},
        {"name": "layered26_f32", "kind": "layered", "n": 26, "precision": "f32", "layers": 20},
        # a deep FP64 circuit at a size where a pass is bound by the chip and not by launches
        {"name": "layered28_f64", "kind": "layered", "n": 28, "precision": "f64", "layers": 10},
        # a whole small search (an odd number of qubits), hundreds of passes over a state that stays in L2
        {"name": "grover17_f32", "kind": "grover", "n": 17, "precision": "f32", "iterations": 0},
        # the benchmark search's iterations: a one-iteration plan run many times on a state larger than L2
        {"name": "grover26_f64", "kind": "grover", "n": 26, "precision": "f64", "iterations": 32},
        # the serving mix's QFTs, near the upper end and at an odd size
        {"name": "qft27_f32", "kind": "qft", "n": 27, "precision": "f32"},
        # one gate layer on a large FP64 state
        {"name": "hadamard28_f64", "kind": "hadamard", "n": 28, "precision": "f64", "repeats": 1},
        # many circuits of 10 to 22 qubits in one launch
        {"name": "batch128_f32", "kind": "batch", "count": 128, "precision": "f32", "lo": 10, "hi": 22, "mix": 5},
        # a burst of requests of the serving mix on plans built beforehand, states kept for the caller
        {"name": "served24_f32", "kind": "served", "count": 24, "precision": "f32", "mix": 7, "max_qubits": 28},
        # the reference's host entry point: state in, circuit, state out
        {"name": "wrapper20_f64", "kind": "wrapper", "n": 20, "precision": "f64", "layers": 10},
        # reading a search's register out: norm, distribution over some bits, most likely value, one qubit measured
        {"name": "readout25_f32", "kind": "readout", "n": 25, "precision": "f32", "bits": 11},
    ]


def draw(rng):
    """One more case: kinds by weight, sizes spread over each kind's range, depths and precisions as in use."""
    kind = rng.choice(["layered"] * 4 + ["qft"] * 3 + ["grover"] * 2 + ["hadamard", "batch", "served", "wrapper", "readout"])
    prec = rng.choice(["f32", "f64"])
    if kind == "layered":
        n = rng.randint(10, 28 if prec == "f32" else 27)
        # the largest states get fewer layers, so that no drawn case costs more than the largest listed one
        return {"kind": kind, "n": n, "precision": prec, "layers": rng.randint(2, 20) if n <= 26 else rng.randint(2, 10)}
    if kind == "qft":
        return {"kind": kind, "n": rng.randint(10, 28), "precision": prec}
    if kind == "grover":
        if rng.random() < 0.6:
            return {"kind": kind, "n": rng.randint(12, 20 if prec == "f32" else 19), "precision": prec, "iterations": 0}
        return {"kind": kind, "n": rng.randint(18, 26), "precision": prec, "iterations": rng.randint(2, 32)}
    if kind == "hadamard":
        return {"kind": kind, "n": rng.randint(8, 28), "precision": prec, "repeats": rng.choice([1, 3])}
    if kind == "batch":
        lo = rng.randint(10, 14)
        return {"kind": kind, "count": rng.randint(16, 128), "precision": prec, "lo": lo,
                "hi": rng.randint(lo + 2, 22 if prec == "f32" else 21), "mix": rng.randint(1, 10 ** 6)}
    if kind == "served":
        return {"kind": kind, "count": rng.randint(6, 24), "precision": "f32", "mix": rng.randint(1, 10 ** 6),
                "max_qubits": rng.randint(20, 28)}
    if kind == "wrapper":
        return {"kind": kind, "n": rng.randint(11, 22), "precision": prec, "layers": rng.randint(2, 10)}
    return {"kind": kind, "n": rng.randint(16, 27), "precision": prec, "bits": rng.randint(3, 14)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _requests(case, seed):
    """The circuits of a batch or a burst: kinds and sizes from the case, angles and inputs from the seed;
    a list of (kind, qubits, layers or 0, seed or basis index or marked index)."""
    shape, val = random.Random(case["mix"]), random.Random(seed)
    out = []
    for i in range(case["count"]):
        if case["kind"] == "batch":
            n = shape.randint(case["lo"], case["hi"])
            out.append(("qft", n, 0, val.randrange(1 << n)) if i % 2 else ("layered", n, 10, val.randrange(1 << 30)))
            continue
        u = shape.random()
        if u < 0.6:
            out.append(("layered", min(shape.randint(12, 26), case["max_qubits"]), 20, val.randrange(1 << 30)))
        elif u < 0.9:
            n = min(shape.randint(16, 28), case["max_qubits"])
            out.append(("qft", n, 0, val.randrange(1 << n)))
        else:
            n = shape.randint(14, 20)
            out.append(("grover", n, 0, val.randrange(1 << n)))
    return out


def _spec(req):
    kind, n, layers, v = req
    if kind == "layered":
        return wl.random_layered(n, layers, v)
    return wl.qft(n, v) if kind == "qft" else wl.grover_search(n, v)


def _circuit(spec):
    return spec.build(sq.Circuit())


def _value(case, seed):
    """The basis index or marked index a seed stands for."""
    return random.Random(seed * 1000003 + case["n"]).randrange(1 << case["n"])


class _Memory:
    """Amplitudes in device memory that `owner` holds, for torch.as_tensor (which keeps this object, and so the owner)."""

    def __init__(self, first, amps, wide, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (amps, 2), "strides": None, "version": 3,
                                         "typestr": "<f8" if wide else "<f4", "data": (first, False)}


def _tensor(state):
    """A device state's memory as a torch tensor of (re, im) pairs, without a copy."""
    first = int(lib.hgm_state_device_ptr(state.h))
    return torch.as_tensor(_Memory(first, 1 << state.qubits, state.nbytes >> state.qubits == 16, state), device="cuda")


def _random_state(n, seed, device):
    """A normalised state with Gaussian amplitudes, as (re, im) pairs in 64 bits."""
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    v = torch.randn((1 << n, 2), generator=g, device=device, dtype=torch.float32).double()
    return v.div_(v.square().sum().sqrt())


class _Run:
    """What a program keeps between calls."""


def prepare(case, seed):
    sq.init()
    s, kind, prec = _Run(), case["kind"], case["precision"]
    s.kind, s.case = kind, case
    if kind in ("hadamard", "layered", "qft", "grover"):
        n = case["n"]
        s.index = 0
        if kind == "hadamard":
            spec = wl.hadamard_benchmark(n, case["repeats"])
            s.index = _value(case, seed)
        elif kind == "layered":
            spec = wl.random_layered(n, case["layers"], seed)
        elif kind == "qft":
            spec = wl.qft(n, 0)
            s.index = _value(case, seed)
        else:
            spec = wl.grover_search(n, _value(case, seed))
        s.plans = []
        if kind == "grover" and case["iterations"]:
            # H on every qubit, then a one-iteration plan run `iterations` times
            (h, _, _), (steps, _, _) = spec.calls
            for calls, times in (([(h, 1, True)], 1), ([(steps, 1, True)], case["iterations"])):
                one = wl.CircuitSpec("grover", n, 0, spec.gates, calls)
                s.plans.append((sq.Plan(_circuit(one), n, prec).upload(), times))
        else:
            s.plans.append((sq.Plan(_circuit(spec), n, prec).upload(), 1))
        s.state = sq.State(n, prec)
        s.out = _tensor(s.state)
    elif kind == "batch":
        s.batch = sq.Batch(prec, 2)
        for req in _requests(case, seed):
            spec = _spec(req)
            s.batch.add(_circuit(spec), spec.qubits, spec.init_index)
        s.batch.finalize()
        views = [s.batch.state(j) for j in range(case["count"])]
        # every job's state lies in one arena, in job order
        first = int(lib.hgm_state_device_ptr(views[0].h))
        s.out = torch.as_tensor(_Memory(first, sum(1 << v.qubits for v in views), prec == "f64", s.batch), device="cuda")
    elif kind == "served":
        s.server = sq.Server(prec, keep_states=True)
        s.requests = [(sq.Plan(_circuit(spec), spec.qubits, prec).upload(), spec.init_index,
                       spec.meta.get("search_mask", 0)) for spec in map(_spec, _requests(case, seed))]
        s.kept = []
    elif kind == "wrapper":
        n = case["n"]
        s.lib = load_dropin(prec)
        s.circuit = _circuit(wl.random_layered(n, case["layers"], seed))
        s.points = s.circuit.ref_pts(prec)
        v = _random_state(n, seed, "cuda").cpu().numpy()
        s.host = np.ascontiguousarray(v.view(np.complex128).reshape(-1).astype(sq.engine.NP_DTYPE[sq.engine.PREC[prec]]))
    else:
        n = case["n"]
        s.state = sq.State(n, prec)
        s.out = _tensor(s.state)
        s.out.copy_(_random_state(n, seed, "cuda"))
        s.mask = _read_mask(case)
    torch.cuda.synchronize()
    return s


def _read_mask(case):
    """The index bits whose distribution is read: every second one from the middle up, then the low ones."""
    n, bits = case["n"], case["bits"]
    order = list(range(n // 3, n, 2)) + list(range(n // 3))
    return sum(1 << b for b in order[:bits])


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def run(s):
    if s.kind in ("hadamard", "layered", "qft", "grover"):
        s.state.set_basis(s.index)
        for plan, times in s.plans:
            s.state.execute(plan, times)
        return s.out
    if s.kind == "batch":
        s.batch.run()
        return s.out
    if s.kind == "served":
        for rid in s.kept:
            s.server.release(rid)
        s.kept = [s.server.submit_plan(*req) for req in s.requests]
        done = {r["id"]: r for r in s.server.drain(len(s.kept))}
        assert all(r["status"] == 0 for r in done.values())
        return {"states": [_tensor(s.server.result_state(rid)) for rid in s.kept],
                "norms": np.array([done[rid]["norm"] for rid in s.kept]),
                "argmax": np.array([done[rid]["argmax"] for rid in s.kept])}
    if s.kind == "wrapper":
        # the reference's default tuning
        s.lib.GpuExecutionWrapper(s.host.ctypes.data_as(ctypes.c_void_p), ctypes.c_void_p(s.points), s.case["n"],
                                  4, 8, 1, 64, 2, 1)
        return s.host
    norm = s.state.norm()
    probs = s.state.marginal_probs(s.mask)
    arg, top = s.state.marginal_argmax((1 << s.case["n"]) - 1)
    # the sample is far from P(0), so the outcome does not hang on rounding
    outcome, p = s.state.measure_qubit(s.case["n"] // 2, 0.25)
    return {"norm": norm, "probs": probs, "argmax": arg, "top": top, "outcome": outcome, "p": p, "state": s.out}


# ---------------------------------------------------------------------------
# the work of a pass
# ---------------------------------------------------------------------------

def _circuit_work(kind, n, layers, prec, repeats=1):
    """One write of the final state, and the arithmetic of the gates one at a time: a complex 2x2 with real
    entries takes 6 operations an amplitude, a diagonal factor 6 on the amplitudes it changes."""
    amps, amp = 1 << n, 2 * REAL_BYTES[prec]
    if kind == "layered":
        ops = layers * n * (6 + 3)
    elif kind == "qft":
        ops = n * 6 + n * (n - 1) // 2 * 1.5
    elif kind == "grover":
        ops = repeats * 2 * n * 6
    else:
        ops = repeats * n * 6
    return amps * amp, amps * ops


def work(case):
    kind, prec = case["kind"], case["precision"]
    if kind in ("batch", "served"):
        b = f = 0
        for k, n, layers, _ in _requests(case, 0):
            rep = int(math.pi / 4.0 * math.sqrt(1 << n)) if k == "grover" else 1
            x, y = _circuit_work(k, n, layers, prec, rep)
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    n = case["n"]
    if kind == "wrapper":
        b, f = _circuit_work("layered", n, case["layers"], prec)
        return {"bytes": 2 * b, "flops": f}
    if kind == "readout":
        amps, amp = 1 << n, 2 * REAL_BYTES[prec]
        # the state is read once for the three figures, and half of it once and all of it written for the measurement
        return {"bytes": amps * amp * 2.5 + 8 * (1 << case["bits"]), "flops": amps * 4}
    if kind == "grover":
        rep = case["iterations"] or int(math.pi / 4.0 * math.sqrt(1 << n))
        b, f = _circuit_work(kind, n, 0, prec, rep)
    else:
        b, f = _circuit_work(kind, n, case.get("layers", 0), prec, case.get("repeats", 1))
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits
# ---------------------------------------------------------------------------

def _pairs(v):
    return torch.view_as_real(v.reshape(-1))


def _layered(n, layers, seed, v):
    """The random layered circuit on v (complex128, index bit n-1-q is qubit q), gate by gate."""
    rng = np.random.default_rng(seed)
    for _ in range(layers):
        theta, phi = rng.uniform(0.0, 2.0 * math.pi, n), rng.uniform(0.0, 2.0 * math.pi, n)
        for q in range(n):
            w = v.view(1 << q, 2, -1)
            c, s = math.cos(phi[q] / 2), math.sin(phi[q] / 2)
            e = complex(math.cos(theta[q] / 2), math.sin(theta[q] / 2))
            a, b = w[:, 0] * e.conjugate(), w[:, 1] * e
            w[:, 0] = c * a - s * b
            w[:, 1] = s * a + c * b
        perm = rng.permutation(n)
        for g in range(n // 2):
            c, t = int(perm[2 * g]), int(perm[2 * g + 1])
            lo, hi = min(c, t), max(c, t)
            w = v.view(1 << lo, 2, 1 << (hi - lo - 1), 2, -1)
            if c < t:
                w[:, 1] = w[:, 1].flip(2)
            else:
                w[:, :, :, 1] = w[:, :, :, 1].flip(1)
    return v


def _basis(n, index):
    v = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    v[index] = 1
    return v


def _qft(n, x):
    """The QFT of |x>: exp(2 pi i x y / 2^n) / 2^(n/2), the product taken modulo 2^n as whole numbers."""
    y = torch.arange(1 << n, dtype=torch.int64, device="cuda")
    turns = ((y * x) & ((1 << n) - 1)).double().mul_(2.0 * math.pi / (1 << n))
    return torch.polar(torch.full_like(turns, 2.0 ** (-n / 2)), turns)


def _grover(n, w, k):
    """Search state after k iterations of phase flip and H (sign flip off |0>) H from the uniform state."""
    t = math.asin(2.0 ** (-n / 2))
    a, b = math.sin((2 * k + 1) * t), math.cos((2 * k + 1) * t) / math.sqrt((1 << n) - 1)
    # the sign of one iteration: H (2|0><0| - 1) H or its negative, by the circuit's own |0> flip
    sign = 1.0 if k % 2 == 0 else _GROVER_SIGN
    v = torch.full((1 << n,), sign * b, dtype=torch.complex128, device="cuda")
    v[w] = sign * a
    return v


# the circuit flips the sign of |0> alone: 1 - 2|0><0|, the negative of 2|0><0| - 1
_GROVER_SIGN = -1.0


def _one(req):
    kind, n, layers, v = req
    if kind == "layered":
        return _layered(n, layers, v, _basis(n, 0))
    return _qft(n, v) if kind == "qft" else _grover(n, v, int(math.pi / 4.0 * math.sqrt(1 << n)))


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return torch.cat([_pairs(_one(r)) for r in _requests(case, seed)])
    if kind == "served":
        states = [_pairs(_one(r)) for r in _requests(case, seed)]
        return {"states": states, "norms": np.ones(len(states)), "argmax": None}
    n = case["n"]
    if kind == "layered":
        return _pairs(_layered(n, case["layers"], seed, _basis(n, 0)))
    if kind == "qft":
        return _pairs(_qft(n, _value(case, seed)))
    if kind == "grover":
        k = case["iterations"] or int(math.pi / 4.0 * math.sqrt(1 << n))
        return _pairs(_grover(n, _value(case, seed), k))
    if kind == "hadamard":
        x = _value(case, seed)
        y = torch.arange(1 << n, dtype=torch.int64, device="cuda") & x
        for sh in (32, 16, 8, 4, 2, 1):
            y ^= y >> sh
        return _pairs((1.0 - 2.0 * (y & 1).double()).mul_(2.0 ** (-n / 2)).to(torch.complex128))
    v = _random_state(n, seed, "cuda")
    if kind == "wrapper":
        if case["precision"] == "f32":
            v = v.float().double()  # the input as the call receives it
        return _layered(n, case["layers"], seed, torch.view_as_complex(v)).cpu().numpy()
    if case["precision"] == "f32":
        v = v.float().double()
    p = v.square().sum(1)
    mask = _read_mask(case)
    bits = [b for b in range(n) if mask >> b & 1]
    probs = p.view((2,) * n).sum([n - 1 - b for b in range(n) if not mask >> b & 1])
    # the amplitudes of the measured branch, rescaled, go where the qubit is 0
    w = v.view(1 << (n // 2), 2, -1, 2)
    p0 = float(p.view(1 << (n // 2), 2, -1)[:, 0].sum())
    after = torch.zeros_like(w)
    after[:, 0] = w[:, 0] / math.sqrt(p0)
    return {"norm": float(p.sum()), "probs": probs.reshape(1 << len(bits)).cpu().numpy(), "argmax": None,
            "top": float(p.max()), "outcome": None, "p": p0, "state": after.reshape(-1, 2)}
