"""FP64 layers of unitary, other invertible and singular gates with phases: each gate takes the cheapest form it has
(csrc/lower.cpp layer)."""
import struct
from decimal import Decimal, localcontext

import numpy as np
import pytest

import simulador_quantico_b200 as sq
from tests import plan_emulator as emu
from tests.helpers import random_state
from simulador_quantico_b200 import workloads as wl
from tests.test_lowering import S_GATE, S_HAD, S_REAL, S_ROT, S_SCALE, S_SPLIT, both, stream_units


def gate(kind, rng):
    a, b = rng.uniform(0.2, 1.3), rng.uniform(0.0, 6.0)
    r = np.array([[np.cos(a), -np.sin(a)], [np.sin(a), np.cos(a)]])
    if kind == "invertible":
        r = r @ np.array([[1.0, 0.3], [0.2, -0.7 if b > 3 else 0.9]])
    elif kind == "steep":  # determinant 1e-5 of its entries' squares
        r = r @ np.array([[1.0, 1.0], [1.0, 1.0 + 1e-5]]) / 2
    elif kind == "narrow":  # a first column of 1e-160: in the in-place form two such gates would leave the range
        r = np.array([[1e-160, 1.0], [2e-161, 3.0]])
    elif kind == "singular":
        r = r @ np.array([[0.8, 0.4], [0.6, 0.3]])
    return (r * np.array([1.0, np.exp(1j * b)])).reshape(-1)


def circuit(n, layers, kinds, swaps, seed):
    rng, c = np.random.default_rng(seed), sq.Circuit()
    for k in range(layers):
        for q in range(n):
            c.append_op(q, 0, 0, gate(kinds[(q + k) % len(kinds)], rng))
        for q in range(k % 2 if swaps else n, n - 1, 2):  # relabelings and controlled swaps between layers
            c.append_op(q, 2 << q, (2 << q) * (q % 2), [0, 1, 1, 0])
    return c


def ops_of(plan):
    units, at, out = stream_units(plan)[0], 0, []
    while at < len(units):
        w = [int(x) for x in units[at]]
        out.append((w[0] & 0xFF, w))
        at += w[0] >> 8
    return out


MIXES = {"unitary": ["unitary"], "quarter": ["unitary"] * 3 + ["invertible"], "invertible": ["invertible"],
         "singular": ["unitary", "singular", "invertible"], "steep": ["steep", "unitary"],
         "narrow": ["unitary", "narrow"], "few": ["singular"] + ["unitary"] * 7}


@pytest.mark.parametrize("name", MIXES)
def test_each_gate_for_itself(name):
    n = 13
    ops = ops_of(sq.Plan(circuit(n, 1, MIXES[name], False, 5), n, "f64", fuse=0))
    bits = lambda kind: sum(bin(w[1] & 0xFF).count("1") for k, w in ops if k == kind)
    kinds = [MIXES[name][q % len(MIXES[name])] for q in range(n)]
    singular = kinds.count("singular") + kinds.count("narrow")
    general = singular if 4 * singular > n else 0  # few: a phase gate and a real 2x2 each
    assert bits(S_ROT) == n - singular and bits(S_SPLIT) == general
    assert bits(S_REAL) == singular - general == sum(1 for k, _ in ops if k == S_GATE)


@pytest.mark.parametrize("swaps", [False, True])
@pytest.mark.parametrize("name", MIXES)
def test_mixed_layers(monkeypatch, name, swaps):
    n = 13
    got, want = both(monkeypatch, sq.Plan(circuit(n, 4, MIXES[name], swaps, 7), n, "f64"), "f64", n, seed=n)
    # 52 gates in a row, each a few roundings of 2^-53 of its operands; a steep gate's of terms up to 2^10 of its result
    assert np.abs(got - want).max() <= 1e-12 * max(1.0, np.abs(want).max())


@pytest.mark.gpu
@pytest.mark.parametrize("swaps", [False, True])
@pytest.mark.parametrize("n", [9, 12, 15])
@pytest.mark.parametrize("name", MIXES)
def test_mixed_layers_on_the_device(name, n, swaps):
    sq.init()
    plan = sq.Plan(circuit(n, 4, MIXES[name], swaps, n), n, "f64")
    v = random_state(n, seed=n)
    want = emu.run(plan, "f64", v)
    st = sq.State(n, "f64").upload(v)
    got = st.execute(plan).download()
    plan.status()
    st.free()
    assert np.abs(got - want).max() <= 1e-12 * max(1.0, np.abs(want).max())


def left_out(plan, factors):
    """The plan's one S_SCALE against the exact product of the factors, in units of its last place."""
    scales = [struct.unpack("<d", struct.pack("<II", w[2], w[3]))[0] for k, w in ops_of(plan) if k == S_SCALE]
    assert len(scales) == 1
    with localcontext() as ctx:
        ctx.prec = 60
        want = Decimal(1)
        for f in factors:
            want *= f
        return abs(Decimal(scales[0]) - want) / Decimal(float(np.spacing(abs(scales[0]))))


def test_left_out_hadamard_factors():
    plan = sq.Plan(wl.grover_search(13, 77, 10).build(sq.Circuit()), 13, "f64")
    n = sum(bin(w[1]).count("1") for k, w in ops_of(plan) if k == S_HAD)
    # H's own factor, not the matrix entry's double; rounded once to double, behind at most 300 roundings of
    # 64 bits (2^-11 of a unit each)
    with localcontext() as ctx:
        ctx.prec = 60
        h = Decimal("0.5").sqrt()
    assert n > 200 and left_out(plan, [h] * n) <= Decimal("0.65")


def test_left_out_rotation_factors():
    n, rng, c = 13, np.random.default_rng(8), sq.Circuit()
    for layer in range(8):
        for q in range(n):
            a = rng.uniform(-0.78, 0.78)  # cos is the larger, and positive: no X, no scalar
            c.append_op(q, 0, 0, (np.array([[np.cos(a), -np.sin(a)], [np.sin(a), np.cos(a)]]) * [1, np.exp(0.5j + 0.2j * q)]).reshape(-1))
    plan = sq.Plan(c, n, "f64", fuse=0)
    e, factors = emu.export(plan, "f64"), []
    i, ops = 0, e["ops"]
    units, at, ts = stream_units(plan)[0], 0, []
    while at < len(units):
        w = [int(x) for x in units[at]]
        if w[0] & 0xFF == S_ROT:
            ts += list(units[at + 1:at + (w[0] >> 8)].reshape(-1).view("<f8").reshape(-1, 4)[:, 0])
        at += w[0] >> 8
    with localcontext() as ctx:
        ctx.prec = 60
        while i < len(ops):
            k = bin(int(ops[i]["cm_reg"])).count("1") if ops[i]["kind"] == emu.K_LAYER_SPLIT else 0
            for m in ops[i + 1:i + 1 + k]["m"]:
                d = 1.0 if m[0] * m[3] - m[1] * m[2] >= 0 else -1.0  # a rotation or one times diag(1, -1)
                c0, s0 = Decimal(0.5 * (m[0] + d * m[3])), Decimal(0.5 * (m[2] - d * m[1]))
                t = Decimal(float(ts[len(factors)]))
                factors.append(((c0 * c0 + s0 * s0) / (1 + t * t)).sqrt())
            i += 1 + k
    # each factor to a few units of 64 bits, 104 of them, rounded once to double
    assert len(factors) == len(ts) == n * 8 and left_out(plan, factors) <= Decimal("0.75")
