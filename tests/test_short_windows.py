"""One-warp plans (warp_bits 0): short stream windows for states of several tiles, long ones for one tile."""
import numpy as np
import pytest

import simulador_quantico_b200 as sq
from simulador_quantico_b200 import workloads as wl
from tests import plan_emulator as emu
from tests.helpers import random_gate_circuit_spec, random_state
from tests.test_lowering import S_END, S_NEXT, both, stream_units


def plan_of(name, n, prec, **kw):
    spec = random_gate_circuit_spec(n, 200, seed=n) if name == "gates" else wl.random_layered(n, 20, n)
    return sq.Plan(spec.build(sq.Circuit()), n, prec, warp_bits=0, renorm_every=0, **kw)


@pytest.mark.parametrize("name", ["gates", "layered"])
@pytest.mark.parametrize("prec,n", [("f64", 9), ("f64", 10), ("f64", 13), ("f32", 10), ("f32", 11), ("f32", 13)])
def test_windows(monkeypatch, name, prec, n):
    plan = plan_of(name, n, prec)
    units, tiles = stream_units(plan)
    short = n > (9 if prec == "f64" else 10)
    at = start = longest = 0
    while at < len(units):
        kind, step = int(units[at][0]) & 0xFF, int(units[at][0]) >> 8
        at += step
        if kind in (S_NEXT, S_END):
            longest, start = max(longest, at - start), at
    assert longest <= (64 if short else 176) and (short or longest > 64)
    assert (tiles["ld_tstep"][:, 7] == 16 * (64 if short else 176)).all()
    got, want = both(monkeypatch, plan, prec, n, seed=n)
    # at most 400 gates in a row, emulated in FP64 both ways
    assert np.abs(got - want).max() <= 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("chained", [1, 0])
@pytest.mark.parametrize("name", ["gates", "layered"])
@pytest.mark.parametrize("prec,n", [("f64", 9), ("f64", 10), ("f64", 14), ("f32", 10), ("f32", 11), ("f32", 14)])
def test_windows_on_the_device(name, prec, n, chained):
    sq.init()
    plan = plan_of(name, n, prec, chained=chained)
    v = random_state(n, seed=n, dtype=np.complex128 if prec == "f64" else np.complex64)
    want = emu.run(plan, prec, v.astype(np.complex128))
    st = sq.State(n, prec).upload(v)
    got = st.execute(plan).download()
    plan.status()
    st.free()
    assert np.abs(got - want).max() <= (1e-12 if prec == "f64" else 2e-5)
