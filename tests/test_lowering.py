"""The device stream against the plan it is lowered from (CPU only).

Decodes a plan's stream (csrc/hgm_internal.h, "device stream") back into plain
records -- every window, transpose and op, each rotation as the matrix it
stands for -- and emulates both forms on the same random state.
"""
import ctypes as C
import struct

import numpy as np
import pytest

import simulador_quantico_b200 as sq
from simulador_quantico_b200 import workloads as wl
from simulador_quantico_b200._lib import check, lib
from tests import plan_emulator as emu
from tests.helpers import random_gate_circuit_spec, random_state

(S_END, S_NEXT, S_TRANS, S_ROT, S_HAD, S_REAL, S_DENSE, S_XSET, S_CSWAP, S_SCALE, S_PHASES, S_TERMS, S_GATE,
 S_SPLIT) = range(14)
WINDOW = 176
plan_export = emu.export


TILE_DT = np.dtype([("ld_gbit", "i1", 16), ("st_gbit", "i1", 16), ("run_pos", "i1", 16), ("run_len", "i1", 16),
                    ("ld_tstep", "<u4", 8), ("stream", "<u8"), ("units", "<i4", 2), ("n", "<i4"), ("k", "<i4"),
                    ("flags", "<i4"), ("nruns", "<i4"), ("ctl", "<u8", 3), ("pass", "<i4"), ("pairs", "<i4")])
PERMUTE, PERM_BITS = 4, 10


def stream_units(plan):
    p, n, t, nt = C.c_void_p(), C.c_int64(), C.c_void_p(), C.c_int64()
    check(lib.hgm_plan_stream(plan.h, C.byref(p), C.byref(n), C.byref(t), C.byref(nt)))
    return (np.frombuffer(C.string_at(p, n.value), "<u4").reshape(-1, 4),
            np.frombuffer(C.string_at(t, nt.value * TILE_DT.itemsize), TILE_DT))


def permuted(tile, v):
    """A permutation pass on the state v, as the kernel walks it: sub-tile u to the place of its partner."""
    n = int(tile["n"])
    gb, to = [int(x) for x in tile["ld_gbit"][:PERM_BITS]], [int(x) for x in tile["st_gbit"][:PERM_BITS]]
    pairs = tile["ld_tstep"].view("i1").astype(int)[:2 * int(tile["pairs"])].reshape(-1, 2)
    assert not tile["units"].any() and not tile["stream"]  # the kernels fetch nothing for it
    j = np.arange(1 << PERM_BITS)
    place = sum(((j >> q) & 1) << gb[q] for q in range(PERM_BITS))
    moved = sum(((j >> q) & 1) << to[q] for q in range(PERM_BITS))
    assert sorted(moved) == list(range(1 << PERM_BITS))
    u = np.arange(1 << (n - PERM_BITS))
    base, shift = np.zeros_like(u), 0
    for k in range(int(tile["nruns"])):
        ln = int(tile["run_len"][k])
        base |= ((u >> shift) & ((1 << ln) - 1)) << int(tile["run_pos"][k])
        shift += ln
    assert shift == n - PERM_BITS
    other = base.copy()
    for a, b in pairs:
        x = ((other >> a) ^ (other >> b)) & 1
        other ^= (x << a) | (x << b)
    out = np.full_like(v, np.nan)
    out[other[:, None] | place[moved][None, :]] = v[base[:, None] | place[None, :]]
    return out


def lowered_export(plan, prec):
    """emu.export's form of what the stream says."""
    e = plan_export(plan, prec)
    units, tiles = stream_units(plan)
    real, esz = ("<f8", 16) if prec == "f64" else ("<f4", 8)
    odt = e["ops"].dtype
    W = e["W"]
    steps = tiles[tiles["flags"] == 0]
    assert (np.diff(steps["pass"]) > 0).all()
    recs, phases, passes = [], [], e["passes"][steps["pass"]].copy()
    at = 0

    def vals(u0, u1):
        return units[u0:u1].reshape(-1).view(real).astype(np.float64)

    def rec(kind, tpos, cm=0, cv=0, m=(0,) * 8, thr=(0, 0), glob=(0, 0)):
        r = np.zeros(1, odt)[0]
        r["kind"], r["tpos"], r["tpos2"], r["cm_reg"], r["cv_reg"] = kind, tpos, tpos, cm, cv
        r["cm_thr"], r["cv_thr"] = thr
        r["cm_glob"], r["cv_glob"] = glob
        r["m"] = m
        recs.append(r)

    def dense(b, mm):
        mm = np.asarray(mm, np.complex128).reshape(4)
        rec(emu.K_DENSE, b, m=np.stack([mm.real, mm.imag], 1).reshape(-1))

    for pi in range(len(passes)):
        R = int(passes[pi]["k"]) - 5 - W
        pad = lambda j: (j + (j >> R)) * esz
        layout_of = {}
        for li, lay in enumerate(e["layouts"]):
            layout_of[tuple(pad(1 << int(lay[k])) for k in range(5 + W + R))] = li
        passes[pi]["phase_begin"] = len(phases)
        layout, begin, xwarp = int(passes[pi]["load_layout"]), len(recs), 0
        assert int(steps[pi]["stream"]) == 16 * at and not units[at][0] & 0xFF == S_NEXT
        window, named = at, []
        sizes = []
        while True:
            w = [int(x) for x in units[at]]
            kind, n = w[0] & 0xFF, w[0] >> 8
            assert n >= 1
            if kind in (S_END, S_NEXT):
                sizes.append(at + 1 - window)
                assert sizes[-1] <= WINDOW
                named.append(w[1])
                window = at + 1
            if kind == S_END:
                at += 1
                break
            body = at + 1
            if kind == S_TRANS:
                old = [int(x) for x in units[at + 1]] + [w[2]]
                new = [int(x) for x in units[at + 2]] + [w[3]]
                thr = [int(x) for x in units[at + 3:at + 5].reshape(-1)]
                assert tuple(old[:R]) == tuple(pad(1 << int(p)) for p in e["layouts"][layout][5 + W:5 + W + R])
                phases.append((layout, begin, len(recs), xwarp))
                layout, begin, xwarp = layout_of[tuple(thr[:5 + W] + new[:R])], len(recs), int(bool(w[1] & 2))
            elif kind in (S_ROT, S_SPLIT, S_REAL, S_DENSE):
                per = {S_ROT: 4, S_SPLIT: 8, S_REAL: 4, S_DENSE: 8}[kind]
                v = vals(body, at + n)
                bits = [b for b in range(R) if (w[1] >> b) & 1]
                if kind == S_SPLIT:
                    rec(emu.K_LAYER_SPLIT, 0, w[1], w[1])
                for k, b in enumerate(bits):
                    g = v[k * per:(k + 1) * per]
                    if kind == S_ROT:
                        # y' = p y; x1 = x + u y'; y1 = y' + t x1; then X
                        t, u, p = g[0], g[1], g[2] + 1j * g[3]
                        mm = np.array([[1, u * p], [t, (1 + u * t) * p]])
                        dense(b, mm[::-1] if (w[1] >> (8 + b)) & 1 else mm)
                    elif kind == S_SPLIT:
                        rec(emu.K_DENSE, b, m=g)
                    elif kind == S_REAL:
                        dense(b, g)
                    else:
                        dense(b, g[0::2] + 1j * g[1::2])
            elif kind == S_HAD:
                for b in range(R):
                    if (w[1] >> b) & 1:
                        dense(b, [1, 1, 1, -1])
            elif kind == S_XSET:
                words = np.concatenate([units[at][2:], units[body:at + n].reshape(-1)])[:w[1]]
                for word in words:
                    t, ck, cb, cv = struct.unpack("4B", struct.pack("<I", int(word)))
                    rec(emu.K_SWAP, t, thr=(1 << cb, cv << cb) if ck == emu.XSET_CTRL_THREAD else (0, 0),
                        glob=(1 << cb, cv << cb) if ck == emu.XSET_CTRL_GLOBAL else (0, 0))
            elif kind == S_CSWAP:
                rec(emu.K_SWAP, w[1] & 0xFFFF, 1 << (w[1] >> 16), w[2] << (w[1] >> 16))
            elif kind == S_SCALE:
                f = struct.unpack("<d", struct.pack("<II", w[2], w[3]))[0]
                rec(emu.K_DIAG, 0, m=[f, 0, 0, 0, 0, 0, f, 0])
            elif kind in (S_PHASES, S_TERMS):
                counts = units[at + 1].tobytes()
                total = sum(counts)
                head = np.zeros(1, odt)[0]
                head["kind"], head["cm_reg"], head["cv_reg"] = emu.K_PHASE_BLOCK, w[1], w[2]
                raw = (counts + units[at + 2].tobytes()[:8]).ljust(head["m"].nbytes, b"\0")
                head["m"] = np.frombuffer(raw, real)
                hi = len(recs)
                recs.append(head)
                if kind == S_PHASES:
                    size = 16 if prec == "f32" else 32
                    data = units[at + 3:].tobytes()[:total * size]
                    per = odt.itemsize // size
                    for k in range(0, total, per):
                        chunk = data[k * size:(k + per) * size].ljust(odt.itemsize, b"\0")
                        recs.append(np.frombuffer(chunk, odt)[0])
                else:
                    tu = 2 + (1 if prec == "f32" else 2)
                    for k in range(total):
                        u = at + 3 + k * tu
                        f = vals(u + 2, u + tu)
                        g = units[u + 1].view("<u8")
                        rec(emu.K_DIAG, int(units[u][2]), m=[f[0], f[1], 0, 0, 0, 0, f[2], f[3]],
                            thr=(int(units[u][0]), int(units[u][1])), glob=(int(g[0]), int(g[1])))
                assert bool(w[1] & 1) == bool(w[3])
                tab = vals(at + w[3], at + n) if w[3] else np.tile([1.0, 0.0], 1 << R)
                if w[1] & emu.PB_GATED or w[3]:
                    # a table of ones is left out; the emulator's gated form wants it
                    head["cm_reg"] |= 1
                    recs[hi] = head
                    assert len(tab) == 2 << R
                    for q in range((1 << R) // 4):
                        rec(0, 0, m=tab[8 * q:8 * q + 8])
                recs[hi]["tpos"] = len(recs) - hi - 1
            elif kind == S_GATE:
                g = units[at + 2].view("<u8")
                m = vals(at + 3, at + n) if n > 3 else [0, 0, 1, 0, 1, 0, 0, 0]
                rec(w[1] & 0xFF, w[1] >> 8, w[2], w[3], m, thr=(int(units[at + 1][0]), int(units[at + 1][1])),
                    glob=(int(g[0]), int(g[1])))
            else:
                assert kind == S_NEXT and n == 1
            at += n
        # each S_NEXT names the window after the one it enters
        assert named == [sizes[k + 2] if k + 2 < len(sizes) else 0 for k in range(len(sizes) - 1)] + [0]
        phases.append((layout, begin, len(recs), xwarp))
        passes[pi]["phase_end"] = len(phases)
        assert list(steps[pi]["units"]) == (sizes + [0])[:2]
        passes[pi]["store_layout"], passes[pi]["store_xwarp"] = layout, 1
        passes[pi]["st_gbit"] = steps[pi]["st_gbit"]
    assert at == len(units)
    ph = np.array(phases, emu.PHASE_DT) if phases else np.zeros(0, emu.PHASE_DT)
    ops = np.array(recs, odt) if recs else np.zeros(0, odt)
    return dict(e, passes=passes, phases=ph, ops=ops)


def both(monkeypatch, plan, prec, n, seed):
    v = random_state(n, seed=seed, dtype=np.complex128)
    want = emu.run(plan, prec, v)
    monkeypatch.setattr(emu, "export", lowered_export)
    got = emu.run(plan, prec, v)
    tiles = stream_units(plan)[1]
    assert not (tiles["flags"][:-1] & PERMUTE).any()
    return (permuted(tiles[-1], got) if tiles["flags"][-1] & PERMUTE else got), want


def chain_of_phases(n, depth):
    """Many diagonal gates on every pair of bits, some of them not pure phases: phase blocks larger than a window."""
    c = sq.Circuit()
    rng = np.random.default_rng(n)
    for d in range(depth):
        for t in range(n):
            for k in range(n):
                if k != t:
                    z = np.exp(1j * rng.uniform(0, 6, 2)) * (rng.uniform(0.9, 1.1, 2) if d % 2 else 1.0)
                    c.append_op(t, 1 << k, rng.integers(2) << k, [z[0], 0, 0, z[1]])
    return c


def odd_gates(n, prec):
    """Single-qubit gates that no rotation form covers, beside ones at its edges."""
    c = sq.Circuit()
    r = lambda a: [np.cos(a), -np.sin(a), np.sin(a), np.cos(a)]
    ph = lambda a: np.exp(1j * a)
    mats = [r(np.pi / 4), r(-np.pi / 4), r(np.pi / 2 - 1e-9), r(1e-9), r(3.0), [0.3, 0.9, -0.2, 0.5],
            [3.0, -4.0, 4.0, 3.0], [0.6, 0.8, 0.8, -0.6], [0.8, 0.6, 0.6, -0.8]]
    if prec == "f64":  # factors that leave the range a factor is left out in
        mats += [[a, a, a, -a] for a in (1e-150, 1e150)]
    for k, m in enumerate(mats):
        for t in range(n):
            c.append_op(t, 0, 0, [m[0], m[1] * ph(0.3 * t + k), m[2], m[3] * ph(0.3 * t + k)] if (k + t) % 2 else m)
        for t in range(0, n - 1, 2):
            c.append_op(t, 2 << t, (2 << t) if k % 2 else 0, [0, 1, 1, 0])
    return c


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("name", ["gates", "layered", "deep", "qft", "grover", "hadamard", "phases", "odd"])
def test_stream_is_the_plan(monkeypatch, name, prec):
    n = {"deep": 12, "qft": 15, "grover": 13}.get(name, 13)
    if name == "phases":
        c = chain_of_phases(n, 3)
    elif name == "odd":
        c = odd_gates(n, prec)
    else:
        spec = {"gates": lambda: random_gate_circuit_spec(n, 150, seed=9), "layered": lambda: wl.random_layered(n, 5, 4),
                "deep": lambda: wl.random_layered(n, 20, 6), "qft": lambda: wl.qft(n),
                "grover": lambda: wl.grover_search(n, 77, 5), "hadamard": lambda: wl.hadamard_benchmark(n, 3)}[name]()
        c = spec.build(sq.Circuit())
    plan = sq.Plan(c, n, prec)
    got, want = both(monkeypatch, plan, prec, n, seed=n)
    # FP32 streams hold the records' own values; FP64 rotations are other
    # roundings of the same matrices; the emulation, in FP64, groups the
    # products of both in other ways: at most 300 gates in a row here
    scale = max(1.0, np.abs(want).max())
    assert np.abs(got - want).max() <= 1e-12 * scale


def swap_ending(n, pairs, seed):
    """Gates, then swaps of the given pairs of index bits."""
    c = random_gate_circuit_spec(n, 40, seed=seed).build(sq.Circuit())
    for a, b in pairs:
        for ctl, t in ((a, b), (b, a), (a, b)):
            c.append_op(t, 1 << ctl, 1 << ctl, [0, 1, 1, 0])
    return c


SWAPS = [(17, [(q, 16 - q) for q in range(8)]), (18, [(q, 17 - q) for q in range(9)]),
         (19, [(0, 18), (1, 2), (3, 9), (4, 17), (5, 16), (6, 15), (7, 14)]), (20, [(q, 19 - q) for q in range(10)]),
         (17, [(0, 1), (2, 3), (4, 16), (5, 15), (6, 14), (7, 13), (8, 12), (9, 11)]), (20, [(q + 4, 19 - q) for q in range(8)])]


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("n,pairs", SWAPS)
def test_final_swaps(monkeypatch, n, pairs, prec):
    plan = sq.Plan(swap_ending(n, pairs, n), n, prec)
    got, want = both(monkeypatch, plan, prec, n, seed=n)
    assert np.abs(got - want).max() <= 1e-12


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_qft_ends_in_one_permutation(prec):
    """From 15 qubits the reversal's passes become one; below, and where the pairs cannot be split, the CNOTs stay."""
    for n in range(12, 29):
        plan = sq.Plan(wl.qft(n).build(sq.Circuit()), n, prec)
        flags = stream_units(plan)[1]["flags"]
        assert (flags == PERMUTE).sum() == (1 if n >= (15 if prec == "f32" else 14) else 0)
        assert len(flags) <= plan.stats()["passes"]


@pytest.mark.gpu
@pytest.mark.parametrize("chained", [1, 0])
@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("n,pairs", SWAPS)
def test_final_swaps_on_the_device(n, pairs, prec, chained):
    sq.init()
    plan = sq.Plan(swap_ending(n, pairs, n), n, prec, chained=chained, renorm_every=3 if prec == "f32" else 0)
    v = random_state(n, seed=n, dtype=np.complex128 if prec == "f64" else np.complex64)
    want = v.astype(np.complex128)
    for _ in range(2):
        want = emu.run(plan, prec, want)
    st = sq.State(n, prec).upload(v)
    got = st.execute(plan, 2).download()
    plan.status()
    st.free()
    assert np.abs(got - want).max() <= (1e-12 if prec == "f64" else 2e-5)


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("name,n", [("phases", 13), ("phases", 16), ("odd", 9), ("odd", 12), ("odd", 15), ("deep", 12),
                                    ("deep", 14)])
def test_stream_on_the_device(name, n, prec):
    """Ops larger than a window, tiles of many windows, rotations at the edges of their form, against the
    emulated plan."""
    sq.init()
    if name == "phases":
        c = chain_of_phases(n, 3)
    elif name == "odd":
        c = odd_gates(n, prec)
    else:
        c = wl.random_layered(n, 40, n).build(sq.Circuit())
    plan = sq.Plan(c, n, prec, renorm_every=0)
    dt = np.complex128 if prec == "f64" else np.complex64
    v = random_state(n, seed=n, dtype=dt)
    want = emu.run(plan, prec, v.astype(np.complex128))
    st = sq.State(n, prec).upload(v)
    got = st.execute(plan).download()
    plan.status()
    st.free()
    scale = max(1.0, np.abs(want).max())
    assert np.abs(got - want).max() <= (1e-12 if prec == "f64" else 2e-5) * scale
