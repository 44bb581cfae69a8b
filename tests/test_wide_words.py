"""Programs with slots beyond 14 bits (CPU).

Their words have four 32-bit fields.  The encoded words run through the
device loops' order of loads and stores, as in test_warp_pipeline.py, and a
whole mechanism of that size runs its table-driven attempt on the host."""

import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

import hostsim_lib
import large_mechanism
from mkpp_gb300.emitter import cuda_emitter
from mkpp_gb300.emitter import warp_schedule as ws
from mkpp_gb300.emitter.plan import load

UP = 1 << 15


def _fields(w):
    return [(w >> 32 * f) & 0xFFFFFFFF for f in range(4)]


def _run(words, S, lanes):
    """The loops of warp_engine.cuh (lanes > 1) and run_program (one lane):
    a step's results are stored after the next operands are loaded (one lane)
    or before (a warp, whose loads run a step later)."""
    S = S.copy()
    steps = [words[i:i + lanes] for i in range(0, len(words), lanes)]
    prev, store = [0.0] * lanes, [None] * lanes

    def operands(s):
        return [[S[x >> 2] for x in _fields(w)[:3]] for w in steps[s]]

    held = operands(0)
    for s, row in enumerate(steps):
        now, out = [], []
        for q, w in enumerate(row):
            fa, fb, fc, fo = _fields(w)
            a, b, c = held[q]
            b = prev[q] if fb & 1 else b
            c = prev[q] if fc & 1 else c
            now.append(1.0 / b if fo & 2 else (-a if fa & 1 else a) * b + c)
            out.append(None if fo & 1 else fo >> 2)
        if lanes > 1:
            for q, at in enumerate(store):
                if at is not None:
                    S[at] = prev[q]
        if s + 1 < len(steps):
            held = operands(s + 1)
        if lanes == 1 and out[0] is not None:
            S[out[0]] = now[0]
        prev, store = now, out
    if lanes > 1:
        for q, at in enumerate(store):
            if at is not None:
                S[at] = prev[q]
    return S


def _in_order(ops, S):
    S = S.copy()
    for kind, out, a, b, c, neg in ops:
        S[out] = 1.0 / S[out] if kind == ws.RCP else (-S[a] if neg else S[a]) * S[b] + S[c]
    return S


@pytest.mark.parametrize("mech", ["chapman", "saprc99_mini"])
def test_wide_words_end_as_program_order(mech):
    plan = load(mech)
    cuda_emitter.emit_mechanism(plan)
    progs, _, info = plan._coop_programs
    # (A reciprocal names its slot alone.)
    ops = [(op[0], op[1] + UP, *(0 if op[0] == ws.RCP else x + UP for x in op[2:5]), op[5]) for p in progs for op in p]
    assert ws.is_wide(ops) and not ws.is_wide(*progs)
    S = np.concatenate([np.ones(UP), np.random.default_rng(1).uniform(0.5, 1.5, info["slots"])])
    S[UP + info["CB"]:UP + info["CB"] + 3] = (-0.0, 0.0, 1.0)
    want = _in_order(ops, S)
    assert np.isfinite(want).all()
    for lanes in (8, 32):
        words = ws.encode(ops, ws.pipeline(ops, lanes), lanes, ws.WIDE)
        assert np.array_equal(_run(words, S, lanes), want)
    words = ws.encode(ops, ws.sequential(ops), 1, ws.WIDE)
    assert np.array_equal(_run(words, S, 1), want)
    for w in words[:64]:
        kind, *fields = ws.decode(w, ws.WIDE)
        if kind:
            assert ws.encode([(kind, *fields)], [[0]], 1, ws.WIDE) == [w] or -1 in fields


def _xfma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def test_a_mechanism_with_wide_slots_runs_its_programs(tmp_path):
    """The emitted attempt and tangent of a mechanism of 4000 reactions, built
    for the host, leave every slot as their operations in program order with
    exactly rounded fma do, bit for bit."""
    plan = large_mechanism.write_header(tmp_path, 1000)
    progs, _, info = plan._coop_programs
    text = (tmp_path / f"{large_mechanism.NAME}.cuh").read_text()
    assert "mkpp::WideWord attempt_prog[" in text and "mkpp::WideWord tlm_prog[" in text
    lib = hostsim_lib.compile(tmp_path, large_mechanism.NAME, tmp_path)
    L = hostsim_lib.layout(lib)
    k = np.tile(np.array([1.0e-11, 6.0e-34 * 2.4e19, 4.0e-4, 8.0e-12]) / 1000, 1000)
    y = np.array([1.0e6, 5.0e18, 5.0e11])[plan.var_phys]
    h = 1.0e-2
    S = np.zeros(L["NSLOTS"])
    S[L["Y"]:L["Y"] + L["NV"]] = y
    st = C.c_int(0)
    lib.hostsim_attempt(S.ctypes.data, k.ctypes.data, h, C.byref(st))
    P = np.zeros(L["NSLOTS"])
    P[info["Y"]:info["Y"] + L["NV"]] = y
    P[info["KT"]:info["KT"] + len(k)] = k
    CB = info["CB"]
    P[CB:CB + 4] = (-0.0, 0.0, 1.0, 1.0 / (plan.tableau["Gamma"][0] * h))
    for (s_, j), slot in info["cterm_slot"].items():
        P[slot] = info["C"][(s_ - 1) * (s_ - 2) // 2 + j - 1] / h
    for v, slot in info["literals"].items():
        P[slot] = v
    for ops in progs:
        for kind, out, a, b, c, neg in ops:
            P[out] = 1.0 / P[out] if kind == ws.RCP else _xfma(-P[a] if neg else P[a], P[b], P[c])
    K = slice(L["K0"], L["K0"] + L["NSTAGE"] * L["NV"])
    assert st.value == 0 and np.all(P[K] != 0.0)
    assert np.array_equal(S[K], P[K])
    assert np.array_equal(S[:len(plan.lu_slots)], P[:len(plan.lu_slots)])
    # The tangent is linear in (dy, dk): powers of two scale it exactly.
    one, _, _ = hostsim_lib.tangent_step(lib, y, k, h, 1e-3 * y, 1e-3 * k)
    two, _, _ = hostsim_lib.tangent_step(lib, y, k, h, 2e-3 * y, 2e-3 * k)
    assert np.all(one != 0.0) and np.array_equal(2.0 * one, two)
