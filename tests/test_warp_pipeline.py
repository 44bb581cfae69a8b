"""Pipelined warp programs (emitter/warp_schedule.py) on the CPU.

The device loop (csrc/warp_engine.cuh) stores a step's results during the
next step, after which it loads the operands of the step that follows.  Here
that loop runs in plain float64 on encoded words; every slot has to end
bit-identical to the operations in program order, so a value that a schedule
reads from its slot too early, or that ``encode`` takes from the wrong
register or does not store, shows up on random data.  The same for the
sequential words that one thread walks.
"""

import numpy as np
import pytest

from mkpp_gb300.emitter import cuda_emitter
from mkpp_gb300.emitter import warp_schedule as ws
from mkpp_gb300.emitter.plan import load


def _fields(w):
    return [(w >> 16 * f) & 0xFFFF for f in range(4)]


def _device_loop(words, S, lanes):
    S = S.copy()
    steps = [[words[2 * lanes * (s // 2) + 2 * q + s % 2] for q in range(lanes)] for s in range(len(words) // lanes)]
    prev, store = [0.0] * lanes, [None] * lanes

    def operands(s):
        return [[S[x >> 2] for x in _fields(w)[:3]] for w in steps[s]]

    held = operands(0)
    for s, row in enumerate(steps):
        now, out = [0.0] * lanes, [None] * lanes
        for q, w in enumerate(row):
            fa, fb, fc, fo = _fields(w)
            a, b, c = held[q]
            b = prev[q] if fb & 1 else b
            c = prev[q] if fc & 1 else c
            now[q] = 1.0 / b if fo & 2 else (-a if fa & 1 else a) * b + c
            out[q] = None if fo & 1 else fo >> 2
        for q in range(lanes):
            if store[q] is not None:
                S[store[q]] = prev[q]
        if s + 1 < len(steps):
            held = operands(s + 1)
        prev, store = now, out
    for q in range(lanes):
        if store[q] is not None:
            S[store[q]] = prev[q]
    return S


def _thread_loop(words, S):
    """run_program: the next word's operands are loaded before a result is
    stored."""
    S, prev = S.copy(), 0.0
    held = [S[x >> 2] for x in _fields(words[0])[:3]]
    for n, w in enumerate(words):
        fa, fb, fc, fo = _fields(w)
        a, b, c = held
        if n + 1 < len(words):
            held = [S[x >> 2] for x in _fields(words[n + 1])[:3]]
        b = prev if fb & 1 else b
        prev = 1.0 / b if fo & 2 else (-a if fa & 1 else a) * b + (prev if fc & 1 else c)
        if not fo & 1:
            S[fo >> 2] = prev
    return S


def _in_order(ops, S):
    S = S.copy()
    for kind, out, a, b, c, neg in ops:
        S[out] = 1.0 / S[out] if kind == ws.RCP else (-S[a] if neg else S[a]) * S[b] + S[c]
    return S


@pytest.mark.parametrize("mech", ["chapman", "small_strato", "small_strato_rodas3", "saprc99_mini", "saprc99"])
def test_device_loop_ends_as_program_order(mech):
    plan = load(mech)
    cuda_emitter.emit_mechanism(plan)
    progs, _, info = plan._coop_programs
    rng = np.random.default_rng(11)
    for ops in [*progs, [op for p in progs for op in p]]:
        S = rng.uniform(0.5, 1.5, info["slots"])
        S[info["CB"]:info["CB"] + 3] = (-0.0, 0.0, 1.0)
        want = _in_order(ops, S)
        assert np.isfinite(want).all()
        for lanes in (1, 8, 16, 32):
            steps = ws.pipeline(ops, lanes)
            assert sorted(i for row in steps for i in row if i is not None) == list(range(len(ops)))
            if lanes > 1:
                assert np.array_equal(_device_loop(ws.encode(ops, steps, lanes), S, lanes), want)
        assert np.array_equal(_thread_loop(ws.encode(ops, ws.sequential(ops), 1), S), want)


@pytest.mark.parametrize("mech", ["chapman", "small_strato_rodas3", "saprc99_mini", "saprc99"])
def test_warp_sweeps_equal_the_sequential_programs(mech):
    """The warps' adjoint and tangent programs (more temporaries, the
    attempt's constants) leave the results of the sequential ones, bit for
    bit, in order and through the device loop."""
    plan = load(mech)
    cuda_emitter.emit_mechanism(plan)
    _, _, info = plan._coop_programs
    warp = plan._sweeps
    tab = plan.tableau
    nv, nr, stages = plan.n_var, len(plan.reactions), int(tab["stages"])
    A, C, M, NewF = tab["A"], tab["C"], tab["M"], tab["NewF"]
    K0, Y, KT, CB = info["K0"], info["Y"], info["KT"], info["CB"]
    rng = np.random.default_rng(3)
    base = max(w["slots"] for w in warp.values())   # the sequential layouts follow the warps' slots
    size = 2 * base

    # Sequential adjoint on its own layout, with the warp's literal slots.
    literals = {**info["literals"], **warp["adj"]["extra"]}
    adj = cuda_emitter._adjoint_layout(base, nv, nr, stages)
    P = ws.Program(CB, CB + 1, CB + 2, lambda v: literals[float(v)])
    cuda_emitter._adjoint_program(plan, P, nv, stages, A, C, M, NewF, K0, Y, KT, adj, info["cterm_slot"])
    seq_t = cuda_emitter._tlm_build(plan, nv, stages, A, C, M, NewF, K0, Y, KT, base)

    def store(extra):
        S = np.zeros(size + base)
        S[:info["slots"]] = np.random.default_rng(4).uniform(0.5, 1.5, info["slots"])
        S[CB:CB + 3] = (-0.0, 0.0, 1.0)
        for v, slot in {**info["literals"], **extra}.items():
            S[slot] = v
        return S

    for name, ops, seq, ins, outs in (
            ("adj", P.ops, adj, (("LAM", nv),), (("LAM", nv), ("KB", nr))),
            ("tlm", seq_t["ops"], seq_t["L"], (("DYT", nv), ("DKR", nr)), (("DYT", nv),))):
        w = warp[name]
        given = {key: rng.uniform(-1.0, 1.0, n) for key, n in ins}
        one, many = store(warp["adj"]["extra"] if name == "adj" else {}), store(w["extra"])
        if name == "tlm":
            t0 = seq_t["L"]["TCB"]
            one[t0:t0 + 3] = (-0.0, 0.0, 1.0)
            for key, slot in seq_t["cterm"].items():
                one[slot] = one[info["cterm_slot"][key]]
            for v, slot in seq_t["literals"].items():
                one[slot] = v
        for key, n in ins:
            one[seq[key]:seq[key] + n] = given[key]
            many[w["L"][key]:w["L"][key] + n] = given[key]
        with np.errstate(all="ignore"):          # idle words compute on slot 0
            threaded = _thread_loop(ws.encode(ops, ws.sequential(ops), 1), one)
        one = _in_order(ops, one)
        for key, n in outs:
            assert np.array_equal(threaded[seq[key]:seq[key] + n], one[seq[key]:seq[key] + n])
        assert max(max(op[1:5]) for op in w["ops"]) < w["slots"]
        looped = _device_loop(ws.encode(w["ops"], w["steps"]), many, ws.LANES)
        for key, n in outs:
            want = one[seq[key]:seq[key] + n]
            assert np.isfinite(want).all() and np.any(want != 0.0)
            assert np.array_equal(looped[w["L"][key]:w["L"][key] + n], want)
