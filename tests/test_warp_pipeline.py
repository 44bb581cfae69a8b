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
    S, prev = S.copy(), 0.0
    for w in words:
        fa, fb, fc, fo = _fields(w)
        b = prev if fb & 1 else S[fb >> 2]
        if fo & 2:
            prev = 1.0 / b
        else:
            prev = (-S[fa >> 2] if fa & 1 else S[fa >> 2]) * b + (prev if fc & 1 else S[fc >> 2])
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
        assert np.array_equal(_thread_loop(ws.encode(ops, [[i] for i in range(len(ops))], 1), S), want)
