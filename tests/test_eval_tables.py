"""The evaluation kernels' tables (namespace eval of a generated header) on
the CPU: rates, tendencies and the dense Jacobian computed from the emitted
numbers, against the mechanism's mass action, for products of many factors
and for thousands of reactions."""

import copy
import re

import numpy as np
import pytest

import large_mechanism
from mkpp_gb300.emitter import cuda_emitter
from mkpp_gb300.emitter.plan import load_raw, reduce_plan


def _tables(plan):
    text = cuda_emitter._eval_tables(plan)
    out = {n: int(v, 0) for n, v in re.findall(r"constexpr (?:int|unsigned) (\w+) = (\w+);", text)}
    for ctype, name, size, body in re.findall(r"const ([\w ]+) (\w+)\[(\d+)\] = \{(.*?)\n\};", text, re.S):
        vals = [x.strip() for x in body.split(",") if x.strip()]
        assert len(vals) == int(size)
        out[name] = [float(x) for x in vals] if ctype == "double" else [int(x) for x in vals]
        if ctype == "unsigned short":
            assert max(out[name]) < 1 << 16
    return out


def _product(T, k, code, y):
    bits = T["LEN_BITS"]
    start, count = code >> bits, code & ((1 << bits) - 1)
    for x in T["factor"][start:start + count]:
        k = k * ((x & (T["POWER"] - 1)) if x & T["POWER"] else y[x])
    return k


def _from_tables(T, ns, k, y):
    q = [_product(T, k[r], T["rate"][r], y) for r in range(len(k))]
    f = [sum(c * q[t] for c, t in zip(T["f_coef"][a:b], T["f_term"][a:b])) for a, b in zip(T["f_ptr"], T["f_ptr"][1:])]
    jac = np.zeros((ns, ns))
    for col in range(ns):
        a, b = T["p_ptr"][col:col + 2]
        d = [_product(T, k[r], code, y) for r, code in zip(T["p_rate"][a:b], T["p_product"][a:b])]
        assert len(d) <= T["MAX_PARTIALS"]
        for row in range(ns):
            a, b = (x >> 2 for x in T["j_ptr"][ns * col + row:ns * col + row + 2])
            jac[row, col] = -sum(c * d[t] for c, t in zip(T["j_coef"][a:b], T["j_term"][a:b]))
    return np.array(f), jac


def _mass_action(raw, k, y):
    ns = len(raw["species"])
    f, jac = np.zeros(ns), np.zeros((ns, ns))
    for r, kr in zip(raw["reactions"], k):
        m = kr * np.prod([y[s] ** p for s, p in r["reactants"]])
        for s, c in r["net"]:
            f[s] += c * m
            for j, p in r["reactants"]:
                jac[s, j] += c * m * p / y[j]
    return f, jac


def _powers():
    """Chapman with O + O2 at 20 and 3 molecules."""
    raw = copy.deepcopy(load_raw("chapman"))
    raw["reactions"][1]["reactants"] = [[0, 20], [1, 3]]
    return raw


@pytest.mark.parametrize("raw, most", [(load_raw("chapman"), 3), (_powers(), 24), (large_mechanism.raw(300), 3)],
                         ids=["chapman", "powers", "split"])
def test_tables_give_mass_action(raw, most):
    plan = reduce_plan(raw)
    T = _tables(plan)
    assert T["RATES"] == len(raw["reactions"]) and 1 << T["LEN_BITS"] > most - 1
    rng = np.random.default_rng(8)
    y, k = rng.uniform(0.5, 1.5, len(raw["species"])), rng.uniform(0.5, 1.5, len(raw["reactions"]))
    for got, want in zip(_from_tables(T, len(y), k, y), _mass_action(raw, k, y)):
        # n terms of products of at most `most` factors: (n + most) eps of the largest sum of magnitudes
        scale = len(k) * 1.5 ** most * most * 2
        np.testing.assert_allclose(got, want, rtol=0, atol=(len(k) + most) * 2.3e-16 * scale)
