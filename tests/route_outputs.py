"""Outputs of one mechanism's calls in a process of its own, for
test_gpu_routes.py: python route_outputs.py WHAT MECH CELLS DT OUT.npz.  With
MKPP_COOP_CELLS=0 in the environment every call runs on lanes; otherwise
these few cells run on whole warps.  Launch settings are the library's
defaults, whatever other tests left in theirs."""

import sys
from pathlib import Path

import numpy as np

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))


def inputs(mech, cells):
    import torch

    from mkpp_gb300 import workloads
    from mkpp_gb300.api import DeviceSolver

    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    w = workloads.make(mech, cells, seed=5)
    w.conc[1, cells // 2] = np.nan
    s = DeviceSolver(mech)
    conc = d(w.conc)
    k, status = s.rate_constants(conc, d(w.temp), d(w.rho), d(w.rh), None, d(w.param))
    assert int(status[cells // 2]) != 0
    return s, conc, k, status


def integrations(mech, cells, dt):
    """The persistent form in cell order and in another one, over two host
    steps with carried step sizes, and capped; the plain form."""
    import torch

    s, start, k, status = inputs(mech, cells)
    order = torch.from_numpy(np.random.default_rng(2).permutation(cells).astype(np.int32)).cuda()
    out = {}
    for name, kw in {"plain": {"mode": "plain"}, "cells": {}, "order": {"order": order}, "capped": {"max_attempts": 4},
                     "carry": {"steps": 2, "dt_carry": torch.zeros(cells, dtype=torch.float64, device="cuda")}}.items():
        conc, st = start.clone(), status.clone()
        acc, rej = (torch.full((cells,), 77, dtype=torch.int32, device="cuda") for _ in range(2))
        s.integrate_k(conc, k, dt, status=st, accepted=acc, rejected=rej, **kw)
        out |= {f"{name}_{i}": x for i, x in enumerate((conc, st, acc, rej, kw.get("dt_carry")))}
    return out


def sweeps(mech, cells, dt):
    """Checkpointed forward, adjoint and tangent: every cell recorded, and a
    checkpoint that most cells outgrow.  The cell that is not finite is
    skipped."""
    import ctypes as C

    import torch

    from mkpp_gb300.adjoint import Checkpoints

    s, start, k, flagged = inputs(mech, cells)
    rng = np.random.default_rng(7)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    lam, dc, dk = (d(rng.standard_normal(x.shape)) for x in (start, start, k))
    out = {}
    for cap in (64, 8):
        ck = Checkpoints(mech, cells, cap, "cuda")
        ck.y.zero_()
        ck.h.zero_()
        conc, status = start.clone(), flagged.clone()
        acc, rej = (torch.full((cells,), 77, dtype=torch.int32, device="cuda") for _ in range(2))
        p = lambda x: C.c_void_p(x.data_ptr())  # noqa: E731
        assert ck.lib.mkpp_gpu_integrate_checkpoint(
            cells, p(conc), p(k), dt, s.default_seed, 20000, cap, p(ck.y), p(ck.h), p(ck.count), p(status), p(acc),
            p(rej), p(ck.ws), ck.ws.numel(), ck._stream()) == 0
        gc, gk = ck.adjoint(k, lam)
        t = [ck.tangent(k, dc * start, dk * k), ck.tangent(k, dc * start)]
        out |= {f"cap{cap}_{i}": x for i, x in enumerate(
            (conc, status, acc, rej, ck.count, ck.y, ck.h, gc, gk, *t))}
    return out


def parking(mech, cells, dt):
    """Persistent calls on lanes that park cells (and how many): after one
    attempt, from the 16th attempt on in the tail, over two host steps with
    carried step sizes; and none parked."""
    import torch

    s, start, k, status = inputs(mech, cells)
    out = {}
    for name, after, tail in (("none", 0, 0), ("first", 1, 0), ("tail", 0, 16)):
        s.set_tuning(defer_after=after)
        s.set_tail_parking(tail)
        for steps in (1, 2):
            conc, st = start.clone(), status.clone()
            carry = torch.zeros(cells, dtype=torch.float64, device="cuda")
            acc, rej = (torch.zeros(cells, dtype=torch.int32, device="cuda") for _ in range(2))
            s.integrate_k(conc, k, dt, steps=steps, status=st, accepted=acc, rejected=rej, dt_carry=carry)
            out |= {f"{name}{steps}_{i}": x for i, x in enumerate((conc, st, acc, rej, carry))}
            # The workspace's second counter is the number of parked cells.
            out[f"{name}{steps}_parked"] = s.workspace(cells)[:8].clone().view(torch.int32)[1:]
    return out


if __name__ == "__main__":
    what, mech, cells, dt, path = sys.argv[1:]
    got = {"integrations": integrations, "sweeps": sweeps, "parking": parking}[what](mech, int(cells), float(dt))
    np.savez(path, **{name: x.cpu().numpy() for name, x in got.items() if x is not None})
