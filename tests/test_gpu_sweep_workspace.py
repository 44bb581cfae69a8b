"""Differentiated calls of few cells and their workspace (GPU).

A call that runs on whole warps keeps its store in shared memory and has no
use for the workspace: it leaves it as it is, so that calls on two streams
may share one."""

import numpy as np
import pytest

from mkpp_gb300 import workloads

pytestmark = pytest.mark.gpu

CELLS = 72


@pytest.fixture(scope="module", autouse=True)
def libs(built_libs):
    return built_libs


def _inputs(mech, seed, cells=CELLS):
    import torch

    from mkpp_gb300.adjoint import Checkpoints
    from mkpp_gb300.api import DeviceSolver

    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    w = workloads.make(mech, cells, seed=seed)
    s = DeviceSolver(mech)
    conc = d(w.conc)
    k, _ = s.rate_constants(conc, d(w.temp), d(w.rho), d(w.rh), None, d(w.param))
    ck = Checkpoints(mech, cells, 64, "cuda")
    rng = np.random.default_rng(seed)
    return s, conc, k, ck, d(rng.standard_normal(conc.shape)), d(rng.standard_normal(k.shape)) * k


def _sweep(mech, dt, s, conc, k, ck, lam, dk):
    """Every output of the three sweeps (the cells that outgrow the
    checkpoint stop there, so a short interval is enough)."""
    ck.forward(conc, k, dt, s.default_seed, 20000)
    gc, gk = ck.adjoint(k, lam)
    return conc, ck.status, ck.acc, ck.count, gc, gk, ck.tangent(k, conc, dk)


@pytest.mark.parametrize("mech, dt", [("chapman", 1.0), ("small_strato", 1.0), ("saprc99", 1e-3)])
def test_warp_sweeps_leave_the_workspace_as_it_is(mech, dt):
    import torch

    s, conc, k, ck, lam, dk = _inputs(mech, 3)
    need = int(ck.lib.mkpp_gpu_tangent_workspace_bytes(CELLS))
    ck.ws.fill_(0xA5)
    ck.tws = torch.full((need + 256,), 0xA5, dtype=torch.uint8, device="cuda")
    _sweep(mech, dt, s, conc, k, ck, lam, dk)
    torch.cuda.synchronize()
    assert bool((ck.ws == 0xA5).all()) and bool((ck.tws == 0xA5).all())


@pytest.mark.parametrize("mech, dt", [("chapman", 1.0), ("small_strato", 1.0)])
def test_two_streams_on_one_workspace(mech, dt):
    import torch

    want = [[x.clone() for x in _sweep(mech, dt, *_inputs(mech, seed, 300))] for seed in (3, 4)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(4):
        sides = [_inputs(mech, seed, 300) for seed in (3, 4)]
        ws = sides[0][3].ws
        need = int(sides[0][3].lib.mkpp_gpu_tangent_workspace_bytes(300))
        tws = torch.zeros(need + 256, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        got = []
        for stream, side in zip(streams, sides):
            side[3].ws, side[3].tws = ws, tws
            with torch.cuda.stream(stream):
                got.append(_sweep(mech, dt, *side))
        torch.cuda.synchronize()
        for a, b in zip(want, got):
            assert all(torch.equal(x, y) for x, y in zip(a, b))
