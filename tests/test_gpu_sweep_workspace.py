"""Differentiated calls of few cells and their workspace (GPU).

Where a mechanism's lanes keep their store in registers they have no use for
the workspace of the checkpointed forward and of the adjoint.  Such a call on
whole warps leaves it as it is too, so that calls on two streams may share
one."""

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
    """Every output of the sweeps that leave the workspace alone (the cells that
    outgrow the checkpoint stop there, so a short interval is enough)."""
    ck.forward(conc, k, dt, s.default_seed, 20000)
    out = [conc, ck.status, ck.acc, ck.count]
    if mech == "chapman":                    # small_strato's adjoint store is a tile
        out += ck.adjoint(k, lam)
    return out


@pytest.mark.parametrize("mech", ["chapman", "small_strato"])
def test_warp_sweeps_leave_the_workspace_as_it_is(mech):
    import torch

    s, conc, k, ck, lam, dk = _inputs(mech, 3)
    ck.ws.fill_(0xA5)
    _sweep(mech, 1.0, s, conc, k, ck, lam, dk)
    torch.cuda.synchronize()
    assert bool((ck.ws == 0xA5).all())


@pytest.mark.parametrize("mech", ["chapman", "small_strato"])
def test_two_streams_on_one_workspace(mech):
    import torch

    want = [[x.clone() for x in _sweep(mech, 1.0, *_inputs(mech, seed, 300))] for seed in (3, 4)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(4):
        sides = [_inputs(mech, seed, 300) for seed in (3, 4)]
        ws = sides[0][3].ws
        torch.cuda.synchronize()
        got = []
        for stream, side in zip(streams, sides):
            side[3].ws = ws
            with torch.cuda.stream(stream):
                got.append(_sweep(mech, 1.0, *side))
        torch.cuda.synchronize()
        for a, b in zip(want, got):
            assert all(torch.equal(x, y) for x, y in zip(a, b))
