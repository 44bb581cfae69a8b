"""Up to which number of cells a call runs on whole warps alone: 8000 of
saprc99_mini, where warps and lanes take the same time (GPU).

The route shows in the workspace: the lanes' tiles lie there, a call on warps
leaves all but the counters alone.  Both give the same bits."""

import numpy as np
import pytest

from mkpp_gb300 import workloads

pytestmark = pytest.mark.gpu

SOME = 64          # cells with inputs of their own, repeated


def test_line_between_warps_and_lanes():
    import torch

    from mkpp_gb300 import build
    from mkpp_gb300.api import DeviceSolver

    build.build(("saprc99_mini",))
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    w = workloads.make("saprc99_mini", SOME, seed=11)
    s = DeviceSolver("saprc99_mini")
    s.set_tuning(defer_after=3000)             # the defaults, whatever other tests left
    s.set_tail_parking(16)
    start = d(w.conc)
    k, _ = s.rate_constants(start, d(w.temp), d(w.rho), d(w.rh), None, d(w.param))
    out = {}
    for n in (SOME, 8000, 8001):
        conc, kn = (x.repeat(1, -(-n // SOME))[:, :n].contiguous() for x in (start, k))
        status = torch.zeros(n, dtype=torch.int32, device="cuda")
        ws = s.workspace(n)
        ws.zero_()
        s.integrate_k(conc, kn, 1.0, status=status)
        assert bool(ws[256:1 << 20].any()) == (n > 8000), n
        out[n] = torch.cat([conc, status[None].double()])
    for n in (8000, 8001):
        assert torch.equal(out[n][:, :SOME], out[SOME])
        assert torch.equal(out[n][:, n - 1], out[SOME][:, (n - 1) % SOME])
