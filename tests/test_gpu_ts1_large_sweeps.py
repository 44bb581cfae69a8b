"""TS1's adjoint and tangent of large batches run on lanes, where the chip is
full and the warps' stores leave room for two or three of them per SM (GPU).

The route shows in the workspace: the lanes' tiles lie there, a call on warps
leaves all but the work counter alone.  Both give the same bits."""

import numpy as np
import pytest

from mkpp_gb300 import workloads

pytestmark = pytest.mark.gpu

SOME = 16          # cells with inputs of their own, repeated


@pytest.mark.parametrize("sweep, most", [("adjoint", 16384), ("tangent", 26000)])
def test_large_batches_run_on_lanes(sweep, most):
    import torch

    from mkpp_gb300 import build
    from mkpp_gb300.adjoint import Checkpoints
    from mkpp_gb300.api import DeviceSolver

    build.build(("ts1",))
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    w = workloads.make("ts1", SOME, seed=7)
    s = DeviceSolver("ts1")
    start = d(w.conc)
    k, _ = s.rate_constants(start, d(w.temp), d(w.rho), d(w.rh), None, d(w.param))
    rng = np.random.default_rng(3)
    ins = [start, k, d(rng.standard_normal(start.shape)), d(rng.standard_normal(k.shape)) * k]
    out = {}
    for n in (SOME, most, most + 1):
        conc, kn, vec, dk = (x.repeat(1, -(-n // SOME))[:, :n].contiguous() for x in ins)
        ck = Checkpoints("ts1", n, 2, "cuda")
        ck.forward(conc, kn, 1.0e-6, 1.0e-6)                   # (the cells stop when the checkpoint is full)
        ck.tws = torch.zeros(int(ck.lib.mkpp_gpu_tangent_workspace_bytes(n)) + 256, dtype=torch.uint8, device="cuda")
        ck.ws.zero_()
        got = ck.adjoint(kn, vec) if sweep == "adjoint" else (ck.tangent(kn, vec, dk),)
        lanes = bool((ck.ws if sweep == "adjoint" else ck.tws)[256:1 << 20].any())
        assert lanes == (n > most), n
        out[n] = [x[:, :SOME].clone() for x in got] + [x[:, n - 1].clone() for x in got]
        del ck
    last = [[x[:, (n - 1) % SOME] for x in out[SOME][:len(out[n]) // 2]] for n in (most, most + 1)]
    for n, want in zip((most, most + 1), last):
        half = len(out[n]) // 2
        for a, b in zip(out[n], out[SOME][:half] + want):
            assert torch.equal(a, b)
