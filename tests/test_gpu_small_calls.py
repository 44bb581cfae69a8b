"""Calls that the cooperative kernel takes as a whole, and the evaluation
kernels, at the sizes where their splits end (GPU).

A persistent call of few cells runs every cell on a whole warp; the plain form
runs a thread per cell.  Both have to end bit-identical, with cells in a given
order, cells flagged as not finite and the attempt cap reached included.  The
evaluation kernels take 32 cells per block: their outputs of a cell do not
depend on the number of cells around it.
"""

import numpy as np
import pytest

from mkpp_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def libs():
    from mkpp_gb300 import build

    return build.build(("saprc99", "ts1"))


def _run(mech, w, mode, dt, order=None, cap=20000, steps=1):
    import torch

    from mkpp_gb300.api import DeviceSolver

    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    s = DeviceSolver(mech)
    conc = d(w.conc)
    k, status = s.rate_constants(conc, d(w.temp), d(w.rho), d(w.rh), None, d(w.param))
    acc, rej = (torch.full((w.ncells,), 77, dtype=torch.int32, device="cuda") for _ in range(2))
    s.integrate_k(conc, k, dt, steps=steps, mode=mode, max_attempts=cap, status=status, accepted=acc, rejected=rej,
                  order=None if order is None else d(order))
    return [x.cpu().numpy() for x in (conc, status, acc, rej)]


@pytest.mark.parametrize("mech, cells, dt, steps", [("saprc99", 1, 1e-3, 1), ("saprc99", 33, 1e-2, 2),
                                                    ("saprc99", 1300, 1e-4, 1), ("ts1", 5, 1e-4, 1)])
def test_cooperative_call_equals_plain(libs, mech, cells, dt, steps):
    w = workloads.make(mech, cells, seed=5)
    if cells > 2:
        w.conc[3, 1] = np.nan
    order = np.random.default_rng(2).permutation(cells).astype(np.int32)
    plain = _run(mech, w, "plain", dt, steps=steps)
    for kw in ({}, {"order": order}):
        got = _run(mech, w, "persistent", dt, steps=steps, **kw)
        for a, b in zip(got, plain):
            assert np.array_equal(a, b, equal_nan=True)
    capped = [_run(mech, w, m, dt, cap=4) for m in ("plain", "persistent")]
    assert (capped[0][1] != 0).any()
    for a, b in zip(*capped):
        assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("mech", ["saprc99", "ts1"])
def test_evaluation_does_not_depend_on_the_batch(libs, mech):
    import torch

    from mkpp_gb300.api import DeviceSolver

    s = DeviceSolver(mech)
    total = 2081                    # two cells per lane of the Jacobian's blocks, the last ones alone
    w = workloads.make(mech, total, seed=6)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    conc = d(w.conc)
    k, _ = s.rate_constants(conc, d(w.temp), d(w.rho), d(w.rh), None, d(w.param))
    f, j = s.evaluate_rates(conc, k), s.evaluate_jacobian(conc, k)
    for n in (1, 31, 32, 33, 64, 65):
        at = total - n
        sub, ks = conc[:, at:].contiguous(), k[:, at:].contiguous()
        cut = lambda a: d(a[..., at:])  # noqa: E731
        again, flagged = s.rate_constants(sub, cut(w.temp), cut(w.rho), cut(w.rh), None, cut(w.param))
        assert torch.equal(again, ks) and not flagged.any()
        assert torch.equal(s.evaluate_rates(sub, ks), f[:, at:])
        assert torch.equal(s.evaluate_jacobian(sub, ks), j[:, :, at:])
