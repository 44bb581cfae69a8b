"""Programs of 128-bit words on the GPU: shipped mechanisms emitted with them
(as a mechanism with slots beyond 14 bits is) end like the shipped libraries,
bit for bit, on warps and on lanes."""

import numpy as np
import pytest

import variant_library
from mkpp_gb300 import workloads

pytestmark = pytest.mark.gpu

# (mechanism, table-driven, dt)
FORMS = [("chapman", True, 600.0), ("saprc99_mini", None, 1.0e-2)]


@pytest.fixture(scope="module", params=FORMS, ids=[f[0] for f in FORMS])
def wide(request, tmp_path_factory):
    from mkpp_gb300 import api, build
    from mkpp_gb300.emitter import warp_schedule

    mech, table, dt = request.param
    build.build((mech,))
    name = f"{mech}_wide"
    with pytest.MonkeyPatch.context() as m:
        m.setattr(warp_schedule, "is_wide", lambda *programs: True)
        variant_library.make(tmp_path_factory.mktemp(name), m, name, mech, table)
    yield mech, name, dt
    api._LIBS.pop(name, None)


def _outputs(mech, name, dt):
    import torch

    from mkpp_gb300.adjoint import Checkpoints
    from mkpp_gb300.api import DeviceSolver

    n = 65
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    w = workloads.make(mech, n, seed=4)
    s = DeviceSolver(name)
    start = d(w.conc)
    k, _ = s.rate_constants(start, d(w.temp), d(w.rho), d(w.rh), None, d(w.param))
    out = []
    for mode in ("persistent", "plain"):
        conc = start.clone()
        st, acc, rej = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(3))
        s.integrate_k(conc, k, dt, seed=1e-6, mode=mode, status=st, accepted=acc, rejected=rej)
        out += [conc, st, acc, rej]
    ck = Checkpoints(name, n, 256, "cuda")
    rng = np.random.default_rng(2)
    lam, dk = d(rng.standard_normal(start.shape)), d(rng.standard_normal(k.shape)) * k
    ck.forward(start.clone(), k, dt, 1e-6)
    gc, gk = ck.adjoint(k, lam)
    out += [ck.status, ck.count, gc, gk, ck.tangent(k, start, dk)]
    return [x.cpu().numpy() for x in out]


def test_wide_programs_end_like_the_shipped_ones(wide):
    mech, name, dt = wide
    for a, b in zip(_outputs(mech, name, dt), _outputs(mech, mech, dt)):
        assert np.array_equal(a, b, equal_nan=True)
