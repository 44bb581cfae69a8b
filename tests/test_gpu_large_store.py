"""A mechanism whose store does not fit in a block's shared memory (GPU).

The cooperative kernels keep a cell's store there; without them a call runs
on lanes, in every entry.  The mechanism is Chapman with its warp stores
declared larger than they are, so that the same cells have known results."""

import re

import numpy as np
import pytest

from mkpp_gb300 import workloads

pytestmark = pytest.mark.gpu

CELLS = 72


@pytest.fixture(scope="module")
def large(built_libs, tmp_path_factory):
    from mkpp_gb300 import api, build

    tmp = tmp_path_factory.mktemp("large")
    text = (build.GEN / "chapman.cuh").read_text().replace("mkpp_chapman", "mkpp_chapman_large")
    for name in ("WARP_SLOTS", "ADJ_COOP_SLOTS", "TLM_COOP_SLOTS"):
        text, n = re.subn(rf"constexpr int {name} = [^;]+;", f"constexpr int {name} = 30000;", text)
        assert n == 1
    (tmp / "chapman_large.cuh").write_text(text)
    with pytest.MonkeyPatch.context() as m:
        m.setattr(build, "GEN", tmp)
        m.setattr(build, "LIB", tmp)
        m.setattr(api, "LIB_DIR", tmp)
        build.compile_mechanism("chapman_large")
        api.load_library("chapman_large")
    yield "chapman_large"
    api._LIBS.pop("chapman_large", None)


def _all(mech, dt):
    """Outputs of every entry that a warp may take, on the same cells."""
    import torch

    from mkpp_gb300.adjoint import Checkpoints
    from mkpp_gb300.api import DeviceSolver

    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    w = workloads.make("chapman", CELLS, seed=9)
    s = DeviceSolver(mech)
    conc = d(w.conc)
    k, status = s.rate_constants(conc, d(w.temp), d(w.rho), d(w.rh), None, d(w.param))
    acc, rej = (torch.zeros(CELLS, dtype=torch.int32, device="cuda") for _ in range(2))
    end = conc.clone()
    s.integrate_k(end, k, dt, seed=1e-6, status=status, accepted=acc, rejected=rej)
    ck = Checkpoints(mech, CELLS, 256, "cuda")
    rng = np.random.default_rng(2)
    lam, dk = d(rng.standard_normal(conc.shape)), d(rng.standard_normal(k.shape)) * k
    ck.forward(conc.clone(), k, dt, 1e-6)
    gc, gk = ck.adjoint(k, lam)
    return [end, status, acc, rej, ck.status, ck.count, gc, gk, ck.tangent(k, conc, dk)]


def test_every_entry_runs_on_lanes_with_the_same_results(large):
    import torch

    for a, b in zip(_all(large, 600.0), _all("chapman", 600.0)):
        assert torch.equal(a, b)
