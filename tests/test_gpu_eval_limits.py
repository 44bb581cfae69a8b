"""Tendencies and Jacobians of a mechanism whose rates, or whose column's
partial derivatives, do not fit in a block's shared memory (GPU): the shipped
mechanism with these numbers declared larger ends like the shipped library,
bit for bit."""

import re

import numpy as np
import pytest

import variant_library
from mkpp_gb300 import workloads

pytestmark = pytest.mark.gpu

MECH = "saprc99_mini"


@pytest.fixture(scope="module")
def unstaged(tmp_path_factory):
    from mkpp_gb300 import api, build

    build.build((MECH,))
    with pytest.MonkeyPatch.context() as m:
        variant_library.make(tmp_path_factory.mktemp("unstaged"), m, "unstaged", MECH, change=lambda text: re.sub(
            r"constexpr int (RATES|MAX_PARTIALS) = \d+;", r"constexpr int \1 = 2000;", text))
    yield "unstaged"
    api._LIBS.pop("unstaged", None)


@pytest.mark.parametrize("cells", [1, 65, 2100])
def test_unstaged_evaluation_equals_the_staged(unstaged, cells):
    import torch

    from mkpp_gb300.api import DeviceSolver

    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    w = workloads.make(MECH, cells, seed=6)
    conc = d(w.conc)
    shipped, other = DeviceSolver(MECH), DeviceSolver(unstaged)
    k, _ = shipped.rate_constants(conc, d(w.temp), d(w.rho), d(w.rh), None, d(w.param))
    assert torch.equal(shipped.evaluate_rates(conc, k), other.evaluate_rates(conc, k))
    assert torch.equal(shipped.evaluate_jacobian(conc, k), other.evaluate_jacobian(conc, k))
