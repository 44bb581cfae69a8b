"""Calls of few cells on whole warps and on lanes end bit-identical, and so do
cells that move from lanes to warps (GPU).

Which form takes a call depends on the number of cells and on launch settings
of the process, so the calls run in processes of their own
(route_outputs.py), on lanes with MKPP_COOP_CELLS=0."""

import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from mkpp_gb300 import workloads

pytestmark = pytest.mark.gpu

SCRIPT = Path(__file__).resolve().parent / "route_outputs.py"
# The most cells whose sweeps run on warps for register stores, else a few.
CASES = [("chapman", 300, 600.0), ("small_strato", 2000, 1.0), ("saprc99_mini", 65, 1.0), ("saprc99", 33, 1.0e-3),
         ("ts1", 5, 1.0e-4)]


@pytest.fixture(scope="module", autouse=True)
def libs():
    from mkpp_gb300 import build

    return build.build(tuple(c[0] for c in CASES))


def _run(tmp, what, mech, cells, dt, lanes):
    path = tmp / f"{what}_{mech}_{lanes}.npz"
    env = {k: v for k, v in os.environ.items() if not k.startswith("MKPP_")}
    if lanes:
        env["MKPP_COOP_CELLS"] = "0"
    subprocess.run([sys.executable, str(SCRIPT), what, mech, str(cells), str(dt), str(path)], check=True, env=env,
                   timeout=600)
    return np.load(path)


def _equal(a, b):
    assert sorted(a.files) == sorted(b.files)
    for name in a.files:
        assert np.array_equal(a[name], b[name], equal_nan=True), name


@pytest.mark.parametrize("mech, cells, dt", CASES)
def test_warps_and_lanes_integrate_alike(tmp_path, mech, cells, dt):
    warps, lanes = (_run(tmp_path, "integrations", mech, cells, dt, x) for x in (False, True))
    _equal(warps, lanes)
    for i in range(4):
        assert np.array_equal(warps[f"cells_{i}"], warps[f"plain_{i}"], equal_nan=True)
        assert np.array_equal(warps[f"cells_{i}"], warps[f"order_{i}"], equal_nan=True)
    assert (warps["capped_1"] == 3).any() and warps["cells_1"][cells // 2] == 2


@pytest.mark.parametrize("mech, cells, dt", CASES)
def test_warps_and_lanes_differentiate_alike(tmp_path, mech, cells, dt):
    warps, lanes = (_run(tmp_path, "sweeps", mech, cells, dt, x) for x in (False, True))
    _equal(warps, lanes)
    assert (warps["cap8_1"] == 5).any() and (warps["cap64_4"] > 8).any() and warps["cap64_4"][cells // 2] == 0


@pytest.mark.parametrize("mech, cells, dt", [("small_strato", 512, 600.0), ("saprc99_mini", 200, 600.0),
                                             ("saprc99", 96, 600.0)])
def test_parked_cells_end_alike(tmp_path, mech, cells, dt):
    got = _run(tmp_path, "parking", mech, cells, dt, True)
    for steps in (1, 2):
        assert got[f"none{steps}_parked"] == 0
        assert got[f"first{steps}_parked"] > cells // 2 and got[f"tail{steps}_parked"] > 0
        for form in ("first", "tail"):
            for i in range(5):
                assert np.array_equal(got[f"{form}{steps}_{i}"], got[f"none{steps}_{i}"], equal_nan=True), (form, i)


@pytest.mark.parametrize("mech, cells", [("saprc99_mini", 6000), ("chapman", 170000)])
def test_cost_order_of_calls_that_do_not_start_at_once(mech, cells):
    """More cells than start at once, on warps and on lanes: each call hands
    out the cells by the attempts of the one before, with the same results
    as in cell order."""
    from mkpp_gb300.api import MechanismContext

    w = workloads.make(mech, cells, seed=1)
    runs = []
    for enable in (False, True):
        ctx = MechanismContext(mech, cells)
        try:
            ctx.set_cost_order(enable)
            host = np.ascontiguousarray(w.conc.copy())
            ctx.set_state(host, w.temp.copy(), w.pressure.copy(), w.rho.copy())
            ctx.set_aerosol(relative_humidity=w.rh.copy())
            for step in range(3):
                ctx.set_rate_parameters(np.ascontiguousarray(w.param_at(step)))
                ctx.integrate(w.dt)
            runs.append((host, *ctx.cell_stats()))
        finally:
            ctx.close()
    for a, b in zip(*runs):
        assert np.array_equal(a, b, equal_nan=True)
