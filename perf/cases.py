"""The calls whose time counts: what programs that use the solver have it do.

Five kinds of call, each through a public entry point:

* ``host``      a host model's chemistry step: ``MechanismContext`` on numpy
                arrays that the model owns, one ``integrate(dt)`` and the
                cells' statuses.  From one column to a regional domain.
* ``window``    device-resident chemistry: ``DeviceSolver``, the rate constants
                of every host step and one integrate over all of them.
* ``gradient``  ``rosenbrock_solve`` and its backward: dL/dC0 and dL/dk of an
                inversion or a training step.
* ``tangent``   forward mode of ``rosenbrock_solve``: a directional derivative.
* ``evaluate``  rate constants, tendencies and the dense Jacobian of given
                states, as diagnostics and implicit couplings ask for them.

Cells come from the repository's seeded workloads (species log-uniform,
meteorology and photolysis as there).  Chapman and small_strato start from
those draws as they are.  The tropospheric mechanisms start as a model's cold
start does: the emitted and background species as drawn, their products and
radicals at zero; TS1's are remote cells on the night side.
"""

import json
import math
from pathlib import Path

import numpy as np
import torch

from mkpp_gb300 import workloads
from mkpp_gb300.adjoint import rosenbrock_solve
from mkpp_gb300.api import DeviceSolver, MechanismContext

MECHANISMS = Path(__file__).resolve().parent.parent / "mkpp_gb300" / "mechanisms"

_BACKGROUND = ("AIR", "M", "O2", "N2", "H2O", "CH4", "H2", "CO2", "CO", "NO", "NO2", "O3", "SO2")
# Species that a cold start gives a value: background and emitted ones.
COLD_START = {
    "saprc99": _BACKGROUND + ("HCHO", "CCHO", "RCHO", "ACET", "MEK", "ETHENE", "ISOPRENE", "ALK1", "ALK2", "ALK3",
                              "ALK4", "ALK5", "ARO1", "ARO2", "OLE1", "OLE2", "TERP", "MEOH"),
    "saprc99_mini": _BACKGROUND,
    # Remote air: no nitrogen oxides and no alkenes.
    "ts1": tuple(x for x in _BACKGROUND if x not in ("NO", "NO2")) + (
        "N2O", "HCL", "CH2O", "C2H6", "C3H8", "CH3OH", "DMS", "OCS", "NH3", "CH3CL", "CFC11", "CFC12"),
}

# Rate constants of 1e33-1e37 1/s in the mechanisms as shipped (the Troe k0 of
# thermal decompositions), which make derivatives meaningless: differentiated
# calls get them at 1e3, as the repository's gradient tests do.
MODERATED = {"saprc99": (11, 32, 69), "saprc99_mini": (7,)}

# Attempted steps per cell: of the first host step and of each later one
# (means of the CPU oracle over seeded cells), and the FP64 operations of one
# attempt and of one tendency and Jacobian evaluation (Jacobian, LU, tendency,
# solves, stages and error norm, a multiply-add counted as two).
ATTEMPTS = {"chapman": (49, 12), "chapman_rodas3": (40, 12), "small_strato": (94, 11), "small_strato_rodas3": (60, 9),
            "saprc99_mini": (15, 11), "saprc99": (35, 14), "ts1": (9, 9)}
FLOPS = {"chapman": 239, "chapman_rodas3": 300, "small_strato": 649, "small_strato_rodas3": 850, "saprc99_mini": 1084,
         "saprc99": 40215, "ts1": 153901}
EVAL_FLOPS = {"chapman": 97, "chapman_rodas3": 97, "small_strato": 260, "small_strato_rodas3": 260,
              "saprc99_mini": 338, "saprc99": 9072, "ts1": 19648}

# Largest cells per call and host steps per window of each kind and mechanism.
RANGES = {
    ("host", "chapman"): (65536, 1), ("host", "chapman_rodas3"): (65536, 1),
    ("host", "small_strato"): (65536, 1), ("host", "small_strato_rodas3"): (65536, 1),
    ("host", "saprc99_mini"): (32768, 1), ("host", "saprc99"): (16384, 1),
    ("window", "chapman"): (262144, 1), ("window", "chapman_rodas3"): (262144, 1),
    ("window", "small_strato"): (65536, 12), ("window", "small_strato_rodas3"): (65536, 12),
    ("window", "saprc99_mini"): (65536, 6), ("window", "saprc99"): (65536, 4), ("window", "ts1"): (4096, 2),
    ("gradient", "chapman"): (16384, 1), ("gradient", "small_strato"): (16384, 1),
    ("gradient", "saprc99_mini"): (8192, 1), ("gradient", "saprc99"): (2048, 1),
    ("tangent", "small_strato"): (16384, 1), ("tangent", "saprc99"): (2048, 1),
    ("evaluate", "small_strato"): (262144, 1), ("evaluate", "saprc99_mini"): (131072, 1),
    ("evaluate", "saprc99"): (20480, 1), ("evaluate", "ts1"): (3072, 1),
}


def listed():
    def case(name, kind, mech, cells, steps=1):
        return {"name": name, "kind": kind, "mechanism": mech, "cells": cells, "steps": steps}

    return [
        # One column of a stratospheric model per call: latency.
        case("host_chapman_column", "host", "chapman", 72),
        # A regional domain of a host model that calls the C ABI each step.
        case("host_small_strato_rodas3", "host", "small_strato_rodas3", 40000),
        # One MPI rank's share of an air-quality model's domain.
        case("host_saprc99_rank", "host", "saprc99", 2500),
        # The repository's Chapman configuration.
        case("window_chapman", "window", "chapman", 4096),
        # The repository's small_strato configuration.
        case("window_small_strato", "window", "small_strato", 65536, 12),
        # A box-model ensemble over four host steps.
        case("window_saprc99_ensemble", "window", "saprc99", 333, 4),
        # A quarter of the repository's SAPRC99 domain over four host steps.
        case("window_saprc99_domain", "window", "saprc99", 65536, 4),
        # A night-side tile of the large global mechanism, 210 species.
        case("window_ts1_tile", "window", "ts1", 4096),
        # Inversion: gradients for a batch of cells.
        case("gradient_saprc99", "gradient", "saprc99", 1500),
        # Sensitivity of a batch of cells along one direction.
        case("tangent_saprc99", "tangent", "saprc99", 600),
        # Diagnostics of a domain: rates, tendencies, Jacobians.
        case("evaluate_saprc99", "evaluate", "saprc99", 20000),
        case("evaluate_ts1", "evaluate", "ts1", 1001),
    ]


def draw(rng):
    kind, mech = rng.choice(sorted(RANGES))
    cells, steps = RANGES[(kind, mech)]
    # Cells over the logarithm of the range, from one warp's worth (a single
    # column) up, odd sizes among them.
    n = int(round(math.exp(rng.uniform(math.log(16), math.log(cells)))))
    return {"kind": kind, "mechanism": mech, "cells": n, "steps": rng.randint(1, steps)}


# ---------------------------------------------------------------------------
# Inputs.
# ---------------------------------------------------------------------------
def _cells(case, seed):
    mech, n = case["mechanism"], case["cells"]
    w = workloads.make(mech, n, seed=seed)
    keep = COLD_START.get(mech)
    if keep is not None:
        raw = _plan(mech)
        for s, name in enumerate(raw["species"]):
            if name not in keep and not raw["fixed"][s]:
                w.conc[s] = 0.0
    if mech == "ts1":
        w.phase[:] = np.pi                      # the sun stays below the horizon
        w.param = w.param_at(0)
    return w


_PLANS = {}
_SOLVERS = {}


def _plan(mech):
    if mech not in _PLANS:
        _PLANS[mech] = json.loads((MECHANISMS / f"{mech}.plan.json").read_text())
    return _PLANS[mech]


def _solver(mech):
    # A program keeps one solver (and its workspace) per mechanism.
    if mech not in _SOLVERS:
        _SOLVERS[mech] = DeviceSolver(mech)
    return _SOLVERS[mech]


def _device(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# Species that an inversion has observations of.
OBSERVED = ("O", "O3", "NO", "NO2", "CO", "HCHO")


def _directions(case, seed, w):
    """Weights of a loss on the observed species' end state, and relative
    perturbations of the start and of the rate constants."""
    rng = np.random.default_rng([seed, 1])
    ns, n = w.conc.shape
    scale = np.maximum(np.abs(w.conc), 1.0).max(axis=1, keepdims=True)
    lam = rng.standard_normal((ns, n)) / scale
    lam[[s not in OBSERVED for s in _plan(case["mechanism"])["species"]]] = 0.0
    dconc = rng.standard_normal((ns, n)) * w.conc
    dk = rng.standard_normal((len(_plan(case["mechanism"])["reactions"]), n))
    return lam, dconc, dk


def prepare(case, seed):
    kind, mech, n, steps = case["kind"], case["mechanism"], case["cells"], case["steps"]
    w = _cells(case, seed)
    st = {"kind": kind, "mechanism": mech, "dt": w.dt, "steps": steps}
    if kind == "host":
        st["start"] = w.conc.copy()
        st["conc"] = w.conc
        st["ctx"] = MechanismContext(mech, n)
        st["ctx"].set_state(st["conc"], w.temp, w.pressure, w.rho)
        st["ctx"].set_rate_parameters(np.ascontiguousarray(w.param))
        st["ctx"].set_aerosol(relative_humidity=w.rh)
        return st
    st["solver"] = _solver(mech)
    st["conc"] = _device(w.conc)
    st["met"] = {"temp": _device(w.temp), "rho": _device(w.rho), "rh": _device(w.rh)}
    st["param"] = [_device(w.param_at(s)) for s in range(steps)]
    if kind == "window":
        nr = len(_plan(mech)["reactions"])
        st["ktab"] = torch.empty((steps, nr, n), dtype=torch.float64, device="cuda")
        st["work"] = torch.empty_like(st["conc"])
        for key in ("status", "accepted", "rejected"):
            st[key] = torch.zeros(n, dtype=torch.int32, device="cuda")
    elif kind in ("gradient", "tangent"):
        k, _ = st["solver"].rate_constants(st["conc"], param=st["param"][0], **st["met"])
        for r in MODERATED.get(mech, ()):
            k[r].clamp_(max=1e3)
        lam, dconc, dk = _directions(case, seed, w)
        st["k"] = k
        st["lam"], st["dconc"], st["dk"] = _device(lam), _device(dconc), _device(dk) * k
    return st


# ---------------------------------------------------------------------------
# One pass.
# ---------------------------------------------------------------------------
# Accepted steps a differentiated call may record.
CAP = 256


def run(st):
    return {"host": _host, "window": _window, "gradient": _gradient, "tangent": _tangent,
            "evaluate": _evaluate}[st["kind"]](st)


def _host(st):
    # The rest of the host model gave the cells their values.
    np.copyto(st["conc"], st["start"])
    st["ctx"].integrate(st["dt"])
    status, accepted, rejected = st["ctx"].cell_stats()
    return {"conc": st["conc"], "status": status, "accepted": accepted, "rejected": rejected}


def _window(st):
    s, conc = st["solver"], st["work"]
    conc.copy_(st["conc"])
    for i in range(st["steps"]):
        s.rate_constants(conc, param=st["param"][i], ktab=st["ktab"][i], status=st["status"], **st["met"])
    s.integrate_k(conc, st["ktab"], st["dt"], steps=st["steps"], status=st["status"], accepted=st["accepted"],
                  rejected=st["rejected"], k_step_stride=st["ktab"].stride(0))
    return {"conc": conc, "status": st["status"], "accepted": st["accepted"], "rejected": st["rejected"]}


def _gradient(st):
    conc = st["conc"].detach().requires_grad_(True)
    k = st["k"].detach().requires_grad_(True)
    end = rosenbrock_solve(conc, k, st["mechanism"], st["dt"], cap=CAP)
    (end * st["lam"]).sum().backward()
    return {"conc": end.detach(), "grad_conc": conc.grad, "grad_k": k.grad}


def _tangent(st):
    import torch.autograd.forward_ad as fwd

    with fwd.dual_level():
        end = rosenbrock_solve(fwd.make_dual(st["conc"], st["dconc"]), fwd.make_dual(st["k"], st["dk"]),
                               st["mechanism"], st["dt"], cap=CAP)
        value, slope = fwd.unpack_dual(end)
    return {"conc": value, "dconc": slope}


def _evaluate(st):
    s = st["solver"]
    k, status = s.rate_constants(st["conc"], param=st["param"][0], **st["met"])
    return {"k": k, "status": status, "f": s.evaluate_rates(st["conc"], k), "jac": s.evaluate_jacobian(st["conc"], k)}


# ---------------------------------------------------------------------------
# What a pass cannot do without.
# ---------------------------------------------------------------------------
def work(case):
    kind, mech, n, steps = case["kind"], case["mechanism"], case["cells"], case["steps"]
    raw = _plan(mech)
    ns, nr, npar = len(raw["species"]), len(raw["reactions"]), raw["num_rate_parameters"]
    first, later = ATTEMPTS[mech]
    attempts = first + later * (steps - 1)
    state, forcing = 8 * ns, 8 * (npar * steps + 3)
    if kind in ("host", "window"):
        return {"bytes": n * (2 * state + forcing + 12), "flops": n * attempts * FLOPS[mech]}
    if kind == "gradient":
        # Forward, then per accepted step its stages again and the transposed
        # solves with the Hessian-vector and dk terms (about one more attempt).
        return {"bytes": n * (4 * state + 16 * nr), "flops": 3 * n * attempts * FLOPS[mech]}
    if kind == "tangent":
        return {"bytes": n * (4 * state + 16 * nr), "flops": 3 * n * attempts * FLOPS[mech]}
    return {"bytes": n * (2 * state + forcing + 8 * nr + 8 * ns * ns), "flops": n * EVAL_FLOPS[mech]}


# ---------------------------------------------------------------------------
# The same results from dense linear algebra, in 64 bits.
# ---------------------------------------------------------------------------
class _Dense:
    """Mass-action kinetics of one mechanism on (species, cells) tensors."""

    def __init__(self, mech):
        self.raw = raw = _plan(mech)
        self.ns = len(raw["species"])
        self.var = [i for i, f in enumerate(raw["fixed"]) if not f]
        col = {s: i for i, s in enumerate(self.var)}
        self.nv = len(self.var)
        self.rx = []
        for r in raw["reactions"]:
            expo = {}
            for s, p in r["reactants"]:
                expo[col[s]] = expo.get(col[s], 0) + p
            self.rx.append((r["k"], expo))
        self.net = torch.zeros((self.nv, len(self.rx)), dtype=torch.float64, device="cuda")
        for r, rr in enumerate(raw["reactions"]):
            for s, c in rr["net"]:
                self.net[col[s], r] += c
        # (reaction, species, coefficient, remaining exponents) of each dm_r/dy_j
        self.partials = []
        for r, (_, expo) in enumerate(self.rx):
            for j in sorted(expo):
                rest = dict(expo)
                rest[j] -= 1
                self.partials.append((r, j, float(expo[j]), rest))
        self.pr = torch.tensor([p[0] for p in self.partials], device="cuda")
        self.pj = torch.tensor([p[1] for p in self.partials], device="cuda")
        tab = raw["tableau"]
        self.stages, self.gamma, self.elo = int(tab["stages"]), tab["Gamma"][0], tab["ELO"]
        self.a, self.c, self.m, self.e, self.newf = tab["A"], tab["C"], tab["M"], tab["E"], tab["NewF"]
        at = torch.tensor(raw["atol"], dtype=torch.float64, device="cuda")
        rt = torch.tensor(raw["rtol"], dtype=torch.float64, device="cuda")
        self.atol, self.rtol = at[self.var][:, None], rt[self.var][:, None]

    def rate_constants(self, w, step):
        raw = self.raw
        t = (lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda())
        run_env = raw["runtime_environment"]
        n = w.ncells
        env = {"pow": torch.pow, "exp": torch.exp, "log": torch.log, "sqrt": torch.sqrt, "fabs": torch.abs,
               "M_LN10": math.log(10.0), "P": t(w.param_at(step)), "FIX": t(w.conc), "RH": t(w.rh),
               "T": t(w.temp) if run_env else torch.full((n,), raw["environment_temperature"],
                                                         dtype=torch.float64, device="cuda"),
               "RHO": t(w.rho) if run_env else torch.full((n,), raw["environment_air_density"],
                                                          dtype=torch.float64, device="cuda"),
               "CLW": torch.zeros(n, dtype=torch.float64, device="cuda")}

        def either(f):
            wrap = (lambda x: x if isinstance(x, torch.Tensor) else torch.tensor(float(x), dtype=torch.float64,
                                                                                  device="cuda"))
            return lambda *xs: f(*(wrap(x) for x in xs))

        for f in ("pow", "exp", "log", "sqrt", "fabs"):
            env[f] = either(env[f])
        rows = []
        for text, _ in self.rx:
            v = eval(text, dict(env))  # noqa: S307  (the mechanism's own expressions)
            rows.append(v.expand(n) if isinstance(v, torch.Tensor) else torch.full((n,), float(v),
                                                                                   dtype=torch.float64, device="cuda"))
        return torch.stack(rows)

    @staticmethod
    def _mono(y, expo):
        out = None
        for j in sorted(expo):
            for _ in range(expo[j]):
                out = y[j] if out is None else out * y[j]
        return out

    def f(self, y, k):
        rows = []
        for r, (_, expo) in enumerate(self.rx):
            m = self._mono(y, expo)
            rows.append(k[r] if m is None else k[r] * m)
        return self.net @ torch.stack(rows)

    def jac(self, y, k):
        """(cells, nv, nv): dF_i/dy_j."""
        rows = []
        for r, _, coef, rest in self.partials:
            m = self._mono(y, rest)
            rows.append(coef * k[r] if m is None else coef * k[r] * m)
        d = torch.stack(rows)                                    # (partials, cells)
        out = torch.zeros((self.nv, self.nv, y.shape[1]), dtype=torch.float64, device=y.device)
        src = self.net[:, self.pr][:, :, None] * d[None]         # (nv, partials, cells)
        out = out.index_add(1, self.pj, src)
        return out.permute(2, 0, 1)

    def attempt(self, y, k, h):
        """(stage sum, error sum) of one step of size h per cell."""
        eye = torch.eye(self.nv, dtype=torch.float64, device=y.device)
        w = eye[None] / (self.gamma * h)[:, None, None] - self.jac(y, k)
        lu, piv = torch.linalg.lu_factor(w)
        ks, fv = [], None
        for i in range(self.stages):
            off = i * (i - 1) // 2
            if self.newf[i]:
                yi = y
                for j in range(i):
                    if self.a[off + j] != 0.0:
                        yi = yi + self.a[off + j] * ks[j]
                fv = self.f(yi, k)
            rhs = fv
            for j in range(i):
                if self.c[off + j] != 0.0:
                    rhs = rhs + (self.c[off + j] / h) * ks[j]
            ks.append(torch.linalg.lu_solve(lu, piv, rhs.t()[:, :, None])[:, :, 0].t())
        dy = sum(m * x for m, x in zip(self.m, ks) if m != 0.0)
        er = sum(e * x for e, x in zip(self.e, ks) if e != 0.0)
        return dy, er

    def integrate(self, y, k, dt, record=None):
        """One chemistry interval of every cell, with the embedded error
        estimate's step control; `record` collects (cells, y, h) per sweep."""
        n = y.shape[1]
        y = y.clone()
        z = torch.zeros(n, dtype=torch.float64, device=y.device)
        t, h = z.clone(), z + dt * self.raw["initial_step_seed"]
        last = torch.zeros(n, dtype=torch.bool, device=y.device)
        more = last.clone()
        for _ in range(20000):
            idx = torch.nonzero(t < dt)[:, 0]
            if idx.numel() == 0:
                break
            yi, ki = y[:, idx], k[:, idx]
            hi = torch.minimum(h[idx], dt - t[idx])
            dy, er = self.attempt(yi, ki, hi)
            sc = self.atol + self.rtol * torch.maximum(yi.abs(), (yi + dy).abs())
            err = torch.sqrt(((er / sc) ** 2).sum(0) / float(self.ns)).clamp_min(1e-10)
            fac = torch.clamp(0.9 * err ** (-1.0 / self.elo), 0.2, 6.0)
            ok = err <= 1.0
            if record is not None:
                record.append((idx[ok], yi[:, ok], hi[ok]))
            grown = torch.clamp(hi * fac, max=dt).clamp_min(dt * 1e-15)
            grown = torch.where(last[idx], torch.minimum(grown, hi), grown)
            shrunk = hi * torch.where(more[idx], torch.full_like(fac, 0.1), fac)
            y[:, idx] = torch.where(ok, yi + dy, yi)
            t[idx] = torch.where(ok, t[idx] + hi, t[idx])
            h[idx] = torch.where(ok, grown, shrunk)
            more[idx] = torch.where(ok, torch.zeros_like(ok), last[idx])
            last[idx] = ~ok
        return y


def exact(case, seed):
    kind, mech, n, steps = case["kind"], case["mechanism"], case["cells"], case["steps"]
    first, later = ATTEMPTS[mech]
    big = {"saprc99": 400_000, "ts1": 20_000}.get(mech, 1 << 40)
    if kind != "evaluate" and n * (first + later * (steps - 1)) * (4 if kind == "gradient" else 1) > big:
        return None  # over 20 seconds of dense factorizations
    d = _Dense(mech)
    w = _cells(case, seed)
    conc = _device(w.conc)
    y0 = conc[d.var]
    k = d.rate_constants(w, 0)
    if kind == "evaluate":
        f, jac = torch.zeros_like(conc), torch.zeros((d.ns, d.ns, n), dtype=torch.float64, device="cuda")
        f[d.var] = d.f(y0, k)
        at = torch.tensor(d.var, device="cuda")
        for c0 in range(0, n, 1024):
            j = d.jac(y0[:, c0:c0 + 1024], k[:, c0:c0 + 1024]).permute(2, 1, 0)
            jac[at[:, None], at[None, :], c0:c0 + 1024] = j
        return {"k": k, "status": None, "f": f, "jac": jac}
    if kind in ("host", "window"):
        y = y0
        for s in range(steps):
            y = d.integrate(y, d.rate_constants(w, s), w.dt)
        end = conc.clone()
        end[d.var] = y
        return {"conc": end if kind == "window" else end.cpu().numpy(), "status": None, "accepted": None,
                "rejected": None}
    for r in MODERATED.get(mech, ()):
        k[r].clamp_(max=1e3)
    lam, dconc, dk = (_device(a) for a in _directions(case, seed, w))
    dk = dk * k
    record = []
    y = d.integrate(y0, k, w.dt, record)
    end = conc.clone()
    end[d.var] = y
    if kind == "tangent":
        v = dconc[d.var].clone()
        for idx, yi, h in record:
            if idx.numel():
                _, dv = torch.func.jvp(lambda a, b: a + d.attempt(a, b, h)[0], (yi, k[:, idx]),
                                       (v[:, idx], dk[:, idx]))
                v[:, idx] = dv
        slope = dconc.clone()
        slope[d.var] = v
        return {"conc": end, "dconc": slope}
    g, gk = lam[d.var].clone(), torch.zeros_like(k)
    for idx, yi, h in reversed(record):
        if idx.numel():
            a, b = yi.detach().requires_grad_(True), k[:, idx].detach().requires_grad_(True)
            out = a + d.attempt(a, b, h)[0]
            ga, gb = torch.autograd.grad(out, (a, b), g[:, idx], allow_unused=True)
            g[:, idx] = ga
            gk[:, idx] += gb if gb is not None else 0.0
    grad = lam.clone()
    grad[d.var] = g
    if mech == "saprc99":
        # Its norm is that of one or two cells' sensitivity to BZNO2_O, a
        # radical at zero, in which two orders of elimination share no digit.
        grad = None
    return {"conc": end, "grad_conc": grad, "grad_k": gk}
