"""Rate-constant texts of a user's mechanism through the emitted rate code
(CPU).

The rate kernel evaluates the texts on mkpp::Num, a double whose divisions
are integer code.  Every C expression of doubles has to compile there as it
does on doubles, and to give the same bits; here the emitted
``rate_constants_part`` is built for the host (tests/hostsim/), where Num
divides as double does.
"""

import copy
import ctypes as C
import math
import subprocess
from pathlib import Path

import numpy as np
import pytest

from mkpp_gb300.emitter import cuda_emitter
from mkpp_gb300.emitter.plan import load_raw, reduce_plan

HERE = Path(__file__).resolve().parent
ROOT = HERE.parent

DRIVER = r"""
#include MKPP_MECH_HEADER
namespace {
using Mech = MKPP_MECH_NS::Mech;
struct Row { const double* v; double operator()(int i) const { return v[i]; } };
struct Out { double* v; void set(int i, double x) const { v[i] = x; } };
template <class V> void run(const double* fix, const double* par, double T, double RHO, double RH, double CLW, double* k) {
  Out out{k};
  for (int p = 0; p < Mech::RATE_PARTS; ++p)
    Mech::rate_constants_part(p, Row{par}, Row{fix}, V(T), V(RHO), V(RH), V(CLW), out);
}
}
extern "C" void rates(int num, const double* fix, const double* par, double T, double RHO, double RH, double CLW, double* k) {
  if (num) run<mkpp::Num>(fix, par, T, RHO, RH, CLW, k);
  else run<double>(fix, par, T, RHO, RH, CLW, k);
}
"""

# (C text, its value)
TEXTS = [
    ("cbrt(T)*1.0e-3", lambda T, RHO, RH: math.cbrt(T) * 1.0e-3),
    ("log10(T)", lambda T, RHO, RH: math.log10(T)),
    ("fmin(T, 300.0)/7.0", lambda T, RHO, RH: min(T, 300.0) / 7.0),
    ("fmax(250.0, T)", lambda T, RHO, RH: max(250.0, T)),
    ("tanh(T/300.0)", lambda T, RHO, RH: math.tanh(T / 300.0)),
    ("T > 300.0 ? 1.0e-3 : T/3.0e5", lambda T, RHO, RH: 1.0e-3 if T > 300.0 else T / 3.0e5),
    ("(T <= 300.0 && RH > 0.1)*2.5", lambda T, RHO, RH: (T <= 300.0 and RH > 0.1) * 2.5),
    ("+T/3.0", lambda T, RHO, RH: T / 3.0),
    ("2*(+T)/3", lambda T, RHO, RH: 2 * T / 3),
    ("std::exp(-1/T)", lambda T, RHO, RH: math.exp(-1 / T)),
    ("1.f/T", lambda T, RHO, RH: 1.0 / T),
    ("pow(10, -3)*RHO/T", lambda T, RHO, RH: math.pow(10, -3) * RHO / T),
    ("1/(1/T + 1.0e-3)", lambda T, RHO, RH: 1 / (1 / T + 1.0e-3)),
    ("4", lambda T, RHO, RH: 4.0),
]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("rates")
    raw = copy.deepcopy(load_raw("chapman"))
    proto = raw["reactions"]
    raw["reactions"] = []
    for i, (text, _) in enumerate(TEXTS):
        r = copy.deepcopy(proto[i % len(proto)])
        r.update(index=i, k=text, dk_dfixed=[])
        raw["reactions"].append(r)
    raw["num_reactions"] = len(TEXTS)
    (tmp / "texts.cuh").write_text(cuda_emitter.emit_mechanism(reduce_plan(raw)))
    (tmp / "driver.cpp").write_text(DRIVER)
    so = tmp / "texts.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", f"-I{HERE / 'hostsim'}",
                    f"-I{tmp}", f"-I{ROOT / 'mkpp_gb300' / 'csrc'}", '-DMKPP_MECH_HEADER="texts.cuh"',
                    f"-DMKPP_MECH_NS=mkpp_{raw['name']}", str(tmp / "driver.cpp"), "-o", str(so)], check=True)
    return C.CDLL(str(so))


@pytest.mark.parametrize("T, RHO, RH", [(298.15, 2.46e19, 0.5), (301.0, 1.0e19, 0.05), (173.7, 3.0e17, 0.9)])
def test_every_text_of_doubles_compiles_and_keeps_its_value(lib, T, RHO, RH):
    fix, par = np.zeros(64), np.zeros(64)
    got = np.full((2, len(TEXTS)), np.nan)
    for num in (0, 1):
        lib.rates(num, C.c_void_p(fix.ctypes.data), C.c_void_p(par.ctypes.data), C.c_double(T), C.c_double(RHO),
                  C.c_double(RH), C.c_double(0.0), C.c_void_p(got[num].ctypes.data))
    assert np.array_equal(got[0], got[1])
    # A function of the C library may round the last bit otherwise than Python's.
    np.testing.assert_allclose(got[0], [f(T, RHO, RH) for _, f in TEXTS], rtol=4e-16, atol=0)


def test_texts_without_such_functions_stay_on_num():
    for text in ("1.0e-12*exp(-1775.0/T)", "RHO*pow(T/300.0, -2.4)/(1 + 3.5*P[0])", "FIX[2]*log(T)", "2.e3/T", "-T"):
        assert cuda_emitter._k_value(text).startswith("mkpp::value(")
