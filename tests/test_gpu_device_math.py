"""The FP64 helpers as the kernels call them (tests/device_math/dev_math.cu compiles
csrc/tns_device.cuh and csrc/tns_adjoint.cuh), against 64-bit-mantissa references.

Bounds, in u = 2^-53, from the steps of each helper.  recip: an estimate good to 2^-20 and two
quadratic steps leave 2^-80 before the last rounding, so u and a little; root likewise from 2^-22;
quot corrects its product's rounding, u.  fifth_roots: the residual carries two roundings (2 u), of
which the corrections take 0.4 and 0.6 a power, and the last rounding: 2 u for T^-0.4, and 3.2 u
with the rounding of y^3 for T^-0.6.  expm1: 4 u, as the older test has it.  The ratios: every
expm1 is off by 2 u and its argument by 2 u (tanh's condition number is at most 1), and each sum,
product and reciprocal adds u: 16 u for FMU, 18 u with the square root for FR2, 14 u for FMU alone;
the reverse's tanh and its reciprocal 5 u, its derivative 14 u (two reciprocals squared).
inlet_density: 8 u in an exponent below 0.72, exp 2 u, the constants and products 4 u; on pow's
side the constants are raised to the 2.5th power: 20 u for both."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from tnsgpu import cases, formats
from tnsgpu.solver import make_params

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
U = 2.0 ** -53
RECIP, ROOT_, QUOT, M04, M06, FMU, FR2, FMU1, TANH, TANH_INV, TANH_D, INLET, EXPM1 = range(13)
ALPHA, BETA = np.longdouble(0.00052), np.longdouble(0.2)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc is needed to compile the harness")
    out = str(tmp_path_factory.mktemp("devmath") / "libdevmath.so")
    subprocess.run(["nvcc", "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC",
                    "-shared", os.path.join(ROOT, "tests", "device_math", "dev_math.cu"), "-o", out], check=True)
    L = C.CDLL(out)
    L.dev_math_fr2k.restype = C.c_double
    return L


@pytest.fixture(scope="module")
def params():
    flow = cases.ramp_flow()
    return make_params(flow, formats.rinit_cold(flow))


def _eval(lib, params, fn, a, b=None):
    a = np.ascontiguousarray(a, np.float64)
    b = np.ascontiguousarray(a if b is None else b, np.float64)
    out = np.empty_like(a)
    assert lib.dev_math(fn, C.byref(params), C.c_longlong(a.size), C.c_void_p(a.ctypes.data), C.c_void_p(b.ctypes.data),
                        C.c_void_p(out.ctypes.data)) == 0
    return out


def _check(got, ref, bound):
    rel = np.abs((got.astype(np.longdouble) - ref) / ref)
    k = int(np.argmax(rel))
    assert np.all(np.isfinite(got)) and rel[k] <= bound, (k, float(rel[k] / U), got[k], float(ref[k]))


def _spread(lo, hi, n=40000, seed=0):
    return 10.0 ** np.random.default_rng(seed).uniform(lo, hi, n)


def test_reciprocal_square_root_and_quotient(lib, params):
    x = np.concatenate([_spread(-290, 290), np.random.default_rng(1).uniform(0.5, 2.0, 40000),
                        np.nextafter(2.0 ** np.arange(-900, 900.0, 37), 0), 2.0 ** np.arange(-900, 900.0, 37)])
    lx = x.astype(np.longdouble)
    _check(_eval(lib, params, RECIP, x), 1 / lx, 1.01 * U)
    _check(_eval(lib, params, RECIP, -x), -1 / lx, 1.01 * U)
    _check(_eval(lib, params, ROOT_, x), np.sqrt(lx), 1.01 * U)
    assert _eval(lib, params, ROOT_, np.zeros(3)).tolist() == [0.0, 0.0, 0.0]
    a, b = _spread(-140, 140, seed=2), _spread(-140, 140, seed=3)
    _check(_eval(lib, params, QUOT, a, b), a.astype(np.longdouble) / b, 1.01 * U)
    assert np.array_equal(_eval(lib, params, QUOT, np.zeros(2), np.array([3.0, -2.0])), [0.0, 0.0])
    # against CUDA's own division (IEEE): equal but for rare cases
    assert np.mean(_eval(lib, params, QUOT, a, b) != a / b) < 1e-3


def test_fifth_roots(lib, params):
    t = np.concatenate([_spread(0, 4), np.random.default_rng(4).uniform(100, 4000, 40000)])
    lt = t.astype(np.longdouble)
    _check(_eval(lib, params, M04, t), np.exp(-np.log(lt) * 2 / 5), 2.2 * U)
    _check(_eval(lib, params, M06, t), np.exp(-np.log(lt) * 3 / 5), 3.4 * U)


def test_expm1(lib, params):
    x = np.concatenate([_spread(-300, -1), np.random.default_rng(5).uniform(0, 40, 40000), [np.log(2) / 2, 40.0]])
    _check(_eval(lib, params, EXPM1, x), np.expm1(x.astype(np.longdouble)), 4 * U)


def _chi():
    """Small and large CHI, and both sides of the arguments at which a tanh counts as 1."""
    at = np.array([10.0, 20.0 / np.sqrt(2.0 * 0.3), 400.0, np.sqrt(20.0 / 0.00052)])
    near = (at[:, None] * (1 + np.linspace(-1e-3, 1e-3, 201))).ravel()
    return np.concatenate([_spread(-150, -3, seed=6), _spread(-3, 4, seed=7), near])


def test_damping_ratios(lib, params):
    chi = _chi()
    x = chi.astype(np.longdouble)
    fmu = np.tanh(ALPHA * x * x) / np.tanh(BETA * x * x)
    _check(_eval(lib, params, FMU, chi), fmu, 16 * U)
    _check(_eval(lib, params, FMU1, chi), fmu, 14 * U)
    k = np.longdouble(lib.dev_math_fr2k(C.byref(params)))
    _check(_eval(lib, params, FR2, chi), np.tanh(np.sqrt(x)) / np.tanh(x * k), 18 * U)


def test_reverse_tanh(lib, params):
    x = np.concatenate([_spread(-150, 0, seed=8), np.random.default_rng(9).uniform(0, 19.99, 40000)])
    lx = x.astype(np.longdouble)
    t = np.tanh(lx)
    _check(_eval(lib, params, TANH, x), t, 5 * U)
    _check(_eval(lib, params, TANH_INV, x), 1 / t, 5 * U)
    _check(_eval(lib, params, TANH_D, x), 1 / np.cosh(lx) ** 2, 14 * U)
    assert np.all(_eval(lib, params, TANH_D, np.array([20.0, 50.0])) == 0.0)


def test_inlet_density(lib, params):
    t0, g = np.longdouble(params.t0), np.longdouble(params.gama)
    rr = np.longdouble(8314.0) / np.longdouble(params.amol)
    z = np.concatenate([np.random.default_rng(10).uniform(-0.2, 0.5, 40000), _spread(-15, -1, seed=11),
                        0.25 + np.linspace(-1e-6, 1e-6, 101), [0.0]])
    t = (float(params.t0) * (1 - z)).astype(np.float64)
    ref = np.longdouble(params.p0) / (rr * t0) * (t.astype(np.longdouble) / t0) ** (1 / (g - 1))
    _check(_eval(lib, params, INLET, t), ref, 20 * U)
