"""The FP64 arithmetic of the generated right-hand sides against 80-bit arithmetic and IEEE 754's special values."""
import ctypes as C
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

import helpers as H
from opendihu_b200 import build as B
from opendihu_b200 import cellml as CM

pytestmark = pytest.mark.gpu


def _library(path, model, params_const=(), params_alg=()):
    """tests/cpp/math_functions.cu compiled with the model's right-hand side"""
    (path / "test_model.cuh").write_text(
        CM.emit_cuda_model(model, params_alg, params_const)
        + f"\n#define TEST_MODEL fdm_model_{CM._ident(model)}_{CM.variant_tag(params_alg, params_const)}\n"
        + f"#define TEST_SCALE {CM._exp_scale_text(Fraction(-1, 10))}\n"
        + f"#define TEST_OFFSET {CM._exp_offset_text(Fraction(-3, 2))}\n")
    lib = str(path / "math_functions.so")
    r = subprocess.run([B.nvcc()] + B.NVCC_FLAGS + ["-I", B.CSRC, "-I", os.path.join(B.CSRC, "generated"), "-I", str(path),
                                                    "-shared", "-o", lib,
                                                    os.path.join(H.ROOT, "tests/cpp/math_functions.cu")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(lib)


def _pointer(a):
    return a.ctypes.data_as(C.c_void_p)


@pytest.fixture(scope="module")
def hodgkin_huxley(tmp_path_factory):
    return _library(tmp_path_factory.mktemp("hh"), CM.builtin_model(H.HH), (2, 3, 4))


def _model(name, n_algebraics, constants, lines, n_states):
    return CM.Model(name=name, source=name + ".c", n_states=n_states, n_algebraics=n_algebraics,
                    n_constants=len(constants), states_initial=[0.0] * n_states, constants=constants, constant_lines=[],
                    lines=[(kind, k, CM.parse_expression(text)) for kind, k, text in lines])


@pytest.fixture(scope="module")
def hill(tmp_path_factory):
    """A Hill term, a Boltzmann term and a bare exponential, a quotient of states"""
    return _library(tmp_path_factory.mktemp("hill"), _model("hill", 3, [0.5], [
        ("A", 0, "1.00000/(1.00000+CONSTANTS[0]/STATES[1])"), ("A", 1, "1.00000/(1.00000+exp(STATES[0]/3.00000))"),
        ("A", 2, "exp(STATES[0]/7.00000)"), ("R", 0, "ALGEBRAIC[0]"), ("R", 1, "ALGEBRAIC[1]"), ("R", 2, "ALGEBRAIC[2]"),
        ("R", 3, "STATES[2]/STATES[1]")], 4))


def _function(lib, f, x, y=None):
    x = np.ascontiguousarray(x, np.float64)
    y = x if y is None else np.ascontiguousarray(y, np.float64)
    out = np.empty_like(x)
    assert lib.eval_function(C.c_int(f), C.c_int64(len(x)), _pointer(x), _pointer(y), _pointer(out)) == 0
    return out


def _rates(lib, approximate, states, params=np.zeros((1, 1))):
    states, params = np.ascontiguousarray(states, np.float64), np.ascontiguousarray(params, np.float64)
    ns, n = states.shape
    out = np.empty((ns, n))
    assert lib.eval_rates(C.c_int(int(approximate)), C.c_int64(n), C.c_double(0.0), _pointer(states), _pointer(params),
                          _pointer(out)) == 0
    return out


def _ulps(got, exact):
    """|got - exact| in units of the last place of exact (80-bit)"""
    assert np.finfo(np.longdouble).nmant >= 63
    return np.abs(got.astype(np.longdouble) - exact) / np.spacing(np.abs(exact.astype(np.float64))).astype(np.longdouble)


def _exp_arguments():
    rng = np.random.default_rng(1)
    k = np.arange(-1000, 1024)
    edges = (k + 0.5) * np.log(2.0)          # the argument's reduction changes its multiple of ln 2
    near = np.concatenate([edges + d * np.spacing(np.abs(edges)) for d in (-2, -1, 0, 1, 2)])
    return np.concatenate([near, k * np.log(2.0), *(rng.uniform(-a, a, 200000) for a in (0.35, 1.0, 5.0, 40.0, 700.0)),
                           10.0 ** rng.uniform(-300, 0, 1000), -10.0 ** rng.uniform(-300, 0, 1000), [-708.0, 709.78]])


# Half an ulp of the last rounding; the polynomial (3.4e-17 and its evaluation) and the roundings of the small terms,
# relative to a result of at least 0.7, are below the other half.  exp(-x/10): the rounding of 1 + r and of r twice
# (2^-55 each) besides.
def test_exponential(hodgkin_huxley):
    x = _exp_arguments()
    assert _ulps(_function(hodgkin_huxley, 0, x), np.exp(x.astype(np.longdouble))).max() < 1.0
    x = 10.0 * x[np.abs(x) < 40.0]
    assert _ulps(_function(hodgkin_huxley, 4, x), np.exp(-x.astype(np.longdouble) / 10)).max() < 1.4
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 709.79, 1e300, -1e300, -750.0, 1e-310])
    big = 2.0 ** 1020
    np.testing.assert_array_equal(_function(hodgkin_huxley, 0, x), [1, 1, np.inf, 0, np.nan, np.inf, np.inf, 0, 0, 1])
    np.testing.assert_array_equal(_function(hodgkin_huxley, 6, x), [1, 1, big, 0, np.nan, big, big, 0, 0, 1])
    np.testing.assert_array_equal(_function(hodgkin_huxley, 4, -10.0 * x), [1, 1, np.inf, 0, np.nan, np.inf, np.inf, 0, 0, 1])


# Half an ulp of the last rounding; where 2 (exp(r) - 1) + 1 cancels (x near ln(2)/2: the result is 0.41, its terms 0.59
# and 1) the other roundings, half an ulp of 0.29 and the polynomial's 3.4e-17, count 2 of the result's ulps at most.
# exp(-x/10) - 1: there the two roundings of r another 1.5.
def test_exponential_minus_one(hodgkin_huxley):
    x = _exp_arguments()
    assert _ulps(_function(hodgkin_huxley, 3, x), np.expm1(x.astype(np.longdouble))).max() < 2.5
    x = 10.0 * x[np.abs(x) < 40.0]
    assert _ulps(_function(hodgkin_huxley, 5, x), np.expm1(-x.astype(np.longdouble) / 10)).max() < 4.0
    x = np.array([0.0, np.inf, -np.inf, np.nan, 709.79, 1e300, -1e300, -750.0])
    np.testing.assert_array_equal(_function(hodgkin_huxley, 3, x), [0, np.inf, -1, np.nan, np.inf, np.inf, -1, -1])
    np.testing.assert_array_equal(_function(hodgkin_huxley, 5, -10.0 * x), [0, np.inf, -1, np.nan, np.inf, np.inf, -1, -1])


# The members of a group, exp(-x/10 - b): the polynomial's 3.4e-17 relative to exp(r) >= 0.7, R as c R (2e-17) and the
# sum's and the product's last roundings are below 1.2 ulp.  Minus 1: two roundings at the result's size, at most 1 ulp,
# and what the exponential brings in before the subtraction, 0.6 of 2^-53 of it.
def test_exponential_group(hodgkin_huxley):
    rng = np.random.default_rng(4)
    x = np.concatenate([10.0 * _exp_arguments(), *(-15.0 + s * 10.0 ** rng.uniform(-12, 1, 100000) for s in (1, -1))])
    x = x[np.abs(x) < 400.0]
    with np.errstate(divide="ignore", invalid="ignore"):
        for f, b in ((7, 1.5), (9, 0.0)):
            exact = np.exp(-x.astype(np.longdouble) / 10 - b)
            assert _ulps(_function(hodgkin_huxley, f, x), exact).max() < 1.3
            exact_m1 = np.expm1(-x.astype(np.longdouble) / 10 - b)
            error = np.abs(_function(hodgkin_huxley, f + 1, x) - exact_m1)
            assert np.all(error <= np.spacing(np.abs(exact_m1).astype(float)) + 0.7 * 2.0 ** -53 * exact)
    x = np.array([np.nan, np.inf, -np.inf, 7.1e3, -7.1e3])
    got = _function(hodgkin_huxley, 8, x)
    assert np.isnan(got[0]) and np.all(got[[1, 3]] == -1.0) and np.all((got[[2, 4]] > 1e300) & (got[[2, 4]] < 1e305))


SPECIAL = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-310, -3e-320, 2.0 ** -1022, 1e-300, 1.0, -3.5, 1e300,
                    2.0 ** 1020, 2.0 ** 1021, 2.0 ** 1022, 1e308, -1.7e308])


# one rounding of a correction that is exact to 2^-100; the reciprocal's cubic step leaves the third power of the
# approximation's error, 2^-60 of the result at most
def test_division_and_reciprocal(hill):
    rng = np.random.default_rng(2)
    a, b = (rng.uniform(1.0, 2.0, 1000000) * 2.0 ** rng.integers(-400, 400, 1000000) for _ in range(2))
    a[::2] *= -1.0
    exact = a.astype(np.longdouble) / b
    for f in (2, 11):
        assert _ulps(_function(hill, f, a, b), exact).max() < 0.51
    assert _ulps(_function(hill, 1, b), 1 / b.astype(np.longdouble)).max() < 0.52
    # the quotient's divisor may reach beyond 2^1022, where its reciprocal is subnormal
    assert np.all(np.abs(_function(hill, 2, np.ones(2), np.array([2.0 ** 1022, 1e308]))) < 1e-307)
    a, b = (m.ravel() for m in np.meshgrid(SPECIAL, SPECIAL))
    with np.errstate(all="ignore"):
        np.testing.assert_allclose(_function(hill, 11, a, b), a / b, rtol=1e-15, atol=5e-324)
        want = np.where(np.abs(SPECIAL) < 2.0 ** 1021, 1 / SPECIAL, 0.0 * SPECIAL)    # subnormal results flushed
        want[np.isnan(SPECIAL)], want[np.isinf(SPECIAL)] = np.nan, 0.0
        np.testing.assert_allclose(_function(hill, 1, SPECIAL), want, rtol=1e-15, atol=2.0 ** -1021)


# as IEEE arithmetic has them: 1/(1 + K/c) is 0 at c = 0, 1/(1 + exp(v)) is 0 where exp(v) overflows
@pytest.mark.parametrize("approximate", [False, True])
def test_terms_with_vanishing_and_infinite_divisors(hill, approximate):
    v = np.array([-6000.0, -300.0, -70.0, 0.0, 70.0, 300.0, 1500.0, 2100.0, 4000.0, 1e6])
    c = np.array([0.0, 1e-310, 1e-300, 1e-3, 0.5, 1.0, 1e3, 1e308, np.inf, 0.0])
    d = np.array([1.0, 1e-305, 0.0, 2.0, -3.0, 1e300, np.inf, 1e308, 7.0, 0.0])
    with np.errstate(all="ignore"):
        e3, e7 = ((1 + v / 3 / 1024) ** 1024, (1 + v / 7 / 1024) ** 1024) if approximate else (np.exp(v / 3), np.exp(v / 7))
        want = np.stack([1 / (1 + 0.5 / c), 1 / (1 + e3), e7, d / c])
    # arguments of up to 857 lose 2^-53 of themselves; the approximate exponential's 1024th power 1e-13
    np.testing.assert_allclose(_rates(hill, approximate, np.stack([v, c, d, c])), want, rtol=4e-13, atol=1e-300)


# alpha_m = x / (exp(x) - 1) at V = -50 mV, alpha_n at -65 mV, around their removable singularities.  alpha_m is as
# exact there as elsewhere; 20 mV away, in halves of an ulp: the argument's 2.5 times u e^u / (e^u - 1) = 2.3, the
# numerator's 2.5, the exponential's 4, quotient, difference, product and sum 4: 17.  alpha_n's exponential is alpha_m's
# times e^-1.5: before 1 is subtracted it is off by 0.7 of 2^-53 at most (an exponential by itself: by 1).
@pytest.mark.parametrize("singularity", [-50.0, -65.0])
def test_rates_at_removable_singularities(hodgkin_huxley, singularity):
    rng = np.random.default_rng(3)
    n = 20000
    v = singularity + np.where(np.arange(n) % 2, 1.0, -1.0) * 10.0 ** rng.uniform(-13, 1.3, n)
    states = np.stack([v, *rng.uniform(0.0, 1.0, (3, n))])
    params = np.stack([np.zeros(n), np.full(n, 120.0), np.full(n, 36.0)])
    V, m, h, g = states.astype(np.longdouble)
    tenth = np.longdouble(1) / 10
    # at the singularity itself the quotient is 0/0, as the equations are
    at = np.repeat([[singularity], [0.1], [0.5], [0.3]], 2, axis=1)
    assert np.isnan(_rates(hodgkin_huxley, False, at, params[:, :2])[1 if singularity == -50.0 else 3]).all()
    got = _rates(hodgkin_huxley, False, states, params)
    for k, y, top, scale, centre, beta in ((1, m, tenth, 10, 50, 4 * np.exp(-(V + 75) / 18)),
                                           (3, g, tenth / 10, 10, 65, np.exp((V + 75) / 80) / 8)):
        alpha = -(V + centre) * top / np.expm1(-(V + centre) / scale)
        error = np.abs(got[k] - (alpha * (1 - y) - beta * y))
        u = np.abs(V + centre) / 10
        cancelled = 0.7 * (1 + 1 / u) * alpha * (1 - y) if k == 3 else 0
        assert np.all(error < 2.0 ** -53 * (18 * (alpha * (1 - y) + beta * y) + cancelled))


# random states around the initial ones, against the equations in C; the tolerances are those of the plain form's test
@pytest.mark.parametrize("model,approximate", [(H.HH, False), (H.HH, True), (H.SHORTEN, False), (H.SHORTEN, True)])
def test_rates_match_equations(model, approximate, tmp_path):
    import test_gpu_cellml_rhs as R
    from opendihu_b200.solver import VARIANT_PARAMETERS
    params_alg, params_const = VARIANT_PARAMETERS[model]
    lib = _library(tmp_path, CM.builtin_model(model), params_const, params_alg)
    states, params, ns, _ = R._inputs(model, 500, 4)
    want, _ = R._oracle(model, states, params, 0.0, approximate)
    np.testing.assert_allclose(_rates(lib, approximate, states, params), want, rtol=1e-11, atol=1e-12 * np.abs(want).max())
