"""Quotient, reciprocal, square root and tangent of the element integrals on
the host with starting values of the hardware's length (20 bits): every
refinement step is needed to reach the stated errors."""
import ctypes
import os
import subprocess
import tempfile

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
P = ctypes.POINTER(ctypes.c_double)


@pytest.fixture(scope="module")
def h():
    so = os.path.join(tempfile.mkdtemp(prefix="fast64_"), "libfast64.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                           os.path.join(HERE, "native", "fast64_harness.cpp"), "-o", so])
    return ctypes.CDLL(so)


def _call(f, *xs):
    xs = [np.ascontiguousarray(x, np.float64) for x in xs]
    out = np.empty_like(xs[0])
    f(*[x.ctypes.data_as(P) for x in xs], xs[0].size, out.ctypes.data_as(P))
    return out


def _numbers(rng, n):
    return rng.standard_normal(n) * np.exp(rng.uniform(-30, 30, n))


def test_quotients_are_rounded(h):
    """A result within 2^-75 before its rounding is the rounded quotient for
    all but one argument in 2^21."""
    rng = np.random.default_rng(2)
    a, b = _numbers(rng, 400000), _numbers(rng, 400000)
    for got, ref in ((_call(h.h_div, a, b), a / b), (_call(h.h_rcp, b), 1.0 / b)):
        assert np.count_nonzero(got != ref) <= 3
        assert np.all(np.abs(got - ref) <= np.spacing(np.abs(ref)))
    edges = np.array([0.0, np.inf, -np.inf, np.nan, 5e-324, 2.0**-1000, 2.0**-499, 2.0**500, 1.7e308, -3.0])
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(_call(h.h_rcp, edges), 1.0 / edges)


def test_square_roots(h):
    a = np.abs(_numbers(np.random.default_rng(3), 400000))
    s = np.sqrt(a.astype(np.longdouble))
    got = _call(h.h_sqrt, a)
    assert np.all(np.abs(got - s) <= 0.51 * np.spacing(s.astype(np.float64)))
    assert np.count_nonzero(got != np.sqrt(a)) <= 0.02 * a.size


def test_tangent_decides_like_the_full_evaluation(h):
    rng = np.random.default_rng(4)
    n = 200000
    x = np.concatenate([rng.uniform(-2.5, 2.5, n), rng.uniform(-1, 1, n) * 2.0 ** -rng.integers(0, 30, n),
                        np.pi / 2 + rng.uniform(-1, 1, n) * 2.0 ** -rng.integers(0, 40, n)])
    np.testing.assert_array_equal(_call(h.h_tan, x), _call(h.h_tan_full, x))
