"""FP64 log, quotient and square root of the element integrals (fast64.cuh), on
the host, against long double (at least 64 bits): the device differs in the
starting approximations only, which the last correction absorbs."""
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


EDGES = np.array([0.0, -0.0, -1.0, np.inf, -np.inf, np.nan, 5e-324, 2.2e-308, 1e-300, 1.7e308, 1.0, 2.0, 0.5])


def test_log(h):
    rng = np.random.default_rng(0)
    c = 1 + np.arange(129) / 128
    x = np.concatenate([np.exp(rng.uniform(-40, 40, 200000)), 1 + rng.uniform(-0.01, 0.01, 50000),
                        1 + rng.uniform(-1, 1, 2000) * 2.0 ** -rng.integers(20, 52, 2000),
                        np.nextafter(c, 0), c, np.nextafter(c + 1 / 256, 9), c - 1 / 256, [1e-300, 1e300]])
    ref = np.log(x.astype(np.longdouble))
    err = np.abs(_call(h.h_log, x) - ref)
    ulp = np.spacing(np.abs(ref.astype(np.float64)))
    # half an ulp and the rounding of log1p's last term, 2^-61, or two ulp
    assert np.all(err <= np.maximum(0.51 * ulp, np.minimum(0.5 * ulp + 2.0 ** -60, 2 * ulp)))
    with np.errstate(all="ignore"):
        assert np.array_equal(_call(h.h_log, EDGES), np.log(EDGES), equal_nan=True) or \
            np.allclose(_call(h.h_log, EDGES), np.log(EDGES), rtol=2e-16, equal_nan=True)


def test_div_and_sqrt(h):
    rng = np.random.default_rng(1)
    a = rng.standard_normal(200000) * np.exp(rng.uniform(-30, 30, 200000))
    b = rng.standard_normal(200000) * np.exp(rng.uniform(-30, 30, 200000))
    q = a.astype(np.longdouble) / b
    assert np.all(np.abs(_call(h.h_div, a, b) - q) <= 0.501 * np.spacing(np.abs(q.astype(np.float64))))
    s = np.sqrt(np.abs(a).astype(np.longdouble))
    assert np.all(np.abs(_call(h.h_sqrt, np.abs(a)) - s) <= 0.51 * np.spacing(s.astype(np.float64)))
    x, y = (v.ravel() for v in np.meshgrid(EDGES, EDGES))
    with np.errstate(all="ignore"):
        np.testing.assert_allclose(_call(h.h_div, x, y), x / y, rtol=2e-16)
        np.testing.assert_allclose(_call(h.h_sqrt, EDGES), np.sqrt(EDGES), rtol=2e-16)


def test_log_table(h):
    mpmath = pytest.importorskip("mpmath")
    mpmath.mp.prec = 300
    t = np.zeros(389)
    h.h_table(t.ctypes.data_as(P))
    assert t[0] == 1.0 and t[384] == 0.5 and t[385] == t[387] and t[386] == t[388]
    for i in range(129):
        rc, hi, lo = t[3 * i:3 * i + 3]
        assert abs(rc * (1 + i / 128) - 1) <= 2.0 ** -15
        assert float(hi * 2.0 ** 42).is_integer()
        assert lo == float(-mpmath.log(mpmath.mpf(float(rc))) - mpmath.mpf(float(hi)))
    assert t[388] == float(mpmath.log(2) - mpmath.mpf(float(t[387])))
