"""The short FP64 functions of the element integrals on the device, from the
hardware's starting values, against IEEE results and 64 bits and more."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

LOG, DIV, RCP, SQRT, TAN, TAN_FULL = range(6)
EDGES = np.array([0.0, -0.0, -1.0, np.inf, -np.inf, np.nan, 5e-324, 2.2e-308, 2.0**-1000, 2.0**-500, 2.0**-499, 2.0**-498,
                  2.0**499, 2.0**500, 2.0**501, 1.7e308, 1.0, 2.0, 0.5, 3.0])


@pytest.fixture(scope="module")
def call(kernels):
    f = kernels.h_function
    f.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]

    def g(which, x, y=None):
        x = torch.from_numpy(np.ascontiguousarray(x)).cuda()
        y = x if y is None else torch.from_numpy(np.ascontiguousarray(y)).cuda()
        o = torch.empty_like(x)
        torch.cuda.synchronize()
        assert f(which, x.data_ptr(), y.data_ptr(), x.numel(), o.data_ptr()) == 0
        return o.cpu().numpy()

    return g


def numbers(rng, n):
    return rng.standard_normal(n) * np.exp(rng.uniform(-30, 30, n))


def test_quotients(call):
    """Within 2^-75 before the rounding: the IEEE quotient for all but one
    argument in 2^21, and everywhere outside the plain range."""
    rng = np.random.default_rng(0)
    a, b = numbers(rng, 1 << 20), numbers(rng, 1 << 20)
    for got, ref in ((call(DIV, a, b), a / b), (call(RCP, b), 1.0 / b)):
        assert np.count_nonzero(got != ref) <= 5
        assert np.all(np.abs(got - ref) <= np.spacing(np.abs(ref)))
    x, y = (v.ravel().copy() for v in np.meshgrid(EDGES, EDGES))
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(call(DIV, x, y), x / y)
        np.testing.assert_array_equal(call(RCP, EDGES), 1.0 / EDGES)


def test_square_root(call):
    a = np.abs(numbers(np.random.default_rng(1), 1 << 20))
    s = np.sqrt(a.astype(np.longdouble))
    assert np.all(np.abs(call(SQRT, a) - s) <= 0.51 * np.spacing(s.astype(np.float64)))
    with np.errstate(all="ignore"):
        np.testing.assert_allclose(call(SQRT, EDGES), np.sqrt(EDGES), rtol=2.0**-52)


def test_logarithm(call):
    rng = np.random.default_rng(2)
    c = 1 + np.arange(129) / 128
    x = np.concatenate([np.exp(rng.uniform(-40, 40, 1 << 19)), 1 + rng.uniform(-0.01, 0.01, 1 << 18),
                        1 + rng.uniform(-1, 1, 4000) * 2.0 ** -rng.integers(20, 52, 4000),
                        np.nextafter(c, 0), c, np.nextafter(c + 1 / 256, 9), c - 1 / 256, [1e-300, 1e300]])
    ref = np.log(x.astype(np.longdouble))
    ulp = np.spacing(np.abs(ref.astype(np.float64)))
    # half an ulp and the rounding of log1p's last term, 2^-61, or two ulp
    assert np.all(np.abs(call(LOG, x) - ref) <= np.maximum(0.51 * ulp, np.minimum(0.5 * ulp + 2.0**-60, 2 * ulp)))
    with np.errstate(all="ignore"):
        np.testing.assert_allclose(call(LOG, EDGES), np.log(EDGES), rtol=2.0**-52)


def test_tangent(call):
    rng = np.random.default_rng(3)
    n = 1 << 18
    x = np.concatenate([rng.uniform(-2.5, 2.5, n), rng.uniform(-1, 1, n) * 2.0 ** -rng.integers(0, 30, n),
                        np.pi / 2 + rng.uniform(-1, 1, n) * 2.0 ** -rng.integers(0, 40, n)])
    np.testing.assert_array_equal(call(TAN, x), call(TAN_FULL, x))
