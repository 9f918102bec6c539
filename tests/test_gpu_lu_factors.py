"""The factors of the look-ahead LU against 64 bits: |L U - A| with steps in
pairs (BEM_OPT_TCGEN05 = 2, above 3712 columns) and without (1)."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def factor(kernels):
    f = kernels.h_factor
    f.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int]

    def error(A, variant):
        n = A.shape[0]
        F = torch.empty(n, n, dtype=torch.float32, device="cuda")
        cs = torch.empty(n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert f(A.data_ptr(), n, F.data_ptr(), cs.data_ptr(), variant) == 0
        F = F.t().double()
        L = torch.tril(F, -1)
        L.diagonal().add_(1.0)
        As = A * cs
        return float((L @ torch.triu(F) - As).norm() / As.norm())

    return error


@pytest.mark.parametrize("signs", ["random", "positive"])
@pytest.mark.parametrize("n", [3712, 4608, 6144])
def test_pairs_lose_no_bits(factor, n, signs):
    """Two steps in one pass over the matrix are as accurate as one by one: the
    same products and one rounding of the matrix less.  (Tensor cores truncate
    their running sums; one sum over both steps would double the error where
    the terms have one sign and add a third where they have none.)"""
    g = torch.Generator(device="cuda").manual_seed(n)
    make = torch.randn if signs == "random" else torch.rand
    A = (make(n, n, dtype=torch.float64, device="cuda", generator=g) / n**0.5).t()
    A.diagonal().add_(2.0 if signs == "random" else 2.0 * n**0.5)
    one, two = factor(A, 1), factor(A, 2)
    # 5 %: the spread between matrices of sums of 10^7 roundings is far less
    assert two <= 1.05 * one and one <= 1e-6, (one, two)
