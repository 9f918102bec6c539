"""The kernels of the refinement loop where they cannot do what they usually
do: clusters that the GPU refuses (BEM_OPT_INJECT bits 2 and 3; the launch is
refused on the host), and vectors that the first pass of Gram-Schmidt reduces
to rounding."""
import ctypes

import pytest

from bem_gmsh_gb300 import _lib
from bem_gmsh_gb300.api import solve_system

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def system(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    A = (torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g) / n**0.5).t()
    A.diagonal().add_(2.0)
    b = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    torch.cuda.synchronize()
    return A, b


def residual(A, x, b):
    return float((A @ x - b).norm() / b.norm())


@pytest.mark.parametrize("n", [300, 4095, 4096, 4200])
def test_refused_clusters(n):
    """No cluster at all: an error, not the former solve's words as this one's
    (that solve's norm, coefficients and status look like success).  Only wide
    ones refused: the portable size takes their place."""
    A, b = system(n, n)
    limit = 1e-14 + 4 * 2.0**-53 * n**0.5  # the solver's target and the product formed here
    ctx = _lib.Context()
    try:
        x, st = solve_system(A, b, ctx=ctx)
        assert residual(A, x, b) <= limit
        ctx.set_option(_lib.BEM_OPT_INJECT, 8)
        for _ in range(2):
            with pytest.raises(_lib.BemError) as e:
                solve_system(A, 3.0 * b.flip(0), ctx=ctx)
            assert e.value.status == 2  # BEM_ERR_CUDA
        ctx.set_option(_lib.BEM_OPT_INJECT, 4)
        b2 = b.flip(0).contiguous()
        torch.cuda.synchronize()
        x, st2 = solve_system(A, b2, ctx=ctx)
        assert residual(A, x, b2) <= limit and abs(st2["iterations"] - st["iterations"]) <= 1
        ctx.set_option(_lib.BEM_OPT_INJECT, 0)
        x, _ = solve_system(A, b, ctx=ctx)
        assert residual(A, x, b) <= limit
    finally:
        ctx.close()


@pytest.mark.parametrize("N, m, breakdown", [(1, 1, True), (8, 8, True), (30, 30, True), (31, 30, False), (200, 7, False),
                                             (4096, 30, False), (20, 3, False)])
def test_gram_schmidt_norm(kernels, N, m, breakdown):
    """The coefficients, |w|^2 and the unit vector against 64-bit sums; with V a
    basis of the whole space (breakdown) what is left of w is the rounding of
    the second pass, and its norm is still the one of what is left."""
    g = torch.Generator(device="cuda").manual_seed(N + m)
    V = torch.linalg.qr(torch.randn(N, N if breakdown else m, dtype=torch.float64, device="cuda", generator=g))[0]
    V = V.t().contiguous()  # rows: the columns of a column-major V
    w = torch.randn(N, dtype=torch.float64, device="cuda", generator=g)
    w0, vn, host = w.clone(), torch.empty_like(w), torch.empty(64, dtype=torch.float64).pin_memory()
    f = kernels.h_gram_schmidt
    f.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int] + [ctypes.c_void_p] * 3
    torch.cuda.synchronize()
    assert f(V.data_ptr(), N, m, w.data_ptr(), vn.data_ptr(), host.data_ptr()) == 0
    h = host[:m].cuda() + host[32:32 + m].cuda()
    assert float((h - V @ w0).abs().max()) <= 1e-14 * float(w0.norm())  # two sums of N roundings each
    n2, unit = float(host[62]), float(vn.norm())
    if n2 > 0.0:
        assert abs(unit - 1.0) <= 1e-14, (n2, unit)
    else:
        assert unit == 0.0
    if breakdown:
        assert 0.0 <= n2 <= (1e-28 * N * float(w0.norm())) ** 2  # twice reduced to rounding
    else:
        rest = w0 - V.t() @ (V @ w0)
        assert abs(n2 - float(rest @ rest)) <= 1e-13 * float(w0 @ w0)
        assert float((V @ vn).abs().max()) <= 1e-14
