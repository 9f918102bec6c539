"""The kernels of the refinement loop where they cannot do what they usually
do: clusters that the GPU refuses (BEM_OPT_INJECT bits 2 and 3; the launch is
refused on the host)."""
import numpy as np
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
