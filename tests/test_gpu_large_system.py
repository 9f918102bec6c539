"""A system with more block rows than the GPU keeps resident (152 SMs, one CTA
of the sweeps each): sweeps in steps, one launch after another."""
import pytest

from bem_gmsh_gb300 import _lib
from bem_gmsh_gb300.api import solve_system

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n, stepwise", [(19456, False), (19457, True)])
def test_sweeps_in_steps(n, stepwise):
    g = torch.Generator(device="cuda").manual_seed(n)
    A = (torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g) / n**0.5).t()
    A.diagonal().add_(2.0)
    b = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    torch.cuda.synchronize()
    ctx = _lib.Context()
    try:
        before = ctx.launch_count()
        x, st = solve_system(A, b, ctx=ctx)
        launches = ctx.launch_count() - before
        torch.cuda.synchronize()
        # the solver's own target plus the rounding of the product formed here
        assert float((A @ x - b).norm() / b.norm()) <= 1e-14 + 4 * 2.0**-53 * n**0.5
        assert st["iterations"] <= 8 and not st["pivoted"]
        # per application 4 K launches in steps, one else; about five K for the factorization
        K = -(-n // 128)
        steps = 4 * K * st["iterations"]
        assert (steps < launches < steps + 8 * K) if stepwise else launches < 8 * K, launches
    finally:
        ctx.close()
