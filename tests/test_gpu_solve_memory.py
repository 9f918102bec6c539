"""Device memory a solve takes: operand buffers of the trailing updates for two
steps, for four only where steps share an update (above 3584 columns)."""
import pytest

from bem_gmsh_gb300 import _lib
from bem_gmsh_gb300.api import solve_system

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def taken(n, variant):
    """Bytes that the first solve of a context leaves allocated."""
    g = torch.Generator(device="cuda").manual_seed(n)
    A = (torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g) / n**0.5).t()
    A.diagonal().add_(2.0)
    b = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    torch.cuda.synchronize()
    ctx = _lib.Context()
    try:
        ctx.set_option(_lib.BEM_OPT_TCGEN05, variant)
        ctx.set_option(_lib.BEM_OPT_GRAPHS, 0)
        before = torch.cuda.mem_get_info()[0]
        solve_system(A, b, ctx=ctx)
        return before - torch.cuda.mem_get_info()[0]
    finally:
        ctx.close()


@pytest.mark.parametrize("n, variant, plans", [(3584, 2, 2), (8192, 1, 2), (8192, 2, 4)])
def test_operand_buffers(n, variant, plans):
    for v in (0, variant):
        taken(n, v)  # modules and kernels loaded, streams made
    got = taken(n, variant) - taken(n, 0)  # 0: no tensor-core operands
    # three buffers a plan of 512 n bytes and an eighth, in pieces of 2 MB
    each = -(-576 * n // 2**21) * 2**21
    assert got <= 3 * plans * each + 2**21, (got, each)
