"""The dense solver at the sizes where its kernels change their split: 32-row
and 128-row blocks, the column scaling's rounds (512 rows), the refinement's
cluster width (4096) and the factorization's schedules (panels of 32 or 64
vectors, steps in pairs, diagonal blocks launched early)."""
import numpy as np
import pytest

from bem_gmsh_gb300 import _lib, star_domain
from bem_gmsh_gb300.api import solve, solve_batch, solve_system

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 65, 127, 128, 129, 256, 257, 511, 512, 513, 1024, 1025, 1536, 1537,
                               2560, 2561, 4095, 4096, 4097, 4608, 4609, 6657, 8704, 8705])
def test_solve_system_sizes(n):
    g = torch.Generator(device="cuda").manual_seed(n)
    At = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g) / n**0.5
    At.diagonal().add_(2.0)
    At *= torch.logspace(-1, 1, n, dtype=torch.float64, device="cuda")[:, None]  # uneven column scales
    A = At.t()  # column-major
    b = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    torch.cuda.synchronize()
    x, st = solve_system(A, b)
    torch.cuda.synchronize()
    # the solver's own target plus the rounding of the product formed here
    r = float((A @ x - b).norm() / b.norm())
    assert r <= 1e-14 + 4 * 2.0**-53 * n**0.5, (r, st)
    assert not st["pivoted"] and st["iterations"] <= 8, st


@pytest.mark.parametrize("variant", [1, 2])
@pytest.mark.parametrize("n", [256, 384, 2432, 2560, 2688, 3072, 3200, 3328, 3584, 3712, 3840, 3968, 4096])
def test_lu_schedules(n, variant):
    """Against the plain schedule on mma.sync, to FP32 rounding."""
    ctx = _lib.Context()
    try:
        ctx.set_option(_lib.BEM_OPT_TCGEN05, variant)
        r = ctx.selftest_lu(n)
        assert r[0] / r[1] < 1e-5, r
    finally:
        ctx.close()


def test_many_small_domains_at_once():
    """Sixteen pipelines of clusters, cooperative sweeps and dependent launches
    on one GPU give what each domain gives alone."""
    dads = [star_domain(20 + 5 * (i % 24), p=1 + i % 2, seed=i) for i in range(64)]
    alone = []
    for d in dads:
        solve(d, npg=16)
        alone.append(d.cache["x"].copy())
    for _ in range(3):
        for x, ref in zip(solve_batch(dads, npg=16, nworkers=16), alone):
            # two residuals of 1e-14 at a condition number below 1e4
            assert np.linalg.norm(x - ref) <= 2e-10 * np.linalg.norm(ref)
