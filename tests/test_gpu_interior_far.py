"""The Gauss rule that interior points take for far elements is not a condition
of the call (it needs memory)."""
import numpy as np
import pytest

from bem_gmsh_gb300 import _lib, star_domain
from bem_gmsh_gb300.api import _ptr, geom_struct

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_no_memory_for_the_far_rule(orc):
    """Device arrays need no workspace but the far rule's: without it every
    pair takes the map, as before there was a far rule."""
    dad = star_domain(100, p=2, seed=1)
    rng = np.random.default_rng(0)
    T, q = rng.standard_normal(dad.n), rng.standard_normal(dad.n)
    pts = 0.9 * dad.Nodes[::7] * rng.uniform(0.1, 1.0, (len(dad.Nodes[::7]), 1))
    ctx = _lib.Context()
    try:
        g, keep = geom_struct(dad, device=True)
        dev = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (T, q, pts[:, 0], pts[:, 1])]
        ctx.set_option(_lib.BEM_OPT_INJECT, 1)  # no workspace at all
        out = torch.zeros(len(pts), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        rc = ctx.L.bem_interior_laplace2d(ctx.h, g, 1.0, 16, *map(_ptr, dev[:2]), len(pts), *map(_ptr, dev[2:]),
                                          _lib.BEM_MEM_DEVICE, _ptr(out))
        assert rc == _lib.BEM_OK, rc
        # the oracle's map to the bit, its sums in another order (as in test_gpu_interior.py)
        ref = orc.interior_laplace(dad, pts, npg=16, T=T, q=q)
        assert np.max(np.abs(out.cpu().numpy() - ref)) <= 1e-11 * np.max(np.abs(ref))
    finally:
        ctx.close()
