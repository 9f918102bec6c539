"""Far terms whose value is known to the bit: no operand of a product is
rounded before it has to be."""
import numpy as np
import pytest

from bem_gmsh_gb300 import star_domain
from bem_gmsh_gb300.api import H_G_gpu

pytestmark = pytest.mark.gpu


def points(r, n=80):
    """Linear elements of no length; node 0 at the origin with weight one, node
    i at -i r, node 1 away."""
    dad = star_domain(n // 2, p=1, seed=0)
    i = np.arange(n)[:, None]
    dad.collocation = -i * np.asarray(r)[None]
    dad.collocation[1] = (-50.0, 20.0)
    dad.elem_length = np.full(dad.ne, 1e-3)
    dad.elem_weight = np.ones(2)
    dad.jacobian = np.ones(n)
    dad.normal = np.zeros((n, 2))
    return dad


def test_orthogonal_normal_gives_zero():
    """r . n = 0 in exact products: H is zero, and so it is when the entry has
    a weight with all its bits."""
    dad = points((0.5, -0.75))
    dad.normal[0] = (0.75, 0.5)
    dad.jacobian[0] = 1.0 / 3.0
    H, G = H_G_gpu(dad, T=np.float64, npg=8, store=False)
    assert np.all(H[2:, 0] == 0.0) and np.all(G[2:, 0] != 0.0)
