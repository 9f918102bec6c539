"""Far terms whose value is known to the bit: no operand of a product is
rounded before it has to be."""
import numpy as np
import pytest

from bem_gmsh_gb300 import star_domain
from bem_gmsh_gb300.api import H_G_gpu, dibem_ifid

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


@pytest.mark.parametrize("rbf, divisor", [("PHS1", 3), ("PHS3", 5), ("PHS5", 7)])
def test_radial_integrals_are_divided(rbf, divisor):
    """phi_int(R) / R^2 (r . n) for R = 5 i / 64 and r . n = 4 i / 64: whole
    numbers over a power of two, divided once."""
    dad = points((4 / 64, 3 / 64))
    dad.normal[0] = (1.0, 0.0)
    IF, _ = dibem_ifid(dad, rbf=rbf)
    i = np.arange(2, 80)
    # R, R^3, R^5 times r . n: at most 31 bits, exact
    want = (5 * i / 64.0) ** {3: 1, 5: 3, 7: 5}[divisor] * (4 * i / 64.0)
    assert np.array_equal(IF[2:], want / divisor)
