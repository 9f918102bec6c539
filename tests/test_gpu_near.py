"""Near and on-element integrals at the edges of their split over warps and
lanes, against the oracle: one pair a warp up to 16 (few and many elements),
1 to 32 rule nodes (a lane with none, or several), 2 to 6 field nodes."""
import numpy as np
import pytest

from bem_gmsh_gb300 import star_domain, Elasticity
from bem_gmsh_gb300.api import H_G_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kelvin", [False, True])
@pytest.mark.parametrize("ne, p, npg", [(5, 1, 20), (8, 2, 1), (9, 2, 7), (40, 3, 32), (33, 4, 9), (40, 5, 17),
                                        (300, 1, 8), (700, 2, 16)])
def test_near_and_own_entries(orc, ne, p, npg, kelvin):
    if kelvin and ne > 300:
        ne = 300
    props = Elasticity(1.0, 0.3) if kelvin else None
    dad = star_domain(ne, p=p, seed=ne, props=props, pontointerno=True)
    H, G = H_G_gpu(dad, T=np.float64, npg=npg, store=False)
    Hr, Gr = orc.assemble(dad, npg=npg, store=False)
    # the same rule nodes to the bit; up to 64 samples of about 20 rounded
    # operations each: 64 * 20 * 2^-53 of the largest entry, and a factor 7 for
    # the cancellation of the basis values
    assert np.max(np.abs(H - Hr)) <= 1e-12 * np.max(np.abs(Hr))
    assert np.max(np.abs(G - Gr)) <= 1e-12 * np.max(np.abs(Gr))


@pytest.mark.parametrize("p, nearfield", [(1, 0), (3, 0), (4, 0), (2, 2)])
def test_gradient_of_every_element_type(p, nearfield):
    """dJ/dx of the adjoint call against central differences of its own J, for
    the element types and the near-field map that take other kernels than the
    quadratic tanp3c case."""
    from bem_gmsh_gb300 import Laplace, _lib, from_nodes, star_adjoint_case
    from bem_gmsh_gb300.api import adjoint_laplace
    ctx = _lib.default_context()
    dad, target = star_adjoint_case(12, p=p, seed=4)
    qt = np.where(dad.BC == 0, 0.1 * target.collocation[:, 0], 0.0)
    X = np.asarray(dad.collocation).reshape(dad.ne, p + 1, 2)

    def J(Y):
        return adjoint_laplace(from_nodes("fd", Y, p, Laplace(1.0), dad.BC, dad.BV), qt, npg=16, ctx=ctx)[0]

    ctx.set_option(_lib.BEM_OPT_NEARFIELD, nearfield)
    try:
        g = adjoint_laplace(dad, qt, npg=16, ctx=ctx)[1].reshape(-1)
        h = 1e-6
        for c in list(np.argsort(-np.abs(g))[:3]) + [1, 2 * p + 2]:
            Y = X.copy().reshape(-1)
            Y[c] += h
            up = J(Y.reshape(X.shape))
            Y[c] -= 2 * h
            # J to 1e-12 of itself over 2 h, and the differences' own h^2 terms
            assert abs((up - J(Y.reshape(X.shape))) / (2 * h) - g[c]) <= 1e-5 * np.max(np.abs(g))
    finally:
        ctx.set_option(_lib.BEM_OPT_NEARFIELD, 0)


@pytest.mark.parametrize("ne, p, npg", [(24, 3, 8), (30, 2, 5), (60, 2, 8), (90, 1, 10), (300, 2, 16), (40, 2, 32)])
def test_interior_far_rule(orc, ne, p, npg):
    """Interior points from the middle to a thousandth of the radius from the
    boundary, and on it: far pairs by the Gauss rule, the others by the map;
    more elements than a round of the kernel takes, and fewer than a warp."""
    from bem_gmsh_gb300.api import interior_laplace
    dad = star_domain(ne, p=p, seed=ne)
    ana = dad.cache["analytical"]
    T, q = ana.u(dad.Nodes), ana.q(dad.Nodes, dad.normal)
    pts = np.concatenate([[[0.0, 0.0]], 0.5 * dad.Nodes[::5], 0.9 * dad.Nodes[::7], 0.999 * dad.Nodes[::11],
                          dad.Nodes[::29]])
    got = interior_laplace(dad, pts, npg=npg, T=T, q=q)
    ref = orc.interior_laplace(dad, pts, npg=npg, T=T, q=q)
    # both rules within 3e-11 of a far integral (8 points and more; fewer
    # points take the map everywhere)
    assert np.max(np.abs(got - ref)) <= 1e-10 * np.max(np.abs(ref))
