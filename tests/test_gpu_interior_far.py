"""The Gauss rule that interior points take for far elements: to rounding at
the edge of its bound, and not a condition of the call (it needs memory)."""
import numpy as np
import pytest

from bem_gmsh_gb300 import _lib, geometry, star_domain
from bem_gmsh_gb300.api import _ptr, geom_struct, interior_laplace

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def gauss_potential(dad, pts, T, q):
    """T(p) with 64 Gauss points on every element."""
    t, w = np.polynomial.legendre.leggauss(64)
    N, dN = geometry.lagrange_basis(geometry.equispaced_nodes(dad.ngeo - 1), t)
    F, _ = geometry.lagrange_basis(geometry.gauss_legendre(dad.p + 1)[0], t)
    x, d = np.einsum("qk,ekc->eqc", N, dad.geo), np.einsum("qk,ekc->eqc", dN, dad.geo)
    J = np.hypot(d[..., 0], d[..., 1])
    n = np.stack([d[..., 1], -d[..., 0]], axis=-1)
    n *= np.sign(np.sum(n[:, :1] * dad.normal[:dad.n:dad.p + 1][:, None], axis=-1))[..., None]
    Tq, qq = (v.reshape(dad.ne, -1) @ F.T for v in (T, q))
    out = []
    for p in pts:
        r = x - p
        R2 = np.sum(r * r, axis=-1)
        h = np.sum(r * n, axis=-1) / R2 / (2 * np.pi) * w
        g = -np.log(R2) / (4 * np.pi) * J * w
        out.append(np.sum(g * qq - h * Tq) / -np.sum(h))
    return np.array(out)


def distances(dad, pts, npg):
    """The smallest |p - x(0)| of each point in units of the bound's reach."""
    rho = 2.0 ** (60.0 / (2 * npg - dad.p))
    a = (rho + 1 / rho) / 2
    V = np.vander(geometry.equispaced_nodes(dad.ngeo - 1), increasing=True)
    c = np.einsum("dk,ekc->edc", np.linalg.inv(V), dad.geo)
    reach = np.linalg.norm(c[:, 1:], axis=-1) @ a ** np.arange(1, dad.ngeo)
    return np.min(np.linalg.norm(pts[:, None] - c[None, :, 0], axis=-1) / reach, axis=1)


@pytest.mark.parametrize("p, npg", [(1, 8), (2, 8), (5, 8), (2, 10), (3, 16), (2, 20), (5, 32)])
def test_far_rule_is_exact(p, npg):
    rho = 2.0 ** (60.0 / (2 * npg - p))
    dad = star_domain(int(4 * rho) + 8, p=p, seed=npg, amp=0.02)
    rng = np.random.default_rng(p)
    c = rng.uniform(-0.9, 0.9, (4000, 2))
    c = c[np.hypot(c[:, 0], c[:, 1]) < 0.8]  # inside
    d = distances(dad, c, npg)
    order = np.argsort(d)
    pts = c[order[d[order] > 1.0][:40]]  # the closest points that are far from every element
    assert len(pts) == 40 and distances(dad, pts, npg).min() < 1.1
    T, q = rng.standard_normal(dad.n), rng.standard_normal(dad.n)
    ref = gauss_potential(dad, pts, T, q)
    # rounding of the sums: some 10^4 terms of size one, 2^-53 sqrt(10^4)
    assert np.max(np.abs(interior_laplace(dad, pts, npg=npg, T=T, q=q) - ref)) <= 2e-14 * np.max(np.abs(T))


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
