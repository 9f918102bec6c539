"""Near-pair lists that the first assembly of a context finds too short (16
pairs a point): found at once where the near factor makes it likely, with the
solve's or the gradient's first results elsewhere."""
import numpy as np
import pytest

from bem_gmsh_gb300 import Laplace, _lib, from_nodes, geometry, star_adjoint_case, star_domain
from bem_gmsh_gb300.api import adjoint_laplace, solve

pytestmark = pytest.mark.gpu


def rings(count=6, ne=80, gap=0.01, p=1):
    """Concentric polygons much closer to each other than their elements are
    long: every point has some four elements of each within 1.5 lengths."""
    t = np.arange(ne + 1) * 2 * np.pi / ne
    xi = geometry.gauss_legendre(p + 1)[0]
    X = []
    for c in range(count):
        v = (1.0 + c * gap) * np.stack([np.cos(t), np.sin(t)], axis=1)
        a, b = v[:-1, None], v[1:, None]
        X.append(a * (1 - xi[None, :, None]) / 2 + b * (1 + xi[None, :, None]) / 2)
    X = np.concatenate(X)
    th = np.arctan2(X[..., 1], X[..., 0]).reshape(-1)
    bc = (th < 0).astype(np.int32)
    return from_nodes("rings", X, p, Laplace(1.0), bc, np.where(bc == 0, np.cos(th), np.sin(3 * th)))


def counted(ctx, f):
    n = ctx.launch_count()
    r = f()
    return r, ctx.launch_count() - n


def test_overflow_costs_one_assembly_and_no_factorization():
    dad = star_domain(333, p=2, seed=3)
    ctx = _lib.Context()
    try:
        (_, first), (_, second) = [counted(ctx, lambda: solve(dad, npg=8, near_factor=np.inf, ctx=ctx).copy())
                                   for _ in range(2)]
        assert first - second <= 6  # the assembly's launches; its LU has 26
        x1 = dad.cache["x"].copy()
        solve(dad, npg=8, near_factor=np.inf, mode="fp64", ctx=ctx)
        # two residuals of 1e-14 at a condition number below 1e4
        assert np.linalg.norm(x1 - dad.cache["x"]) <= 2e-10 * np.linalg.norm(x1)
    finally:
        ctx.close()


def test_overflow_found_by_the_solve():
    dad = rings()
    ctx = _lib.Context()
    try:
        (_, first), (_, second) = [counted(ctx, lambda: solve(dad, npg=8, ctx=ctx).copy()) for _ in range(2)]
        x1 = dad.cache["x"].copy()
        other = rings()
        fresh = _lib.Context()
        try:
            solve(other, npg=8, mode="fp64", ctx=fresh)  # waits for the pair count at once
        finally:
            fresh.close()
        assert first > second + 6, (first, second)  # the list was too short: an LU and a sweep more
        r = other.cache["x"]
        # two residuals of 1e-14 at a condition number of 2100
        assert np.linalg.norm(x1 - r) <= 1e-10 * np.linalg.norm(r)
    finally:
        ctx.close()


@pytest.mark.parametrize("mesh, near_factor", [("rings", 1.5), ("star", 12.0)])
def test_gradient_overflow(mesh, near_factor):
    """Some 25 elements near each point, more than the assembly's list holds
    and fewer than the gradient's own (32)."""
    dad = rings() if mesh == "rings" else star_adjoint_case(300, p=1, seed=2)[0]
    qt = np.where(dad.BC == 0, 0.1 * dad.collocation[:, 0], 0.0)
    fresh, used = _lib.Context(), _lib.Context()
    try:
        solve(star_domain(333, p=2, seed=3), npg=8, near_factor=np.inf, ctx=used)  # leaves a long list
        J0, g0 = adjoint_laplace(dad, qt, npg=12, near_factor=near_factor, ctx=used)
        J1, g1 = adjoint_laplace(dad, qt, npg=12, near_factor=near_factor, ctx=fresh)
        # the differences' rounding, 2^-53 over their step of 1e-5, and sums in another order
        assert abs(J1 - J0) <= 1e-10 * abs(J0)
        assert np.max(np.abs(g1 - g0)) <= 1e-9 * np.max(np.abs(g0))
    finally:
        fresh.close()
        used.close()
