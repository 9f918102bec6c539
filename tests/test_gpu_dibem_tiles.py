"""Pairwise DIBEM matrices at the edges of their tiles (32 and 64 points):
counts around a tile and its multiples, odd leading dimensions, guarded
columns around the results."""
import numpy as np
import pytest

from bem_gmsh_gb300 import _lib

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("f64", [True, False])
@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("nt", [1, 2, 31, 32, 33, 63, 64, 65, 97, 193])
def test_tiles_match_oracle(orc, nt, kind, f64):
    rng = np.random.default_rng(nt)
    # distinct multiples of 1/64: coordinate differences are exact in FP32
    cells = rng.choice(128 * 128, nt, replace=False)
    pts = np.stack([cells // 128, cells % 128], axis=1) / 64.0
    p0, p1 = (2.0, 0.0) if kind == 0 else (1.5, 0.3)
    dof, ldf, ldd = kind + 1, nt + 3, (kind + 1) * nt + 1
    dt = torch.float64 if f64 else torch.float32
    F = torch.full((nt, ldf), 7.0, dtype=dt, device="cuda")
    D = torch.full((dof * nt, ldd), 7.0, dtype=dt, device="cuda")
    xy = torch.tensor(pts.T.copy(), device="cuda")
    ctx = _lib.default_context()
    torch.cuda.synchronize()
    rc = ctx.L.bem_dibem_fd2d(ctx.h, nt, xy[0].data_ptr(), xy[1].data_ptr(), kind, p0, p1, 2, 1e-16,
                              _lib.BEM_F64 if f64 else _lib.BEM_F32, _lib.BEM_MEM_DEVICE, F.data_ptr(), ldf,
                              D.data_ptr(), ldd)
    ctx.check(rc, "dibem_fd")
    F, D = F.cpu().numpy(), D.cpu().numpy()
    # nothing beyond the rows of a column is written
    assert (F[:, nt:] == 7.0).all() and (D[:, dof * nt:] == 7.0).all()
    F, D = F[:, :nt].T, D[:, : dof * nt].T
    assert (F == F.T).all() and (D == D.T).all()
    Fr, Dr = orc.dibem_fd(pts, kind=kind, prm0=p0, prm1=p1, rbf=2)
    # R^2, sqrt, log and three products, 0.5 to 1 ulp each, on values whose
    # logarithm passes zero: 16 units of the last place of the largest entry
    eps = 2.0 ** (-52 if f64 else -23)
    assert np.abs(F - Fr).max() <= 16 * eps * max(np.abs(Fr).max(), 1e-300)
    assert np.abs(D - Dr).max() <= 16 * eps * max(np.abs(Dr).max(), 1e-300)
