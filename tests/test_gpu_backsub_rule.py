"""Back-substitution on both sides of its rule (a thread per point from 65,536 points on,
FP64 98,304, up to 256 MB of W blocks: the last size has 269 MB in FP64):
dV = V^-1 (-bV - W' dU) of the returned dU in numpy, on a caller-assembled system.

Tolerance per value: the FP32 path rounds V^-1 once (formed and applied in FP64), so
2^-24 of sum |V^-1| |t| with t = -bV - W' dU, doubled; FP64: the condition of V (below
20) and of the sums, 1e-13 of the same quantity with |W'| |dU| + |bV| in t's place."""
import numpy as np
import pytest

from nelson_b200 import native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [N.PREC_FP64, N.PREC_MIXED])
@pytest.mark.parametrize("bu,nv,k", [(2, 65537, 2), (3, 65535, 3), (6, 65536, 2), (9, 65535, 2), (9, 65536, 3), (3, 98303, 2), (9, 98304, 2),
                                     (9, 150000, 8)])
def test_points(bu, nv, k, prec):
    r = np.random.default_rng(bu * nv + k)
    nu = 12
    u, v = np.divmod(np.arange(nu * nv), nv)
    keep = (u - 5 * v) % nu < k  # k cameras per point
    u, v = u[keep], v[keep]
    q = lambda a: np.asarray(a, np.float32).astype(np.float64)  # exact in either precision
    W = q(0.05 * r.uniform(-1, 1, (u.size, bu, 3)))
    V = r.uniform(-1, 1, (nv, 3, 3))
    V = q(0.3 * (V + V.transpose(0, 2, 1)) + 4.0 * np.eye(3))
    bU, bV = q(r.normal(size=nu * bu)), q(r.normal(size=3 * nv))
    rc = np.stack([np.arange(nu)] * 2, 1).astype(np.int32)
    U = np.broadcast_to(q((100.0 + nv) * np.eye(bu)), (nu, bu, bu))
    g = N.SchurSolverGPU(bu, nu, nv, rc, np.stack([np.arange(nv)] * 2, 1).astype(np.int32),
                         np.stack([u, v], 1).astype(np.int32), precision=prec)
    g.set_hessian(U, V, W, bU, bV)
    ok, du, dv = g.compute_increment(0.0, 0.0)
    assert ok
    x = du.reshape(nu, bu)[u]
    wx, size = np.zeros((nv, 3)), np.abs(bV.reshape(nv, 3))
    np.add.at(wx, v, np.einsum("eij,ei->ej", W, x))
    np.add.at(size, v, np.einsum("eij,ei->ej", np.abs(W), np.abs(x)))
    Vi = np.linalg.inv(V)
    t = -bV.reshape(nv, 3) - wx
    want = np.einsum("pij,pj->pi", Vi, t)
    tol = 1e-13 * np.einsum("pij,pj->pi", np.abs(Vi), size)
    if prec == N.PREC_MIXED:
        tol += 2.0 ** -23 * np.einsum("pij,pj->pi", np.abs(Vi), np.abs(t))
    assert (np.abs(dv.reshape(nv, 3) - want) <= tol).all()
    V[nv - 1] *= -1.0  # a refused increment is zero
    g.set_hessian(U, V, W, bU, bV)
    ok, du, dv = g.compute_increment(0.0, 0.0)
    assert not ok and not du.any() and not dv.any()
    g.close()
