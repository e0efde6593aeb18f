"""Schur formation over block lists of every length class: one pair, a partial
batch, a full one, one work item, the limits of an item and several items whose
partial sums are added by the last warp.  Three U blocks see n points; the
increment is compared with the dense solve of the whole system.

Tolerances: the systems are built with a condition number below 300.  FP64:
300 (n + 3 bu) eps < 1e-10.  Mixed: blocks rounded to FP32 (6e-8 relative), S
summed in FP32 in batches (a few eps): 300 x 1.2e-7 < 5e-5."""
import numpy as np
import pytest

from nelson_b200 import native as N

pytestmark = pytest.mark.gpu


def system(bu, n, seed):
    r = np.random.default_rng(seed)
    nu = 3
    w_rc = sorted({(u, p) for p in range(n) for u in ((0, 1) if p % 3 else (0, 1, 2))})
    W = r.normal(size=(len(w_rc), bu, 3)) / np.sqrt(3.0 * (n + 8))
    V = np.tile(np.eye(3), (n, 1, 1)) + 0.1 * np.einsum("pij,pkj->pik", *[r.normal(size=(n, 3, 3))] * 2)
    u_rc = [(i, j) for j in range(nu) for i in range(j + 1)]
    U = np.zeros((len(u_rc), bu, bu))
    for q, (i, j) in enumerate(u_rc):
        m = 0.1 * r.normal(size=(bu, bu))
        U[q] = 6.0 * np.eye(bu) + 0.5 * (m + m.T) if i == j else m
    H = np.zeros((nu * bu + 3 * n,) * 2)
    for q, (i, j) in enumerate(u_rc):
        H[bu * i:bu * i + bu, bu * j:bu * j + bu] = U[q]
        H[bu * j:bu * j + bu, bu * i:bu * i + bu] = U[q].T
    for p in range(n):
        s = slice(nu * bu + 3 * p, nu * bu + 3 * p + 3)
        H[s, s] = V[p]
    for q, (u, p) in enumerate(w_rc):
        s = slice(nu * bu + 3 * p, nu * bu + 3 * p + 3)
        H[bu * u:bu * u + bu, s] = W[q]
        H[s, bu * u:bu * u + bu] = W[q].T
    return np.array(u_rc, np.int32), np.array(w_rc, np.int32), U, V, W, H, r.normal(size=nu * bu + 3 * n)


@pytest.mark.parametrize("prec,tol", [(N.PREC_FP64, 1e-10), (N.PREC_MIXED, 5e-5)])
@pytest.mark.parametrize("bu", [2, 3, 6, 9])
@pytest.mark.parametrize("n", [1, 2, 11, 12, 13, 31, 33, 48, 49, 64, 65, 97, 500])
def test_increment(bu, n, prec, tol):
    u_rc, w_rc, U, V, W, H, b = system(bu, n, 100 * bu + n)
    assert np.linalg.eigvalsh(H)[0] > 0 and np.linalg.cond(H) < 300
    nub = 3 * bu
    v_rc = np.stack([np.arange(n)] * 2, 1).astype(np.int32)
    g = N.SchurSolverGPU(bu, 3, n, u_rc, v_rc, w_rc, precision=prec)
    g.set_hessian(U, V, W, b[:nub], b[nub:])
    x0 = None
    for mu in (0.0, 0.3, 0.0):  # the third call repeats the first on the same handle, bit for bit
        ok, du, dv = g.compute_increment(0.0, mu)
        x = np.linalg.solve(H + mu * np.eye(len(b)), -b)
        assert ok
        assert np.abs(np.r_[du, dv] - x).max() <= tol * np.abs(x).max()
        if mu == 0.0 and x0 is not None:
            assert np.array_equal(np.r_[du, dv], x0)
        if x0 is None:
            x0 = np.r_[du, dv]
    g.close()
