"""The tiled Cholesky at the edges of its 128-row tiles and 16-column blocks:
a caller-assembled symmetric system (no V blocks) against numpy, for sizes that
leave one block, a nearly empty and a nearly full last tile, one group of four
panels and more than one.

Tolerances: the matrices have a condition number below 100 (random symmetric
blocks plus a diagonal that dominates every row).  FP64: 100 n eps < 1e-10 at n
= 1,300.  Mixed: the entries are rounded to FP32 once (2^-24 relative, times the
condition number: 6e-6) and the refinement solves that system, so 2e-5."""
import numpy as np
import pytest

from nelson_b200 import native as N

pytestmark = pytest.mark.gpu


def system(bu, nu, seed):
    r = np.random.default_rng(seed)
    n = bu * nu
    A = r.normal(size=(n, n))
    A = 0.5 * (A + A.T) / np.sqrt(n)
    A[np.arange(n), np.arange(n)] = 3.0 + r.uniform(0.0, 4.0, n)  # |off-diagonal part|_2 < 1.6
    rc = np.array([(i, j) for j in range(nu) for i in range(j + 1)], np.int32)
    U = np.stack([A[bu * i:bu * i + bu, bu * j:bu * j + bu] for i, j in rc])
    return A, rc, U, r.normal(size=n)


@pytest.mark.parametrize("prec,tol", [(N.PREC_FP64, 1e-10), (N.PREC_MIXED, 2e-5)])
@pytest.mark.parametrize("kind", [N.SOLVER_DENSE, N.SOLVER_ENVELOPE])
@pytest.mark.parametrize("bu,nu", [(2, 1), (3, 5), (3, 43), (9, 14), (9, 15), (2, 64), (6, 43), (9, 57), (6, 107),
                                   (9, 143)])
def test_factor_and_solve(bu, nu, kind, prec, tol):
    A, rc, U, b = system(bu, nu, 10 * bu + nu)
    assert np.linalg.cond(A) < 100
    g = N.SchurSolverGPU(bu, nu, 0, rc, np.zeros((0, 2), np.int32), np.zeros((0, 2), np.int32), precision=prec)
    g.set_solver_kind(kind)
    g.set_hessian(U, np.zeros((0, 3, 3)), np.zeros((0, bu, 3)), b, np.zeros(0))
    for rel, ab in ((0.0, 0.0), (0.25, 0.5)):  # the second solve overwrites the first one's factor and inverses
        ok, du, _ = g.compute_increment(rel, ab)
        x = np.linalg.solve(A + np.diag(rel * np.diag(A) + ab), -b)
        assert ok
        assert np.abs(du - x).max() <= tol * np.abs(x).max()
    g.close()


@pytest.mark.parametrize("prec", [N.PREC_FP64, N.PREC_MIXED])
@pytest.mark.parametrize("row", [0, 15, 16, 127, 128, 130])
def test_negative_pivot_is_reported(row, prec):
    """A diagonal entry made negative: the increment is refused, and the handle
    solves the next (definite) system as if nothing had happened."""
    A, rc, U, b = system(3, 47, 5)
    bad = U.copy()
    q = int(np.flatnonzero((rc[:, 0] == row // 3) & (rc[:, 1] == row // 3))[0])
    bad[q, row % 3, row % 3] = -5.0
    g = N.SchurSolverGPU(3, 47, 0, rc, np.zeros((0, 2), np.int32), np.zeros((0, 2), np.int32), precision=prec)
    z = np.zeros((0, 3, 3))
    g.set_hessian(bad, z, z, b, np.zeros(0))
    ok, du, _ = g.compute_increment(0.0, 0.0)
    assert not ok and not du.any()
    g.set_hessian(U, z, z, b, np.zeros(0))
    ok, du, _ = g.compute_increment(0.0, 0.0)
    x = np.linalg.solve(A, -b)
    assert ok and np.abs(du - x).max() <= (1e-10 if prec == N.PREC_FP64 else 2e-5) * np.abs(x).max()
    g.close()
