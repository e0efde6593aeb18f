"""A handle whose factorisation failed solves the next system as a fresh one does,
where the reduced system has tiles outside the Cholesky envelope: the failed factor
overflows, and zero times infinity reaches those tiles as well.

Systems of 3 x 3 blocks in five 128-row tiles: a band (tiles two below the diagonal
are outside), and the band with one long row in the middle (the tiles between its
first column and the band are outside, but inside the rows that the panels' solves
cover).  Tolerances as in test_gpu_factor_tiles: condition number below 100, FP64
100 n eps, mixed the FP32 rounding of the entries times the condition number."""
import numpy as np
import pytest

from nelson_b200 import native as N

pytestmark = pytest.mark.gpu
BU, NU = 3, 200


def system(long_row, seed):
    r = np.random.default_rng(seed)
    n = BU * NU
    rc = [(i, j) for j in range(NU) for i in range(max(0, j - 2), j + 1)]
    if long_row:
        rc = sorted(set(rc) | {(i, 90) for i in range(90)}, key=lambda t: (t[1], t[0]))
    A = np.zeros((n, n))
    for i, j in rc:
        B = 0.1 * r.uniform(-1.0, 1.0, (BU, BU)) * (0.3 if j - i > 2 else 1.0)
        A[BU * i:BU * i + BU, BU * j:BU * j + BU] = B
    A = np.triu(A, 1)
    A = A + A.T
    A[np.arange(n), np.arange(n)] = 4.0 + r.uniform(0.0, 4.0, n)
    rc = np.array(rc, np.int32)
    U = np.stack([A[BU * i:BU * i + BU, BU * j:BU * j + BU] for i, j in rc])
    return A, rc, U, r.normal(size=n)


@pytest.mark.parametrize("prec,tol", [(N.PREC_FP64, 1e-10), (N.PREC_MIXED, 2e-5)])
@pytest.mark.parametrize("kind", [N.SOLVER_DENSE, N.SOLVER_ENVELOPE])
@pytest.mark.parametrize("long_row", [False, True])
@pytest.mark.parametrize("row", [1, 126])
def test_next_system_solves(row, long_row, kind, prec, tol):
    A, rc, U, b = system(long_row, 7)
    assert np.linalg.cond(A) < 100
    bad = U.copy()
    bad[int(np.flatnonzero((rc[:, 0] == row // 3) & (rc[:, 1] == row // 3))[0]), row % 3, row % 3] = -5.0
    none = np.zeros((0, 2), np.int32)
    g = N.SchurSolverGPU(BU, NU, 0, rc, none, none, precision=prec)
    g.set_solver_kind(kind)
    z = np.zeros((0, 3, 3))
    x = np.linalg.solve(A, -b)
    for blocks, want in ((U, True), (bad, False), (U, True), (U, True)):
        g.set_hessian(blocks, z, z, b, np.zeros(0))
        ok, du, _ = g.compute_increment(0.0, 0.0)
        assert ok == want
        assert np.abs(du - (x if want else 0.0)).max() <= tol * np.abs(x).max()
    # the damping makes the indefinite system definite: the retry of an LM loop
    g.set_hessian(bad, z, z, b, np.zeros(0))
    assert not g.compute_increment(0.0, 0.0)[0]
    ok, du, _ = g.compute_increment(0.0, 20.0)
    B = A.copy()
    B[row, row] = -5.0
    y = np.linalg.solve(B + 20.0 * np.eye(len(B)), -b)
    assert ok and np.abs(du - y).max() <= tol * np.abs(y).max()
    g.close()
