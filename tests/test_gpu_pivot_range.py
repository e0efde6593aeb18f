"""FP32 pivots near both ends of the range: D^1/2 R D^1/2 with a well-conditioned R and
diagonals of 1e38 (reciprocals below the smallest normal FP32 number), of 1e-29 and
of both in turn.  A Cholesky factorisation does not see the scaling, so the scaled
solution has the tolerance of the unscaled system (test_gpu_factor_tiles): FP32
rounding of the entries, 2^-24, times a condition number below 100, twice over."""
import numpy as np
import pytest

from nelson_b200 import native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", ["large", "small", "mixed"])
@pytest.mark.parametrize("bu,nu", [(3, 5), (6, 43)])
def test_scaled_system(bu, nu, scale):
    r = np.random.default_rng(11 * bu + nu)
    n = bu * nu
    R = r.normal(size=(n, n))
    R = 0.1 * (R + R.T) / np.sqrt(n)
    R[np.arange(n), np.arange(n)] = 1.0 + r.uniform(0.0, 1.0, n)
    assert np.linalg.cond(R) < 100 and np.linalg.eigvalsh(R)[0] > 0.4
    d = {"large": np.full(n, 1.5e38), "small": np.full(n, 1e-29),
         "mixed": np.where(np.arange(n) % 2, 1.5e38, 1e-29)}[scale] ** 0.5
    A = d[:, None] * R * d
    assert np.abs(A).max() < 3.4e38
    y = r.normal(size=n)
    b = d * y
    rc = np.array([(i, j) for j in range(nu) for i in range(j + 1)], np.int32)
    U = np.stack([A[bu * i:bu * i + bu, bu * j:bu * j + bu] for i, j in rc])
    none = np.zeros((0, 2), np.int32)
    g = N.SchurSolverGPU(bu, nu, 0, rc, none, none, precision=N.PREC_MIXED)
    g.set_hessian(U, np.zeros((0, 3, 3)), np.zeros((0, bu, 3)), b, np.zeros(0))
    ok, du, _ = g.compute_increment(0.0, 0.0)
    x = np.linalg.solve(R, -y)
    assert ok and np.abs(d * du - x).max() <= 2e-5 * np.abs(x).max()
    g.close()
