"""The triangular solves over 1 .. 5 tiles (below, at and above the depth of the hop
matrices) and with more CTAs than fit on the chip at once (FP64 78 tiles, mixed 152
tiles), dense and envelope order, with a coupling that reaches from the first block
to the last.

Tolerances: H is block-diagonally dominant (off-diagonal row sums below half of the
smallest eigenvalue of the diagonal blocks): condition number below 60, the residual
of a solve below cond x (a few eps) x row length: FP64 1e-11, mixed (FP32 blocks and
factor, one refinement sweep against the FP32 matrix) 2e-5."""
import numpy as np
import pytest
import scipy.sparse as sp

from nelson_b200 import native as N

pytestmark = pytest.mark.gpu


def system(bu, nu, seed):
    r = np.random.default_rng(seed)
    pairs = {(i, i) for i in range(nu)} | {(i - 1, i) for i in range(1, nu)} | {(0, nu - 1)}
    u_rc = sorted(pairs, key=lambda t: (t[1], t[0]))
    U = np.zeros((len(u_rc), bu, bu))
    for q, (i, j) in enumerate(u_rc):
        m = r.uniform(-1, 1, (bu, bu))
        U[q] = 8.0 * np.eye(bu) + 0.5 * (m + m.T) / bu if i == j else m / bu
    V = np.tile(8.0 * np.eye(3), (nu, 1, 1))
    w_rc = sorted({(p, p) for p in range(nu)} | {((p + 1) % nu, p) for p in range(nu)})
    W = r.uniform(-1, 1, (len(w_rc), bu, 3)) / 9.0
    rows, cols, vals = [], [], []

    def put(r0, c0, m):
        i, j = np.meshgrid(np.arange(m.shape[0]), np.arange(m.shape[1]), indexing="ij")
        rows.append((r0 + i).ravel()), cols.append((c0 + j).ravel()), vals.append(m.ravel())

    for q, (i, j) in enumerate(u_rc):
        put(bu * i, bu * j, U[q])
        if i != j:
            put(bu * j, bu * i, U[q].T)
    for p in range(nu):
        put(bu * nu + 3 * p, bu * nu + 3 * p, V[p])
    for q, (u, p) in enumerate(w_rc):
        put(bu * u, bu * nu + 3 * p, W[q])
        put(bu * nu + 3 * p, bu * u, W[q].T)
    n = (bu + 3) * nu
    H = sp.csr_matrix((np.concatenate(vals), (np.concatenate(rows), np.concatenate(cols))), (n, n))
    v_rc = np.stack([np.arange(nu)] * 2, 1).astype(np.int32)
    return np.array(u_rc, np.int32), v_rc, np.array(w_rc, np.int32), U, V, W, H, r.normal(size=n)


SMALL = [(2, 2), (2, 64), (2, 65), (2, 128), (2, 129), (3, 128), (3, 129), (2, 256), (2, 257), (6, 107)]


@pytest.mark.parametrize("kind", [N.SOLVER_DENSE, N.SOLVER_ENVELOPE])
@pytest.mark.parametrize("prec,bu,nu", [(p, *s) for p in (N.PREC_FP64, N.PREC_MIXED) for s in SMALL] +
                         [(N.PREC_FP64, 9, 1100), (N.PREC_MIXED, 9, 2150)])
def test_residual(prec, bu, nu, kind):
    u_rc, v_rc, w_rc, U, V, W, H, b = system(bu, nu, nu)
    g = N.SchurSolverGPU(bu, nu, nu, u_rc, v_rc, w_rc, precision=prec)
    g.set_solver_kind(kind)
    g.set_hessian(U, V, W, b[:bu * nu], b[bu * nu:])
    tol = 1e-11 if prec == N.PREC_FP64 else 2e-5
    for mu in (0.0, 0.5):
        ok, du, dv = g.compute_increment(0.0, mu)
        x = np.r_[du, dv]
        assert ok
        assert np.abs(H @ x + mu * x + b).max() <= tol * np.abs(b).max()
    g.close()


@pytest.mark.parametrize("prec", [N.PREC_FP64, N.PREC_MIXED])
@pytest.mark.parametrize("links", [(), ((63, 64),), ((0, 191),), ((63, 64), (64, 191), (130, 255))])
def test_separate_tiles(prec, links):
    """Envelope order where tile rows have no neighbour below, the next one only, or
    one further down: four tiles of 64 independent 2 x 2 blocks and a few couplings.
    The Schur complement is known exactly: same tolerances."""
    bu, nu = 2, 256
    r = np.random.default_rng(len(links))
    u_rc = sorted([(i, i) for i in range(nu)] + list(links), key=lambda t: (t[1], t[0]))
    U = np.array([8.0 * np.eye(2) if i == j else r.uniform(-1, 1, (2, 2)) for i, j in u_rc])
    v_rc = w_rc = np.stack([np.arange(nu)] * 2, 1).astype(np.int32)
    V, W = np.tile(8.0 * np.eye(3), (nu, 1, 1)), r.uniform(-1, 1, (nu, 2, 3))
    H = np.zeros((5 * nu, 5 * nu))
    for q, (i, j) in enumerate(u_rc):
        H[2 * i:2 * i + 2, 2 * j:2 * j + 2] = U[q]
        H[2 * j:2 * j + 2, 2 * i:2 * i + 2] = U[q].T
    for p in range(nu):
        s = slice(2 * nu + 3 * p, 2 * nu + 3 * p + 3)
        H[s, s] = V[p]
        H[2 * p:2 * p + 2, s] = W[p]
        H[s, 2 * p:2 * p + 2] = W[p].T
    b = r.normal(size=5 * nu)
    g = N.SchurSolverGPU(bu, nu, nu, np.array(u_rc, np.int32), v_rc, w_rc, precision=prec)
    g.set_solver_kind(N.SOLVER_ENVELOPE)
    g.set_hessian(U, V, W, b[:2 * nu], b[2 * nu:])
    for _ in range(2):
        ok, du, dv = g.compute_increment(0.0, 0.0)
        assert ok
        assert np.abs(H @ np.r_[du, dv] + b).max() <= (1e-11 if prec == N.PREC_FP64 else 2e-5) * np.abs(b).max()
    g.close()
