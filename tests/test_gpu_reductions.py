"""Reductions whose last CTA adds the partial sums, over counts around the CTA
and grid limits (256 edges per CTA, 592 CTAs), and refinement sweeps beyond those
that have solve flags of their own.

Tolerances: the cost is FP64 on both sides, ne terms of one sign, each with a
relative error of some 100 eps: 1e-12.  Maxima of values that are read back:
equal to the last bit."""
import numpy as np
import pytest

from nelson_b200 import native as N
from nelson_b200.problems import make_config, problem_from_pairs, project

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ne", [1, 255, 256, 257, 592 * 256, 592 * 256 + 1])
def test_cost_and_maxima(ne):
    nc = 1 if ne < 3 else 3
    p = problem_from_pairs(nc, ne, np.arange(ne) % nc, np.arange(ne), bc=9, seed=ne)
    assert p.ne == ne
    g = N.BAProblemGPU.from_ba(p, precision=N.PREC_FP64)
    r = project(p.cams, p.pts, p.cam_idx, p.pt_idx, 9) - p.obs
    for _ in range(2):  # the counters are back at zero after a call
        assert g.update(True) == pytest.approx(float((r * r).sum()), rel=1e-12)
        U, V, W, bU, bV = g.hessian()
        assert g.max_abs_b() == max(np.abs(bU).max(), np.abs(bV).max())
        i = np.arange(3)
        diag = max(np.abs(V.reshape(-1, 3, 3)[:, i, i]).max(), np.abs(U.reshape(-1, 9, 9)[:, range(9), range(9)]).max())
        assert g.max_abs_hdiag() == diag
    g.close()


@pytest.mark.parametrize("sweeps", [0, 1, 3, 4, 6])
def test_refinement_sweeps(sweeps):
    """Mixed mode against the same system solved in FP64 from its own blocks:
    a sweep gains a factor of at least 100 at this damping until the residual
    (FP64 sums over the FP32 matrix) is at its end, cond x eps < 1e-10."""
    p = make_config(1, 0.1)
    g = N.BAProblemGPU.from_ba(p, precision=N.PREC_MIXED, refine_sweeps=sweeps)
    g.update(True)
    mu = 1e-3 * g.max_abs_hdiag()
    xs = []
    for _ in range(2):
        assert g.compute_increment(0.0, mu)
        S, b = g.schur()
        x = np.concatenate([np.asarray(a, np.float64).ravel() for a in g.increment()])
        xs.append(x)
    n = len(b)
    S = np.asarray(S, np.float64).reshape(n, n)
    S = np.triu(S) + np.triu(S, 1).T  # the upper triangle is given
    ref = np.linalg.solve(S, b)
    err = min(np.abs(xs[0][:n] - ref).max(), np.abs(xs[0][:n] + ref).max()) / np.abs(ref).max()
    assert err <= max(1e-3 * 1e-2 ** sweeps, 1e-10)
    assert np.array_equal(xs[0], xs[1])
    g.close()
