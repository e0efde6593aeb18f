"""LM solves of dense systems of 48 and 49 tiles, up to which the launches are programmatic
dependents, against the same handle's envelope solver (dependents at every size): the
same factor but for the tiles that are zero, so the same costs to the FP64 and
mixed parity tolerances (1e-9, 1e-6), and the second solve equal to the first bit for bit."""
import numpy as np
import pytest

from nelson_b200 import native as N
from nelson_b200.problems import problem_from_pairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [(N.PREC_FP64, 1e-9), (N.PREC_MIXED, 1e-6)])
@pytest.mark.parametrize("cams", [1024, 1025])  # x 6 parameters
def test_lm(cams, prec, tol):
    pt = np.repeat(np.arange(6000), 3)
    p = problem_from_pairs(cams, 6000, pt % (cams - 2) + np.tile(np.arange(3), 6000), pt, bc=6, seed=9)
    g = N.BAProblemGPU.from_ba(p, precision=prec)
    out = []
    for kind in (N.SOLVER_DENSE, N.SOLVER_DENSE, N.SOLVER_ENVELOPE):
        g.set_solver_kind(kind)
        g.set_params(p.cams, p.pts)
        _, tr, its, _ = g.lm_solve(N.LMSettings(maxNumIt=2))
        assert its == 2
        out.append(np.array(tr)[:, 2])
    g.close()
    assert np.array_equal(out[0], out[1])
    assert out[0].shape == out[2].shape and np.abs(out[0] - out[2]).max() <= tol * out[0].max()
