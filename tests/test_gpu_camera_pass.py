"""Camera and point passes where the work of a camera is split over several CTAs
(2, 3 and 8 per camera) and not, with remainders of a warp, against the FP64 oracle's
Hessian.  Tolerances: those of the Hessian parity test (FP64 1e-11; mixed 1e-5,
relative to the largest entry), sums of up to 5,000 terms."""
import numpy as np
import pytest

from nelson_b200 import native as N
from nelson_b200.problems import problem_from_pairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [(N.PREC_FP64, 1e-11), (N.PREC_MIXED, 1e-5)])
@pytest.mark.parametrize("bc", [6, 9])
@pytest.mark.parametrize("nc,per", [(1, 31), (1, 511), (1, 512), (1, 767), (2, 2049), (3, 5000), (250, 900), (600, 33)])
def test_hessian(oracle_lib, nc, per, bc, prec, tol):
    n = per * max(1, nc // 2)
    cam = np.concatenate([(np.arange(n) + k) % nc for k in range(min(nc, 2))])
    pt = np.concatenate([np.arange(n)] * min(nc, 2))
    p = problem_from_pairs(nc, n, cam, pt, bc=bc, seed=nc + per)
    o = oracle_lib.Oracle.from_ba(p)
    o.update(True)
    g = N.BAProblemGPU.from_ba(p, precision=prec)
    for _ in range(2):  # the counters are back at zero after a pass
        g.update(True)
        for a, b in zip(g.hessian(), o.hessian()):
            assert np.abs(a - b).max() <= tol * np.abs(b).max()
    g.close()
