"""LM solves at and just above the size up to which the launches are programmatic
dependents (65,536 W blocks), against the FP64 oracle's trace (the parity test's
tolerances: cost 1e-9 FP64, 1e-6 mixed), the second solve on the handle equal to the
first bit for bit."""
import numpy as np
import pytest

from nelson_b200 import native as N
from nelson_b200.problems import problem_from_pairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [(N.PREC_FP64, 1e-9), (N.PREC_MIXED, 1e-6)])
@pytest.mark.parametrize("npts", [8192, 8193])
def test_lm(oracle_lib, npts, prec, tol):
    cam, pt = np.tile(np.arange(8), npts), np.repeat(np.arange(npts), 8)
    p = problem_from_pairs(8, npts, cam, pt, bc=6, seed=3)
    o = oracle_lib.Oracle.from_ba(p)
    _, tr_o, _, _ = o.lm_solve(oracle_lib.LMSettings(maxNumIt=2))
    g = N.BAProblemGPU.from_ba(p, precision=prec)
    traces = []
    for _ in range(2):
        g.set_params(p.cams, p.pts)
        _, tr, _, _ = g.lm_solve(N.LMSettings(maxNumIt=2))
        traces.append(np.array(tr))
    assert np.array_equal(traces[0], traces[1])
    a, b = traces[0][:, 2], np.array(tr_o)[:, 2]
    assert a.shape == b.shape and np.abs(a - b).max() <= tol * np.abs(b).max()
    g.close()
