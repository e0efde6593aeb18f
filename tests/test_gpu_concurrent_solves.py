"""Handles of eleven tiles (143 cameras x 9) whose triangular solves share the chip: eight
at once through nl_lm_solve_batch give what each gives alone, bit for bit (the waits
between the CTAs of a solve never depend on another handle's)."""
import numpy as np
import pytest

from nelson_b200 import native as N
from nelson_b200.problems import ring_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [N.PREC_FP64, N.PREC_MIXED])
def test_eight_handles(prec):
    ps = [ring_scene(143, 1200, 3, 8, 9, 40 + i) for i in range(8)]
    gs = [N.BAProblemGPU.from_ba(p, precision=prec) for p in ps]
    s = N.LMSettings(maxNumIt=4)

    def solve(ids):
        for i in ids:
            gs[i].set_params(ps[i].cams, ps[i].pts)
        reasons, chi2, its, _ = N.lm_solve_batch([gs[i] for i in ids], s)
        return [(r, c, k) + gs[i].get_params() for r, c, k, i in zip(reasons, chi2, its, ids)]

    alone = [solve([i])[0] for i in range(8)]
    for _ in range(3):
        for a, b in zip(alone, solve(range(8))):
            assert a[:3] == b[:3] and a[2] == 4
            assert np.array_equal(a[3], b[3]) and np.array_equal(a[4], b[4])
    for g in gs:
        g.close()
