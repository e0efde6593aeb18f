"""The persistent batch at the edges of its 32-column Cholesky panels, its
16-row tiles and its warps' edge groups: reduced systems whose last panel holds
1 to 32 columns, the largest system it takes (768 rows), 9-parameter cameras
(blocks of 27 values), fixed nodes and weights, against the handle's own FP64
solve (nl_lm_solve) of the same problem.  Four iterations, far from convergence:
cost to 1e-9 (the tolerance of the batch's oracle test), parameters to 1e-7."""
import numpy as np
import pytest

from nelson_b200 import native as N
from nelson_b200.problems import ring_scene, with_fixed_nodes

pytestmark = pytest.mark.gpu


def check(ps):
    s = N.LMSettings(maxNumIt=4)
    hs = [N.BAProblemGPU.from_ba(p) for p in ps]
    ref = []
    for p, g in zip(ps, hs):
        _, tr, its, _ = g.lm_solve(s)
        ref.append((tr[-1, 2], its, g.get_params()))
        g.set_params(p.cams, p.pts)
    b = N.PersistentBatch(hs)
    _, chi2, its, _, _, _ = b.lm_solve(s)
    for k, g in enumerate(hs):
        c, p = g.get_params()
        assert its[k] == ref[k][1]
        assert chi2[k] == pytest.approx(ref[k][0], rel=1e-9)
        assert np.abs(c - ref[k][2][0]).max() <= 1e-7 * np.abs(c).max()
        assert np.abs(p - ref[k][2][1]).max() <= 1e-7 * np.abs(p).max()
    b.close()
    for g in hs:
        g.close()


@pytest.mark.parametrize("bc,cams", [(6, (3, 5, 6, 11, 16, 22, 43)), (9, (3, 4, 7, 11, 32, 57))])
def test_panel_remainders(bc, cams):
    check([ring_scene(nc, 40 + 7 * nc, 3, min(8, nc), bc, 100 + nc, weights=nc % 2 == 0) for nc in cams])


@pytest.mark.parametrize("bc,cams", [(6, 128), (9, 85)])
def test_largest_system(bc, cams):
    check([ring_scene(cams, 900, 3, 8, bc, 9)])


@pytest.mark.parametrize("bc,nc,npts,fc,fp", [(6, 13, 301, 3, 11), (9, 9, 150, 2, 0)])
def test_fixed_nodes(bc, nc, npts, fc, fp):
    check([with_fixed_nodes(ring_scene(nc, npts, 3, 8, bc, 4, weights=bc == 6), fc, fp)])
