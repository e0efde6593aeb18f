"""Parameter exchange below, at and above the size that goes through pinned memory
(512 KB set, 2 MB get), with cameras over the edges of a CTA (128 cameras).  Points are copied:
equal to the last bit.  Cameras pass through a rotation matrix: 1e-12."""
import numpy as np
import pytest

from nelson_b200 import native as N

pytestmark = pytest.mark.gpu
LIMIT = (2 << 20) // 8


@pytest.mark.parametrize("bc", [6, 9])
@pytest.mark.parametrize("nc", [1, 127, 128, 129, 300])
@pytest.mark.parametrize("np_", [1, 43, 21000, "limit", "over"])
def test_round_trip(bc, nc, np_):
    if np_ in ("limit", "over"):
        np_ = (LIMIT - nc * bc) // 3 + (np_ == "over")
    r = np.random.default_rng(nc + np_)
    g = N.BAProblemGPU(bc, nc, np_)
    for _ in range(2):
        u, v = r.uniform(-0.9, 0.9, (nc, bc)), r.normal(size=(np_, 3))
        g.set_params(u, v)
        gu, gv = g.get_params()
        assert np.array_equal(gv, v)
        assert np.abs(gu - u).max() <= 1e-12
    g.close()
