"""The trailing update's figures in nl_phase_timings (flops, bytes, launches) against a count
over tiles: what the timed launches do, no more -- the diagonal tiles that the chain's own
kernel updates and the rows past the envelope are not theirs."""
import numpy as np
import pytest

from nelson_b200 import native as N
from nelson_b200.problems import problem_from_pairs

pytestmark = pytest.mark.gpu
NB = 128


def handle(span, prec, kind):
    """100 cameras x 9 (eight tiles), each point in `span` consecutive cameras."""
    npts = 1500
    pt = np.repeat(np.arange(npts), 3)
    cam = pt % (101 - span) + np.tile([0, span // 2, span - 1], npts)
    p = problem_from_pairs(100, npts, cam, pt, bc=9, seed=4)
    g = N.BAProblemGPU.from_ba(p, precision=prec)
    g.set_solver_kind(kind)
    g.update(True)
    assert g.compute_increment(0.0, 1e-3 * g.max_abs_hdiag())
    t = g.phase_times()
    g.close()
    return t


def last_tiles(span, kind, nt=8):
    """Last tile row with nonzeros in the panels' rows, never before an earlier panel's."""
    if kind == N.SOLVER_DENSE:
        return [nt - 1] * nt
    i, j = np.tril_indices(900)
    a, b = j // 9, i // 9  # cameras of a lower-triangle entry
    d = b - a
    nz = (d == 0) | (d == span // 2) | (d == span - 1) | (d == span - 1 - span // 2)
    first = [min((j[nz & (i // NB == t)] // NB).min(), t) for t in range(nt)]
    run = [max(t for t in range(nt) if first[t] <= k) for k in range(nt)]
    return list(np.maximum.accumulate(run))


@pytest.mark.parametrize("kind", [N.SOLVER_DENSE, N.SOLVER_ENVELOPE])
@pytest.mark.parametrize("span", [3, 31, 61])
def test_fp64(span, kind):
    t = handle(span, N.PREC_FP64, kind)
    flop = tiles = launches = 0
    for k, last in enumerate(last_tiles(span, kind)):
        r = last - k - 1  # tile rows below the next diagonal tile: a column, a triangle
        if r > 0:
            flop += 2 * NB * NB * NB * r + NB * (NB * r) * (NB * r + 1)
            tiles += r + r * (r + 1) // 2
            launches += 2
    assert t["update_flop"] == flop
    assert t["update_bytes"] == tiles * NB * NB * 8 * 2
    assert t["update_launches"] == launches


def test_mixed_dense():
    t = handle(61, N.PREC_MIXED, N.SOLVER_DENSE)
    nt, group = 8, 4
    flop = sum(NB * (NB * (nt - 1 - k)) * (NB * (nt - 1 - k) + 1) for k in range(nt))
    # the chain's kernel: the last panel on a tile inside a group of panels, all four of a
    # group on the next group's first tile
    chain = sum(group if j % group == 0 else 1 for j in range(1, nt))
    assert t["update_flop"] == flop - chain * NB * NB * (NB + 1)
    assert t["update_launches"] > 0 and t["update_bytes"] > 0
