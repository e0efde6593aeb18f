"""nl_lm_solve_batch keeps one captured sub-iteration per handle: what the capture
froze may not outlive the setting it was made under."""
import numpy as np
import pytest

from nelson_b200 import native as N
from nelson_b200.problems import make_config, problem_from_pairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [N.PREC_FP64, N.PREC_MIXED])
def test_settings_after_the_capture(prec):
    """A wait bound of one poll makes every solve of several tiles give up, so each
    sub-iteration is rejected; with the default bound the first result comes back.
    The solver kind, set after the capture, gives the same parameters (the envelope
    solver skips zero tiles only)."""
    p = make_config(1, 0.3)  # 60 cameras x 9: five tiles
    g = N.BAProblemGPU.from_ba(p, precision=prec)
    s = N.LMSettings(maxNumIt=3, maxNumSubIt=4)

    def solve():
        g.set_params(p.cams, p.pts)
        reason, chi2, its, _ = N.lm_solve_batch([g], s)
        return reason[0], float(chi2[0]), int(its[0]), g.get_params()[1]

    first = solve()
    assert first[2] == 3
    g.set_wait_limit(1)
    limited = solve()
    assert limited[2] == 0 and limited[0] == "MaxSubIterationReached"
    g.set_wait_limit(0)
    again = solve()
    assert again[:3] == first[:3] and np.array_equal(again[3], first[3])
    g.set_solver_kind(N.SOLVER_ENVELOPE)
    env = solve()
    assert env[2] == 3 and env[1] == pytest.approx(first[1], rel=1e-12)
    g.close()


@pytest.mark.parametrize("kind", [N.SOLVER_DENSE, N.SOLVER_ENVELOPE])
def test_no_iteration_then_increment(kind):
    """A batch that may not iterate captures nothing that the next call relies on: the
    handle's first increment after it equals a fresh handle's, also where the memory
    of the reduced system (a band of three tiles) held other values before."""
    pt = np.repeat(np.arange(1500), 3)
    p = problem_from_pairs(40, 1500, pt % 38 + np.tile(np.arange(3), 1500), pt, bc=9, seed=2)

    def handle():
        g = N.BAProblemGPU.from_ba(p, precision=N.PREC_MIXED)
        g.set_solver_kind(kind)
        return g

    # handles whose factorisation overflows leave their memory to the next ones (every
    # other one stays, so that the allocator keeps the memory's blocks)
    old = [handle() for _ in range(12)]
    for g in old:
        g.update(True)
        assert not g.compute_increment(0.0, -1e9)
    for g in old[::2]:
        g.close()

    def increment(g):
        g.update(True)
        assert g.compute_increment(0.0, 1e-3 * g.max_abs_hdiag())
        return g.increment()

    gs = [handle() for _ in range(6)]
    want = None
    for i, g in enumerate(gs):
        if i > 0:  # the first one is the fresh handle
            reason, _, its, _ = N.lm_solve_batch([g], N.LMSettings(maxNumIt=0))
            assert reason[0] == "MaxIterationReached" and its[0] == 0
        got = increment(g)
        want = want or got
        for a, b in zip(got, want):
            assert np.array_equal(a, b)
    for g in gs + old:
        g.close()
