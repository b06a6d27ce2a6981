"""The fused 2D sweeps of the blocked mode where their control flow depends on the
grid: one to four warps of a line's group with equations, more in one direction than
in the other, lines that end at and around a warp's 128 equations, and step counts
around the sub-blocks of 8 and the blocks of 64 steps, against the oracle.

Tolerance: the mode's 1e-9 of the largest value.  Calls of any length run the same
arithmetic, so they must agree bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _solve(sN, M, steps, calls, alpha, seed):
    from theses_code_gb300 import _lib, workloads
    from theses_code_gb300._lib import Context
    from theses_code_gb300.solvers import TGSolver
    p, V2, C0 = workloads.convection_2d(sN, M, alpha=alpha, tau=5e-4, d=0.1, seed=seed, C1=0.1)
    ctx = Context(0)
    s = TGSolver(ctx, p, steps, _lib.FH_TG_BLOCKED)
    s.set_state(V2, C0)
    for n in calls:
        s.calc_step(n)
    got = s.get_c()
    s.close()
    ctx.close()
    return got, (p, V2, C0)


@pytest.mark.parametrize("sN,M,steps", [(2, 300, 73), (300, 2, 73), (40, 500, 65), (500, 40, 66), (129, 128, 72),
                                        (128, 129, 72), (130, 257, 71), (257, 130, 70), (258, 129, 64), (385, 386, 17),
                                        (386, 385, 16), (513, 2, 9), (513, 513, 9)])
def test_warps_per_line(sN, M, steps):
    got, (p, V2, C0) = _solve(sN, M, steps, (steps,), 0.8, sN + M)
    ref = np.asarray(O.tg_solve(p, V2, C0, steps)[0]).ravel()
    assert float(np.max(np.abs(got - ref))) <= 1e-9 * float(np.max(np.abs(ref)))


@pytest.mark.parametrize("sN,M", [(40, 300), (300, 129)])
def test_calls_of_any_length(sN, M):
    base, _ = _solve(sN, M, 80, (80,), 0.7, 5)
    for calls in ((7, 1, 1, 55, 1, 15), (8, 56, 16), (63, 9, 8)):
        assert np.array_equal(_solve(sN, M, 80, calls, 0.7, 5)[0], base)


@pytest.mark.parametrize("alpha,seed", [(0.55, 21), (0.7, 22), (0.95, 23)])
def test_largest_grid(alpha, seed):
    """513 x 513 past a block, against the FP64 mode."""
    from theses_code_gb300 import _lib
    from theses_code_gb300._lib import Context
    from theses_code_gb300.solvers import TGSolver
    steps = 140
    got, (p, V2, C0) = _solve(513, 513, steps, (steps,), alpha, seed)
    ctx = Context(0)
    s = TGSolver(ctx, p, steps, _lib.FH_TG_FP64)
    s.set_state(V2, C0)
    s.calc_step(steps)
    ref = s.get_c()
    s.close()
    ctx.close()
    assert float(np.max(np.abs(got - ref))) <= 1e-9 * float(np.max(np.abs(ref)))
