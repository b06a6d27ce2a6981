"""The resident Atangana-Baleanu solve (k_ab_resident) at the edges of its
tiling: one equation, partly filled chunks, the limits of four, eight and
sixteen solving warps, a block boundary, several source rows with boundary
values, one captured call and uneven calls, against the oracle.

Tolerances: the modes' bounds, 1e-9 (blocked) and 1e-12 (FP64) of the largest
value; the call patterns run the same sums on the same entries, so they agree to
the roundings of the field's round trip through FP64 (none) and must be equal."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

STEPS = 150  # block boundaries at 64 (FP64) and 128


@pytest.mark.parametrize("mode,tol", [("FH_AB_BLOCKED", 1e-9), ("FH_AB_FP64", 1e-12)])
@pytest.mark.parametrize("m", [2, 3, 33, 129, 130, 513, 514, 1025, 1026, 2049, 2559])
def test_resident_tiling(m, mode, tol):
    from theses_code_gb300 import _lib, workloads
    from theses_code_gb300._lib import Context
    from theses_code_gb300.solvers import ABSolver
    cfg, src, _, _, C0 = workloads.ab_1d(m=m, alpha=0.7, tau=1e-3, seed=m)
    rows = 5
    src = np.concatenate([src * (1.0 + 0.3 * k) for k in range(rows)])
    bl, br = 0.01 * np.arange(rows), -0.02 * np.arange(rows)
    at = np.minimum(np.arange(STEPS), rows - 1)
    w = O.ab_weights(STEPS, cfg["tau"], cfg["alpha"])
    ref, _ = O.ab_solve(m, STEPS, cfg["tau"], cfg["alpha"], w, src[at], bl[at], br[at], C0)
    ctx = Context(0)
    got = []
    for solves in (((STEPS,),), ((1, 60, 80, 9),), ((64, 64, 22),), ((140,), (140, 10))):
        s = ABSolver(ctx, m, STEPS, cfg["tau"], cfg["alpha"], getattr(_lib, mode))
        s.set_source(src, bl, br)
        for calls in solves:  # the second solve replays the first one's steps, then goes on
            s.set_c(C0)
            for n in calls:
                s.calc_step(n)
        got.append(s.get_c())
        s.close()
    ctx.close()
    assert float(np.max(np.abs(got[0] - ref)) / np.max(np.abs(ref))) <= tol
    for g in got[1:]:
        assert np.array_equal(g, got[0])


def test_source_and_coefficient_after_a_captured_solve():
    """A second solve after a new source and current-step coefficient uses them."""
    from theses_code_gb300 import workloads
    from theses_code_gb300._lib import FH_AB_BLOCKED, FH_AB_FP64, Context
    from theses_code_gb300.solvers import ABSolver
    m, n = 100, 40
    cfg, src, bl, br, C0 = workloads.ab_1d(m=m, alpha=0.7, tau=1e-3, seed=1)
    ctx = Context(0)
    for mode in (FH_AB_FP64, FH_AB_BLOCKED):
        def fresh(rows, coef):
            s = ABSolver(ctx, m, n, cfg["tau"], cfg["alpha"], mode)
            s.set_source(rows, np.zeros(len(rows)), np.zeros(len(rows)))
            s.set_current_coef(coef)
            s.set_c(C0)
            s.calc_step(n)
            out = s.get_c()
            s.close()
            return out
        two = np.concatenate([2.0 * src, 3.0 * src])
        s = ABSolver(ctx, m, n, cfg["tau"], cfg["alpha"], mode)
        s.set_source(src, bl, br)
        s.set_current_coef(1e-3)
        for rows, coef in ((src, 1e-3), (two, 1e-3), (two, 2e-3)):
            s.set_source(rows, np.zeros(len(rows)), np.zeros(len(rows)))
            s.set_current_coef(coef)
            s.set_c(C0)
            s.calc_step(n)
            assert np.array_equal(s.get_c(), fresh(rows, coef))
        s.close()
    ctx.close()
