"""The 2D solver's weight table (psi = t) against the weights a step computes by
itself: restricted summing with a cut below every weight leaves each weight as the
formula gives it, so the blocked solve must repeat the plain one bit for bit, also
where the half-step scheme lets the field grow (alpha near 1/2 on fine grids) and
would turn another rounding of the weights into another field."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sN,M,steps,alpha", [(64, 48, 200, 0.7), (33, 40, 70, 0.95), (160, 500, 300, 0.51)])
def test_table_keeps_the_formula(sN, M, steps, alpha):
    from theses_code_gb300 import _lib, workloads
    from theses_code_gb300._lib import Context
    from theses_code_gb300.solvers import TGSolver
    p, V2, C0 = workloads.convection_2d(sN, M, alpha=alpha, tau=5e-4, d=0.1, seed=3)
    ctx = Context(0)
    got = []
    for cut in (0.0, 1e-300):
        s = TGSolver(ctx, p, steps, _lib.FH_TG_BLOCKED)
        s.set_restricted(cut)
        s.set_state(V2, C0)
        s.calc_step(steps)
        got.append(s.get_c())
        s.close()
    ctx.close()
    assert np.array_equal(got[0], got[1])
