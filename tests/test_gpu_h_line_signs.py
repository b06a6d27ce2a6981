"""The 1D line solve where its factors are no sums of positive terms: negative kc
and cinv, and u_0 = al_left u_1 + bt_left with al_left outside [0, 1], against the
oracle (the reference's serial order).

Tolerance: that order itself loses N^2 2^-53 of the largest value to cancellation."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 160])  # the persistent solve and the batch's
@pytest.mark.parametrize("kind", ["const", "exp"])
@pytest.mark.parametrize("change", [dict(kc=-0.3, cinv=-1.0), dict(kc=-1e-4), dict(al_left=1.5, bt_left=0.1),
                                    dict(al_left=-0.5, bt_left=0.1), dict(al_left=3.0, bt_left=0.1)])
def test_signs(change, kind, n):
    from theses_code_gb300 import _lib, workloads
    from theses_code_gb300._lib import Context
    from theses_code_gb300.solvers import HSolverBatch
    N, steps = 200, 30
    p, u = workloads.caputo_1d(N - 1, 0.7, 0.5, 1e-3)
    p = dict(p, **change)
    if kind == "exp":
        p.update(kmodel=_lib.FH_K_EXP, kgam=0.7, gravity=1)
    ctx = Context(0)
    s = HSolverBatch(ctx, [p] * n, steps + 1)
    s.set_u([u] * n)
    s.calc_step(steps)
    got = s.get_u()[n - 1]
    s.close()
    ctx.close()
    ref, _ = O.h_solve(p, u, steps)
    assert np.max(np.abs(got - ref)) <= N * N * 2.0 ** -53 * np.max(np.abs(ref))
