"""Which lines of the mixed-precision mode the double-float solve may take
(fh_hline_df.cuh): none so short that pairs cost accuracy, none whose states or
boundary values pairs do not hold.

Tolerances.  Short lines against the FP64 mode within one history block: the plain
path's 1e-12 and, for the sums in pairs, 2^-47 of the solution per step.  Scaled
states: the mode's own 1e-9 (a line is linear for constant K; before the fourth
step no history counts)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(params, U0, steps, mode):
    from theses_code_gb300._lib import Context
    from theses_code_gb300.solvers import HSolverBatch
    ctx = Context(0)
    s = HSolverBatch(ctx, params, steps + 1, mode)
    s.set_u(U0)
    s.calc_step(steps)
    u = s.get_u()
    s.close()
    ctx.close()
    return u


@pytest.mark.parametrize("N,seed", [(256, 2), (512, 1), (640, 2), (640, 3), (767, 3)])
def test_short_lines_keep_fp64(N, seed):
    from theses_code_gb300 import _lib, workloads
    steps = 60
    params = [dict(p, N=N) for p in workloads.psi_batch(8, seed=seed)[0]]
    u = 0.25 * (1 + np.cos(np.pi * np.arange(N + 2) / N))
    u[N:] = 0.0
    a = _run(params, [u] * 8, steps, _lib.FH_H_BLOCKED)
    b = _run(params, [u] * 8, steps, _lib.FH_H_FP64)
    for x, y in zip(a, b):
        assert np.max(np.abs(x - y)) <= (1e-12 + steps * 2.0 ** -47) * np.max(np.abs(y))


@pytest.mark.parametrize("what,k,steps", [("state", -60, 3), ("state", -120, 3), ("state", -200, 3), ("right", -200, 3),
                                          ("left", -140, 3), ("right", 140, 2), ("left", 140, 2)])
@pytest.mark.parametrize("N", [900, 1025])
def test_scaled_values(N, what, k, steps):
    """The whole state, or a boundary value beside a zero state, times 2^k."""
    from theses_code_gb300 import _lib, workloads
    p, u = workloads.caputo_1d(N - 1, 0.7, 0.5, 1e-3)
    if what == "state":
        u = u * 2.0 ** k
    else:
        u = np.zeros(N + 2)
        p["u_right" if what == "right" else "bt_left"] = 2.0 ** k
    a, = _run([p], [u], steps, _lib.FH_H_BLOCKED)
    b, = _run([p], [u], steps, _lib.FH_H_FP64)
    assert np.all(np.isfinite(b)) and np.max(np.abs(b)) > 0.0
    assert np.max(np.abs(a - b)) <= 1e-9 * np.max(np.abs(b))


@pytest.mark.parametrize("left", [1.5, -0.5])
def test_left_condition_outside_the_unit_interval(left):
    """u_0 = left u_1 + bt: the factors are no longer sums of positive terms."""
    from theses_code_gb300 import _lib, workloads
    p, u = workloads.caputo_1d(899, 0.7, 0.5, 1e-3)
    p.update(al_left=left, bt_left=0.2)
    a, = _run([p], [u], 20, _lib.FH_H_BLOCKED)
    b, = _run([p], [u], 20, _lib.FH_H_FP64)
    assert np.max(np.abs(a - b)) <= (1e-12 + 20 * 2.0 ** -47) * np.max(np.abs(b))
