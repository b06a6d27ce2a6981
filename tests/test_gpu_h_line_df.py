"""The double-float 1D line solve of the mixed-precision mode (fh_hline_df.cuh)
against the plain FP64 mode, at the edges of its tiling (one equation, partly
filled chunks, the longest single panel, the first line past it) for both CTA
sizes, and where a line leaves its range and runs the FP64 solve.

Tolerance: elimination and substitutions are products and sums of positive
terms, at most ~8 double-float operations (2^-47 each) per equation along a
line of N; the steps damp earlier errors.  Together with the plain path's own
parity bound: 8 N 2^-47 + 1e-12 of the largest value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 20  # all within the first history block: no sliced far rows


def _solve(params, U0, mode):
    from theses_code_gb300._lib import Context
    from theses_code_gb300.solvers import HSolverBatch
    s = HSolverBatch(Context(0), params, STEPS + 1, mode)
    s.set_u(U0)
    s.calc_step(STEPS)
    return s.get_u()


def _instance(N, kind, seed):
    from theses_code_gb300 import workloads
    if kind == "l1":
        p = workloads.caputo_1d(N - 1, 0.8, 1.0, 1e-3)[0]
    else:
        p = dict(workloads.psi_batch(n=1, seed=seed)[0][0], N=N)
    if kind == "dirichlet":
        p.update(al_left=0.0, bt_left=0.3)
    x = np.arange(N + 2) / N
    u = 0.25 * (1 + np.cos(np.pi * x))
    u[N:] = p["u_right"]
    return p, u


@pytest.mark.parametrize("n", [1, 152])  # eight and four warps per line
@pytest.mark.parametrize("kind", ["psi", "dirichlet", "l1"])
@pytest.mark.parametrize("N", [2, 3, 34, 129, 130, 513, 1024, 1025, 1026])
def test_edges(N, kind, n):
    from theses_code_gb300 import _lib
    # uneven companions for the four-warp form
    sizes = [N] + [max(2, N - 7 * k % N) for k in range(1, n)]
    params, U0 = zip(*(_instance(Nk, kind, 3 + k) for k, Nk in enumerate(sizes)))
    a = _solve(list(params), list(U0), _lib.FH_H_BLOCKED)
    b = _solve(list(params), list(U0), _lib.FH_H_FP64)
    for x, y, Nk in zip(a, b, sizes):
        assert np.max(np.abs(x - y)) <= (8 * Nk * 2.0 ** -47 + 1e-12) * np.max(np.abs(y))


@pytest.mark.parametrize("change", [dict(kgam=60.0), dict(kgam=-60.0), dict(kc=1e-300, cinv=1e300), dict(kc=1e-25)],
                         ids=["steep", "steep-", "scaled", "weak"])
def test_out_of_range(change):
    """exp(gam u) or the row sums past the pairs' range, or only their factors."""
    from theses_code_gb300 import _lib
    p, u = _instance(200, "psi", 5)
    p = dict(p, **change)
    a, = _solve([p], [u], _lib.FH_H_BLOCKED)
    b, = _solve([p], [u], _lib.FH_H_FP64)
    live = np.isfinite(b)  # "steep" leaves FP64 too
    np.testing.assert_array_equal(np.isfinite(a), live)
    assert np.max(np.abs(a - b)[live]) <= (8 * 200 * 2.0 ** -47 + 1e-12) * np.max(np.abs(b[live]))
