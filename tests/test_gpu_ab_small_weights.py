"""Atangana-Baleanu blocked mode with lag weights far below 1 (a short step: they
are integrals over it), where the entries, differences over that step, are as far
above: the weights' slices must keep their 32 bits.

Tolerance: the mode's 1e-9 of the largest value, against the FP64 mode."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [-14, -60, -112])
@pytest.mark.parametrize("m", [2, 5])
def test_short_steps(m, k):
    from theses_code_gb300 import _lib
    from theses_code_gb300._lib import Context
    from theses_code_gb300.solvers import ABSolver
    steps = 300
    x = np.arange(m + 1) / m
    src = np.sin(0.05 * np.arange(steps))[:, None] * np.sin(np.pi * x)[None, :]
    ctx = Context(0)
    got = []
    for mode in (_lib.FH_AB_BLOCKED, _lib.FH_AB_FP64):
        s = ABSolver(ctx, m, steps, 2.0 ** k, 0.6, mode)
        s.set_source(src, np.zeros(steps), np.zeros(steps))
        s.set_c(np.zeros(m + 1))
        s.calc_step(steps)
        got.append(s.get_c())
        s.close()
    ctx.close()
    assert np.max(np.abs(got[0] - got[1])) <= 1e-9 * np.max(np.abs(got[1]))
