"""One contracted history sum (fh_far64.cu) against exact arithmetic, where the
history falls in time and the weights rise towards the newest layer.

A line of one unknown (m = 2, zero ends): C' = (c C + f - S / (1 - a)) / (c + 8),
S = sum of weight times stored difference.  The source f of every step is chosen so
that the differences are about k^-fall with alternating signs, so that S outweighs
C; C is read after each step, so that S of a step is known exactly from what the
solver stored.  The step is so long that a difference's own share of the next one
is 1/15: roundings die out.

Tolerance.  The seven digits cut a value 2^-55 below its group's largest D, a
weight likewise below W, and the dropped levels start 2^-56 below: about 2^-53 D W
per layer together, with random signs 2^3.5 times that for 128 layers.  The weights
in digits differ by at most 2^4 (exponents by 3), so the sum of the terms'
magnitudes is at least D W / 16: an error of 2^-45.5 of it; 2^-45 is allowed, and
eight roundings of the other terms."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alpha", [0.5, 0.7, 0.95])
@pytest.mark.parametrize("fall", [0, 1, 2])
def test_one_sum_of_a_falling_history(alpha, fall):
    from theses_code_gb300 import _lib
    from theses_code_gb300._lib import Context
    from theses_code_gb300.solvers import ABSolver
    steps, a, tau, coef = 194, 0.0625, 2.0, 2.0 ** -4
    lag = np.arange(1, steps + 2, dtype=np.float64)
    b = 1.0 - alpha
    w = np.concatenate([[1.0], lag ** b - (lag - 1.0) ** b])[:steps + 1]  # lag 2 weighs 1: the newest layer
    c = coef / (1 - a)
    rng = np.random.default_rng(3)
    # wanted differences / tau; C ends at 0
    d = (np.arange(steps) + 1.0) ** -fall * (1.0 + 0.3 * rng.random(steps)) * (-1.0) ** np.arange(steps)
    C = np.concatenate([[0.0], np.cumsum(d) * tau])
    C -= C[-1]
    f = np.zeros(steps)
    for i in range(steps):
        S = float(w[1:i + 1][::-1] @ d[:i]) if i else 0.0  # entry t has lag i + 1 - t
        f[i] = (c + 8.0) * C[i + 1] - c * C[i] + S / (1 - a)
    src = np.zeros((steps, 3))
    src[:, 1] = f
    ctx = Context(0)
    s = ABSolver(ctx, 2, steps, tau, a, _lib.FH_AB_FP64)
    s.set_lag_weights(w)
    s.set_current_coef(coef)
    s.set_source(src, np.zeros(steps), np.zeros(steps))
    s.set_c(np.array([0.0, C[0], 0.0]))
    got = [float(C[0])]
    for _ in range(steps):
        s.calc_step(1)
        got.append(float(s.get_c()[1]))
    s.close()
    ctx.close()
    D = [(got[t + 1] - got[t]) / tau for t in range(steps)]  # tau is a power of two
    W = [Fraction(x) for x in w]
    for i in (128, 129, 140, 192, 193):  # first steps of the blocks and others
        terms = [W[i - t] * Fraction(D[t]) for t in range(i)]  # w[l - 1] is lag l
        ref = (Fraction(c) * Fraction(got[i]) + Fraction(f[i]) - sum(terms) / Fraction(1 - a)) / Fraction(c + 8.0)
        mag = float(sum(abs(x) for x in terms)) / (1 - a) / (c + 8.0)
        rest = (abs(c * got[i]) + abs(f[i])) / (c + 8.0) + mag
        err = abs(float(Fraction(got[i + 1]) - ref))
        assert err <= 2.0 ** -45 * mag + 8 * 2.0 ** -53 * rest, (i, err / mag)
