"""The older layers' sums at FP64 accuracy on the tensor cores (fh_far64.cu),
through the 2D solver's FP64 and DF64 modes: fewer points than a tile, ragged
last tiles, one K split and several, and step counts around the blocks of 32
steps and the groups of 128 layers, against the oracle.

Tolerance: the plain path's 1e-12 of the largest value; the digits cut a layer at
2^-55 of its group's largest, below FP64's own rounding of the same sums.

The sums are scale-free: every digit is relative to its point's and row's
largest exponent, FP64 operations and power-of-two scalings are exact, so a
field times 2^k gives the result times 2^k bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _solve(sN, M, steps, mode, calls=None, beta=1.0, scale=1.0):
    from theses_code_gb300 import _lib, workloads
    from theses_code_gb300._lib import Context
    from theses_code_gb300.solvers import TGSolver
    p, V2, C0 = workloads.convection_2d(sN, M, alpha=0.7, tau=5e-4, d=0.1, seed=sN + M)
    p["beta"] = beta
    ctx = Context(0)
    s = TGSolver(ctx, p, steps, getattr(_lib, mode))
    for cs in calls or ((steps,),):
        s.set_state(V2, C0 * scale)
        for n in cs:
            s.calc_step(n)
    got = s.get_c()
    s.close()
    ctx.close()
    return got, (p, V2, C0)


@pytest.mark.parametrize("mode", ["FH_TG_FP64", "FH_TG_DF64"])
@pytest.mark.parametrize("sN,M,steps,beta", [(2, 2, 40, 1.0), (9, 7, 33, 1.0), (10, 8, 64, 1.0), (11, 13, 65, 1.3),
                                             (30, 31, 129, 1.0), (61, 64, 161, 1.0), (62, 62, 300, 1.0),
                                             (170, 155, 97, 0.8)])
def test_far_rows_vs_oracle(sN, M, steps, beta, mode):
    got, (p, V2, C0) = _solve(sN, M, steps, mode, beta=beta)
    ref, _ = O.tg_solve(p, V2, C0, steps)
    ref = np.asarray(ref).ravel()
    assert float(np.max(np.abs(got - ref)) / np.max(np.abs(ref))) <= 1e-12


@pytest.mark.parametrize("mode", ["FH_TG_FP64", "FH_TG_DF64"])
def test_far_rows_call_patterns(mode):
    base, _ = _solve(33, 40, 150, mode)
    for calls in (((1, 31, 1, 100, 17),), ((32, 64, 54),), ((140,), (140, 10))):
        assert np.array_equal(_solve(33, 40, 150, mode, calls)[0], base)


@pytest.mark.parametrize("mode,k", [("FH_TG_FP64", -600), ("FH_TG_FP64", 500), ("FH_TG_DF64", -40), ("FH_TG_DF64", 40)])
def test_far_rows_scale_free(mode, k):
    base, _ = _solve(33, 40, 100, mode)
    got, _ = _solve(33, 40, 100, mode, scale=2.0 ** k)
    keep = np.abs(base) > 1e-6 * np.max(np.abs(base))  # clear of the FP32 pairs' smallest numbers
    assert np.array_equal(np.ldexp(got, -k)[keep], base[keep])


@pytest.mark.parametrize("mode", ["FH_TG_FP64", "FH_TG_DF64"])
@pytest.mark.parametrize("sN,M", [(153, 154), (154, 153), (305, 306), (306, 305)])
def test_sweep_lines_vs_oracle(sN, M, mode):
    """One, two and four lines per CTA, the sums ahead among their idle warps."""
    got, (p, V2, C0) = _solve(sN, M, 36, mode)
    ref = np.asarray(O.tg_solve(p, V2, C0, 36)[0]).ravel()
    assert float(np.max(np.abs(got - ref)) / np.max(np.abs(ref))) <= 1e-12


@pytest.mark.parametrize("seed", [2, 3])
def test_pair_rows_keep_their_precision(seed):
    """DF64 against FP64 where a group's level sums cancel: a far row's pair holds 2^-48 of its sum,
    and the steps add such errors with random signs (2-norm; bound 2^-47)."""
    from theses_code_gb300 import _lib, workloads
    from theses_code_gb300._lib import Context
    from theses_code_gb300.solvers import TGSolver
    alpha = float(np.random.default_rng(seed).uniform(0.5, 0.95))
    p, V2, C0 = workloads.convection_2d(150, 90, alpha=alpha, tau=5e-4, d=0.1, seed=seed)
    got = []
    for mode in (_lib.FH_TG_DF64, _lib.FH_TG_FP64):
        ctx = Context(0)
        s = TGSolver(ctx, p, 300, mode)
        s.set_state(V2, C0)
        s.calc_step(300)
        got.append(np.array(s.get_c()))
        s.close()
        ctx.close()
    assert np.linalg.norm(got[0] - got[1]) <= 2.0 ** -47 * np.linalg.norm(got[1])


@pytest.mark.parametrize("steps", [1, 2, 3, 128, 129, 256, 257])
def test_lag_weights_vs_oracle(steps):
    """psi = t: the weight table from its lags, at the edges of the CTAs that make and copy it."""
    got, (p, V2, C0) = _solve(12, 9, steps, "FH_TG_FP64")
    ref = np.asarray(O.tg_solve(p, V2, C0, steps)[0]).ravel()
    assert float(np.max(np.abs(got - ref)) / np.max(np.abs(ref))) <= 1e-12
