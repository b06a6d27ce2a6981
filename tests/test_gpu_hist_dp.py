"""The history sum by integer dot products (k_hist_dp) at the edges of its
groups (16 layers), stages (512) and CTAs (256 points), and where values or
weights leave what its digits hold, against sums in extended precision.

Tolerance: FP64's own bound for a sum of K terms, K 2^-53 of the sum of
magnitudes, and as much as 64 terms for the digits' cut (16 terms of a group,
2^-55 of its largest value and weight, which within a group are at most 2^4
above those of the largest term)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sum(W, D, name="fh_history_sum"):
    import torch
    from theses_code_gb300._lib import Context
    ctx = Context(0)
    M, K = W.shape
    P = D.shape[1]
    Wd, Dd = torch.as_tensor(W, device="cuda"), torch.as_tensor(D, device="cuda")
    S = torch.full((M, P), 7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.call(name, M, K, P, Wd.data_ptr(), K, Dd.data_ptr(), P, S.data_ptr(), P)
    ctx.sync()
    got = S.cpu().numpy()
    ctx.close()
    return got


def _check(W, D, live=slice(None)):
    ld = np.longdouble
    K = W.shape[1]
    with np.errstate(invalid="ignore"):
        ref = (W.astype(ld)[:, :, None] * D.astype(ld)[None, :, live]).sum(axis=1)
        scale = (np.abs(W).astype(ld)[:, :, None] * np.abs(D).astype(ld)[None, :, live]).sum(axis=1)
    for name in ("fh_history_sum", "fh_history_sum_noalloc"):
        got = _sum(W, D, name)[:, live]
        assert np.all(np.abs(got - ref) <= (K + 64) * ld(2) ** -53 * scale + 1e-300)


@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("K,P", [(63, 258), (64, 2), (65, 254), (79, 256), (80, 258), (512, 514), (513, 1026),
                                 (1100, 30), (20001, 64)])
def test_edges(K, P, M):
    rng = np.random.default_rng(K + P + M)
    lag = np.arange(K, 0, -1.0)
    W = np.stack([(lag + 0.5 * m + 0.5) ** 0.3 - (lag + 0.5 * m - 0.5) ** 0.3 for m in range(M)])
    _check(W, rng.standard_normal((K, P)))


def test_values_of_any_size():
    rng = np.random.default_rng(3)
    K, P = 200, 300
    D = rng.standard_normal((K, P)) * 2.0 ** rng.integers(-80, 80, size=(K, P))
    D[:, :40] *= 2.0 ** rng.integers(-900, 850, size=(1, 40))
    D[:, 50] = 0.0
    D[7, 51:60] = 0.0
    D[:, 60] = 5e-324
    W = rng.uniform(0.5, 1.0, size=(2, K))
    _check(W, D)


def test_weights_of_any_size():
    rng = np.random.default_rng(4)
    K, P = 200, 300
    W = rng.standard_normal((2, K)) * 2.0 ** rng.integers(-60, 60, size=(2, K))
    W[0, 16:48] = 0.0
    W[1, 100] = 0.0
    # large values where the weights are small
    D = rng.standard_normal((K, P)) / np.where(W[:1] != 0, np.abs(W[:1]), 1.0).T
    _check(W, D)


def test_not_finite():
    rng = np.random.default_rng(5)
    K, P = 100, 64
    D, W = rng.standard_normal((K, P)), rng.uniform(0.5, 1.0, size=(2, K))
    D[20, 5], D[21, 6], D[90, 7] = np.inf, np.nan, -np.inf
    _check(W, D, live=np.r_[0:5, 8:64])
    got = _sum(W, D)
    assert np.all(np.isnan(got[:, 6])) and np.all(got[:, 5] == np.inf) and np.all(got[:, 7] == -np.inf)


def test_batch_tiles():
    """k_hist_tiles_dp: instances at the edges of its 128-node CTAs against the oracle, and a slot
    whose earlier occupant left layers that are not finite (tolerance of the plain path, or twice the
    distance by which the oracle moves under perturbations of 2^-53)."""
    from oracle import oracle as O
    from theses_code_gb300 import workloads
    from theses_code_gb300._lib import Context
    from theses_code_gb300.solvers import HSolverBatch
    sizes = (2, 125, 126, 127, 128, 254, 255, 256, 513)
    params, U0 = [], []
    for k, N in enumerate(sizes):
        p = dict(workloads.psi_batch(n=1, seed=40 + k)[0][0], N=N)
        x = np.arange(N + 2) / N
        u = 0.3 + 0.1 * np.cos(3 * x)
        u[N:] = 0.0
        params.append(p)
        U0.append(u)
    ctx = Context(0)
    ctx.set_graphs(False)
    s = HSolverBatch(ctx, params, 200)
    s.set_persistent(False)
    bad = [u.copy() for u in U0]
    bad[4][3] = np.inf
    s.set_u(bad)
    s.calc_step(30)
    s.restart(4, params[4], U0[4])
    s.calc_step(100)
    got = s.get_u()
    s.close()
    ctx.close()
    for k, (p, u) in enumerate(zip(params, U0)):
        n = 100 if k == 4 else 130
        ref = O.h_solve(p, u, n)[0]
        sens = np.max(np.abs(O.h_solve(dict(p, pert=2.0 ** -53), u, n)[0] - ref)) / np.max(np.abs(ref))
        assert np.max(np.abs(got[k] - ref)) <= max(1e-12, 2.0 * sens) * np.max(np.abs(ref)), p["N"]
