"""The 1D line solve (one CTA per instance, fh_hline.cuh) at the edges of its
tiling: one equation, partly filled chunks, exactly full panels and lines of
several panels, for both CTA sizes.

The reference is the oracle's step with its elimination in long double: in the
reference solver's own order a 2050-node line rounds by 1.5e-12 of its largest
value, more than the bound below.

Tolerance: the factors and both substitutions are sums and products of
positive terms with ~2 N roundings along a line; the parity bound of the plain
path, 1e-12 of the largest value, is the bound of every solver test here.
Where an instance itself is more sensitive than that (a long fine line), twice
the distance by which the oracle moves under perturbations of 2^-53."""
import math

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _relmax(a, b):
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


def _problem(N, kind, seed):
    from theses_code_gb300 import workloads
    rng = np.random.default_rng(seed)
    if kind == "l1":
        return workloads.caputo_1d(N - 1, 0.8, 1.0, 1e-3)
    p = workloads.psi_batch(n=1, seed=seed)[0][0]
    p = dict(p, N=N)
    if kind == "dirichlet":  # fixed value at the left end: Al[1] = 0
        p.update(al_left=0.0, bt_left=0.3)
    x = np.arange(N + 2) / N
    u = 0.3 + 0.1 * rng.random() * np.cos(3 * x)
    u[N:] = 0.0
    return p, u


def _solve(p, u0, steps):
    """The oracle's H_solver step (fho_h_solve) with the Thomas recurrences in long double."""
    ld = np.longdouble
    N, a, tau = p["N"], p["alpha"], p["tau"]
    dL = p["L"] / N
    Dg = dL ** -2.0
    l1 = p["weights"] == 0
    Da = tau ** (-a if l1 else -1.0) / math.gamma(2.0 - a)
    u = np.array(u0, dtype=np.float64)
    hist = []
    for step in range(1, steps + 1):
        n = len(hist)
        ts = np.zeros(N + 2)
        for t in range(1, n - 1):  # slot 0 carries no weight
            w = O.l1_b(n - t - 1, a) if l1 else O.psi_int(t, t + 1, step + 1, tau, a, p["beta"]) * (1 - a)
            ts += w * (hist[t + 1] - hist[t])
        wc = 1.0 if l1 else O.psi_int(step, step + 1, step + 1, tau, a, p["beta"]) * (1 - a)
        K = np.full(N + 1, p["kc"]) if p["kmodel"] == 0 else p["kc"] * np.exp(p["kgam"] * u[:N + 1])
        A, B = Dg * K[:N - 1] * p["cinv"], Dg * K[2:] * p["cinv"]
        R = p["cinv"] * (K[2:] + K[:N - 1]) * Dg + Da * wc
        om = -Da * wc * u[1:N]
        if p["gravity"]:
            om = om + (K[1:N] - K[:N - 1]) / dL
        om = om + Da * ts[1:N]
        A, B, R, om = (x.astype(ld) for x in (A, B, R, om))
        al, bt = np.empty(N, dtype=ld), np.empty(N, dtype=ld)  # Al[i+1], Bt[i+1] at i
        al[0], bt[0] = ld(p["al_left"]), ld(p["bt_left"])
        for i in range(1, N):
            g = 1 / (R[i - 1] - A[i - 1] * al[i - 1])
            al[i] = B[i - 1] * g
            bt[i] = g * (A[i - 1] * bt[i - 1] - om[i - 1])
        x = ld(p["u_right"])
        u[N:] = p["u_right"]
        for i in range(N - 1, -1, -1):
            x = al[i] * x + bt[i]
            u[i] = x
        hist.append(u.copy())
    return u


# equations = N - 1: up to 8 per thread of 128 or 256 threads, then panels of 1024 / 2048
SIZES = (2, 3, 33, 128, 129, 130, 256, 257, 1024, 1025, 1026, 1100, 2049, 2050, 2500)


@pytest.mark.parametrize("small", [True, False])  # eight warps per line below 152 instances, four from there on
@pytest.mark.parametrize("kind", ["psi", "dirichlet", "l1"])
def test_line_solve_tiling(small, kind):
    from theses_code_gb300._lib import Context
    from theses_code_gb300.solvers import HSolverBatch
    probs = [_problem(N, kind, 100 + k) for k, N in enumerate(SIZES)]
    steps = 12
    jobs = probs if small else probs + [_problem(9, kind, 7)] * (152 - len(probs))
    ctx = Context(0)
    s = HSolverBatch(ctx, [p for p, _ in jobs], steps + 1)
    s.set_persistent(False)
    s.set_u([u for _, u in jobs])
    s.calc_step(steps)
    got = s.get_u()
    s.close()
    ctx.close()
    for (p, u), g in zip(probs, got):
        ref = _solve(p, u, steps)
        sens = _relmax(O.h_solve(dict(p, pert=2.0 ** -53), u, steps)[0], O.h_solve(p, u, steps)[0])
        assert _relmax(g, ref) <= max(1e-12, 2.0 * sens), (kind, p["N"], _relmax(g, ref), sens)


@pytest.mark.parametrize("kind,sizes", [
    ("psi", (2,)),                                 # one owner per node
    ("psi", (3, 31, 200, 257, 766, 1024, 1025)),   # up to the largest line, its layers beyond shared memory
    ("psi", (40,) * 25 + (1025,) * 7),             # three owners of up to 343 nodes
    ("l1", (66, 255, 1025)),
    ("dirichlet", (29, 512)),
    ("psi", (2046, 70)),                           # lines of more nodes: k_h_persistent
])
def test_persistent_shared_nodes(kind, sizes):
    """k_h_pers_own (and k_h_persistent) against the kernel-by-kernel path, and the same bits
    however the steps are spread over calls (tolerance as above)."""
    from theses_code_gb300._lib import Context
    from theses_code_gb300.solvers import HSolverBatch
    steps = 90
    jobs = [_problem(N, kind, 300 + k) for k, N in enumerate(sizes)]
    ctx = Context(0)
    got = []
    for persistent, calls in ((False, (steps,)), (True, (steps,)), (True, (1, 2, 37, 50))):
        s = HSolverBatch(ctx, [p for p, _ in jobs], steps + 1)
        s.set_persistent(persistent)
        s.set_u([u for _, u in jobs])
        for n in calls:
            s.calc_step(n)
        got.append(s.get_u())
        s.close()
    ctx.close()
    seen = {}
    for (p, u), a, b, c in zip(jobs, *got):
        np.testing.assert_array_equal(b, c)
        if p["N"] not in seen:
            seen[p["N"]] = _relmax(O.h_solve(dict(p, pert=2.0 ** -53), u, steps)[0], O.h_solve(p, u, steps)[0])
        assert _relmax(b, a) <= max(1e-12, 2.0 * seen[p["N"]]), (kind, p["N"], _relmax(b, a), seen[p["N"]])
