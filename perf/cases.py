"""The work a user has this library do, as cases that can be timed and compared.

A case is a dict of plain values; `listed()` names the fixed ones, `draw(rng)`
gives others of the same ranges.  Kinds:

  h      1D H_solver solves (HSolverBatch): `n` instances of Nmin..Nmax nodes,
         `steps` steps; problem "l1" (L1 Caputo weights, constant K: the
         mt_minimal form), "psi" (psi-Caputo, psi = t^beta with beta per
         instance, D(u) = D0 exp(gamma u), gravity: moisture transport)
  tg     one 2D ADI solve (TGSolver), sN x M intervals
  ab     one 1D Atangana-Baleanu solve (ABSolver), m intervals
  sum    one history sum over stored layers (fh_history_sum), the call that
         replaces the reference's Sum kernels

`mode` is the history mode of the solver ("fp64", "df64", "blocked").  A pass
of a solve sets the initial state from the host, runs every step and reads the
solution back, as a driver loop does; with `chunk` it advances that many steps
per call without graph replay, as the serving loop does.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from theses_code_gb300 import _lib, workloads
from theses_code_gb300._lib import Context
from theses_code_gb300.solvers import ABSolver, HSolverBatch, TGSolver

H_MODES = {"fp64": _lib.FH_H_FP64, "df64": _lib.FH_H_DF64, "blocked": _lib.FH_H_BLOCKED}
TG_MODES = {"fp64": _lib.FH_TG_FP64, "df64": _lib.FH_TG_DF64, "blocked": _lib.FH_TG_BLOCKED}
AB_MODES = {"fp64": _lib.FH_AB_FP64, "blocked": _lib.FH_AB_BLOCKED}


def listed():
    return [
        # a single short solve inside someone else's loop: the smallest call
        dict(name="h_l1_short", kind="h", problem="l1", n=1, Nmin=65, Nmax=65, steps=40, mode="fp64"),
        # the 1D Caputo configuration: N = 200 interior points, 1000 steps
        dict(name="h_l1_N200", kind="h", problem="l1", n=1, Nmin=201, Nmax=201, steps=1000, mode="fp64"),
        # one round of a parameter fit: 32 candidate solves of one soil column
        dict(name="h_psi_fit32", kind="h", problem="psi", n=32, Nmin=512, Nmax=512, steps=250, mode="fp64"),
        # a batch of uneven instances on the plain path
        dict(name="h_psi_batch", kind="h", problem="psi", n=1000, Nmin=64, Nmax=1024, steps=250, mode="fp64"),
        # a long batch on the mixed-precision path
        dict(name="h_psi_blocked", kind="h", problem="psi", n=512, Nmin=64, Nmax=1024, steps=1500, mode="blocked"),
        # the smallest 2D grid of the serving mix, advanced in the serving loop's chunks
        dict(name="tg_64_served", kind="tg", sN=64, M=64, steps=500, mode="blocked", chunk=250),
        # an ordinary 2D solve on the plain path, odd and uneven sizes
        dict(name="tg_251x187_fp64", kind="tg", sN=251, M=187, steps=500, mode="fp64", chunk=0),
        # plain-path accuracy at HBM speed on the benchmark's grid
        dict(name="tg_512_df64", kind="tg", sN=512, M=512, steps=500, mode="df64", chunk=0),
        # the headline configuration: 512 x 512, 2000 steps, mixed precision
        dict(name="tg_512_blocked", kind="tg", sN=512, M=512, steps=2000, mode="blocked", chunk=0),
        # an ordinary Atangana-Baleanu solve on the plain path
        dict(name="ab_1023_fp64", kind="ab", m=1023, steps=2500, mode="fp64"),
        # the Atangana-Baleanu configuration: 2048 intervals, 20000 steps
        dict(name="ab_2048_blocked", kind="ab", m=2048, steps=20000, mode="blocked"),
        # the history sum as a call of its own, both half-step sums of one step
        dict(name="sum_386x386", kind="sum", rows=2, layers=777, points=386 * 386),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["h", "h", "h", "tg", "tg", "tg", "ab", "sum"])
    if kind == "h":
        problem = rng.choice(["l1", "psi", "psi"])
        if problem == "l1":
            N = _log_int(rng, 65, 1024)
            return dict(kind="h", problem="l1", n=_log_int(rng, 1, 32), Nmin=N, Nmax=N, steps=_log_int(rng, 40, 1000),
                        mode="fp64")
        n = _log_int(rng, 8, 1000)
        Nmax = _log_int(rng, 128, 1024)
        mode = rng.choice(["fp64", "df64", "blocked"])
        return dict(kind="h", problem="psi", n=n, Nmin=rng.randint(64, Nmax), Nmax=Nmax,
                    steps=_log_int(rng, 50, 250 if mode != "blocked" else 800), mode=mode)
    if kind == "tg":
        mode = rng.choice(["fp64", "df64", "blocked", "blocked"])
        top = 2000 if mode == "blocked" else 500
        return dict(kind="tg", sN=_log_int(rng, 48, 512), M=_log_int(rng, 48, 512), steps=_log_int(rng, 100, top),
                    mode=mode, chunk=rng.choice([0, 0, 250]))
    if kind == "ab":
        mode = rng.choice(["fp64", "blocked"])
        return dict(kind="ab", m=_log_int(rng, 128, 2048), steps=_log_int(rng, 200, 2500 if mode == "fp64" else 8000),
                    mode=mode)
    return dict(kind="sum", rows=rng.choice([1, 2]), layers=_log_int(rng, 20, 2000),
                points=2 * _log_int(rng, 1000, 140000))


# ------------------------------------------------------------------- inputs
def _h_problem(case, seed):
    """(params, U0) per instance.  The node counts belong to the case, the rest to the seed."""
    if case["problem"] == "psi":
        Ns = np.random.default_rng(case["n"]).integers(case["Nmin"], case["Nmax"] + 1, size=case["n"])
        params, _ = workloads.psi_batch(case["n"], seed=seed)
        params = [dict(p, N=int(N)) for p, N in zip(params, Ns)]
        U0s = []
        for N in Ns:
            u = 0.25 * (1.0 + np.cos(math.pi * np.arange(N + 2) / N))
            u[N:] = 0.0
            U0s.append(u)
        return params, U0s
    rng = np.random.default_rng(seed)
    params, U0s = [], []
    for _ in range(case["n"]):
        p, U0 = workloads.caputo_1d(case["Nmax"] - 1, alpha=float(rng.uniform(0.5, 0.95)),
                                    D=float(rng.uniform(0.1, 1.0)))
        x = np.arange(p["N"] + 2) / p["N"]
        for q in range(2, 6):  # sin(pi x) and a few seeded higher modes
            U0 = U0 + rng.normal() / q ** 2 * np.sin(q * math.pi * x)
        U0[0] = U0[p["N"]] = U0[p["N"] + 1] = 0.0
        params.append(p)
        U0s.append(U0)
    return params, U0s


def _tg_problem(case, seed):
    rng = np.random.default_rng(seed)
    return workloads.convection_2d(case["sN"], case["M"], alpha=float(rng.uniform(0.5, 0.95)), tau=5e-4, d=0.1,
                                   seed=seed)


def _ab_problem(case, seed):
    rng = np.random.default_rng(seed)
    return workloads.ab_1d(case["m"], alpha=float(rng.uniform(0.5, 0.8)), tau=1e-4, seed=seed)


def _sum_problem(case, seed, device):
    """L1-like decaying weights and layer differences of mixed sign."""
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    K, P, M = case["layers"], case["points"], case["rows"]
    D = torch.randn(K, P, dtype=torch.float64, device=device, generator=g)
    a = 0.3 + 0.6 * torch.rand(1, dtype=torch.float64, device=device, generator=g)
    lag = torch.arange(K, 0, -1, dtype=torch.float64, device=device)
    W = torch.stack([(lag + 0.5 * m + 0.5) ** (1 - a) - (lag + 0.5 * m - 0.5) ** (1 - a) for m in range(M)]).contiguous()
    return W, D


def prepare(case, seed):
    kind = case["kind"]
    ctx = Context(0)
    s = dict(case=case, ctx=ctx)
    if kind == "h":
        params, U0 = _h_problem(case, seed)
        s["solver"] = HSolverBatch(ctx, params, case["steps"] + 1, H_MODES[case["mode"]])
        s["U0"] = U0
    elif kind == "tg":
        p, V2, C0 = _tg_problem(case, seed)
        if case["chunk"]:
            ctx.set_graphs(False)
        s["solver"] = TGSolver(ctx, p, case["steps"], TG_MODES[case["mode"]])
        s["V2"], s["C0"] = V2, C0
    elif kind == "ab":
        p, src, bl, br, C0 = _ab_problem(case, seed)
        sv = ABSolver(ctx, p["m"], case["steps"], p["tau"], p["alpha"], AB_MODES[case["mode"]])
        sv.set_source(src, bl, br)
        s["solver"], s["C0"] = sv, C0
    else:
        # on torch's stream, like the rest of a torch program
        ctx.set_stream(torch.cuda.current_stream().cuda_stream)
        s["W"], s["D"] = _sum_problem(case, seed, "cuda")
        s["S"] = torch.empty(case["rows"], case["points"], dtype=torch.float64, device="cuda")
    return s


# --------------------------------------------------------------------- pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sum":
        W, D, S = state["W"], state["D"], state["S"]
        state["ctx"].call("fh_history_sum", case["rows"], case["layers"], case["points"], W.data_ptr(), W.shape[1],
                          D.data_ptr(), D.shape[1], S.data_ptr(), S.shape[1])
        return S
    sv = state["solver"]
    if kind == "h":
        sv.set_u(state["U0"])
        sv.calc_step(case["steps"])
        return np.concatenate(sv.get_u())
    if kind == "tg":
        sv.set_state(state["V2"], state["C0"])
        left = case["steps"]
        while left > 0:
            k = min(left, case["chunk"] or left)
            sv.calc_step(k)
            left -= k
        return sv.get_c()
    sv.set_c(state["C0"])
    sv.calc_step(case["steps"])
    return sv.get_c()


def work(case):
    """Inputs read once, the result written once; the history terms (one
    multiply-add per stored difference, row and node) and ~8 multiply-adds per
    node and line solve."""
    kind = case["kind"]
    if kind == "sum":
        K, P, M = case["layers"], case["points"], case["rows"]
        return dict(bytes=8 * (K * P + M * K + M * P), flops=2 * M * K * P)
    n = case["steps"]
    if kind == "h":
        P = case["n"] * ((case["Nmin"] + case["Nmax"]) // 2 + 2)  # the mean instance
        return dict(bytes=16 * P, flops=P * (n * (n - 1) + 16 * n))
    if kind == "tg":
        P = (case["sN"] + 2) * (case["M"] + 2)
        return dict(bytes=24 * P, flops=2 * P * (n * (n - 1) + 16 * n))
    P = case["m"] + 1
    return dict(bytes=24 * P, flops=P * (n * (n - 1) + 16 * n))


# -------------------------------------------------------------------- exact
def exact(case, seed):
    """The same results in 64 bits from the definitions, in torch: weights by
    quadrature or closed form, dense history sums, line solves by cyclic
    reduction."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    if kind == "sum":
        W, D = _sum_problem(case, seed, dev)
        return W @ D
    if kind == "h":
        return _exact_h(*_h_problem(case, seed), case["steps"], dev)
    if kind == "tg":
        return _exact_tg(*_tg_problem(case, seed), case["steps"], dev)
    return _exact_ab(*_ab_problem(case, seed), case["steps"], dev)


def _t_weights(lag0, lag1, b):
    """lag0^b - lag1^b for lag0 > lag1 >= 0 (b = 1 - alpha), without cancellation."""
    r = torch.where(lag1 > 0, torch.log1p((lag1 - lag0) / lag0), torch.full_like(lag0 + lag1, -math.inf))
    return -(lag0 ** b) * torch.expm1(b * r)


def _pcr(a, b, c, d):
    """a x[i-1] + b x[i] + c x[i+1] = d along the last axis (a[0] = c[-1] = 0)."""
    n, s = d.shape[-1], 1
    while s < n:
        z = lambda x, k: torch.nn.functional.pad(x, (k, 0))[..., :n] if k > 0 else torch.nn.functional.pad(x, (0, -k))[..., -k:]  # noqa: E731
        one = lambda x, k: torch.nn.functional.pad(x, (k, 0), value=1.0)[..., :n] if k > 0 else torch.nn.functional.pad(x, (0, -k), value=1.0)[..., -k:]  # noqa: E731
        k1, k2 = a / one(b, s), c / one(b, -s)
        b = b - z(c, s) * k1 - z(a, -s) * k2
        d = d - z(d, s) * k1 - z(d, -s) * k2
        a, c = -z(a, s) * k1, -z(c, -s) * k2
        s *= 2
    return d / b


def _exact_h(params, U0, steps, dev):
    f8 = torch.float64
    col = lambda k: torch.tensor([float(p[k]) for p in params], dtype=f8, device=dev)[:, None]  # noqa: E731
    n = len(params)
    Ns = torch.tensor([p["N"] for p in params], device=dev)[:, None]
    Nm = int(Ns.max())
    tau, al, be, kc, kg, cinv = (col(k) for k in ("tau", "alpha", "beta", "kc", "kgam", "cinv"))
    grav, al1, bt1, ur = (col(k) for k in ("gravity", "al_left", "bt_left", "u_right"))
    psi, const = params[0]["weights"] == _lib.FH_W_PSI, params[0]["kmodel"] == _lib.FH_K_CONST
    dL = col("L") / Ns
    Dg, b1 = dL ** -2, 1 - al
    Da = tau ** (-1.0 if psi else -al) / torch.exp(torch.lgamma(2 - al))
    u = torch.zeros(n, Nm + 2, dtype=f8, device=dev)
    for i, x in enumerate(U0):
        u[i, :len(x)] = torch.from_numpy(np.asarray(x))
    node = torch.arange(1, Nm, device=dev)[None, :]
    live, first, last = node < Ns, node == 1, node == Ns - 1
    hist = torch.zeros(n, steps + 1, Nm + 1 - 2, dtype=f8, device=dev)  # differences of the solved layers
    glx, glw = np.polynomial.legendre.leggauss(20)
    glx, glw = (torch.from_numpy(x).to(dev) for x in ((glx + 1) / 2, glw / 2))
    if psi:
        # Gauss-Jacobi nodes for the weight (1 - x)^-alpha on [0, 1] (Golub-Welsch)
        k = torch.arange(24, dtype=f8, device=dev)[None, :]
        ab = -al
        diag = -ab * ab / ((2 * k + ab) * (2 * k + ab + 2))
        diag[:, 0] = (-ab / (ab + 2))[:, 0]
        q = k[:, 1:]
        off = 4 * q * (q + ab) * q * (q + ab) / ((2 * q + ab) ** 2 * (2 * q + ab + 1) * (2 * q + ab - 1))
        off[:, 0] = (4 * (1 + ab) / ((2 + ab) ** 2 * (3 + ab)))[:, 0]
        e, v = torch.linalg.eigh((torch.diag_embed(diag) + torch.diag_embed(off.sqrt(), 1) +
                                  torch.diag_embed(off.sqrt(), -1)).cpu())
        e, v = e.to(dev), v.to(dev)
        gjx, gjw = (e + 1) / 2, v[:, 0, :] ** 2 / b1
        scale = tau ** (1 - al * be) * b1
    unit = torch.ones(1, device=dev, dtype=f8)

    def rel(x, X):  # 1 - (x/X)^beta
        return -torch.expm1(be * torch.log1p((x - X) / X))

    for os in range(steps):
        X = float(os + 2)  # the step's time index, tstep + 1
        if psi:
            x = X - 1 + gjx
            wc = (gjw * (X ** be * rel(x, X) / (X - x)) ** -al).sum(1, keepdim=True) * scale
        else:
            wc = torch.ones(n, 1, dtype=f8, device=dev)
        ts = None
        if os >= 3:
            t = torch.arange(1, os - 1, dtype=f8, device=dev)  # slot 0 carries no weight
            if psi:
                w = torch.zeros(n, t.numel(), dtype=f8, device=dev)
                for g in range(20):
                    w += glw[g] * (X ** be * rel(t[None, :] + glx[g], X)) ** -al
                w *= scale
            else:
                w = _t_weights((os - t)[None, :], (os - t - 1)[None, :], b1)
            ts = torch.bmm(w[:, None, :], hist[:, 1:os - 1])[:, 0]
        K = kc.expand(n, Nm + 2) if const else kc * torch.exp(kg * u)
        A, B = Dg * K[:, :Nm - 1] * cinv, Dg * K[:, 2:Nm + 1] * cinv
        R = cinv * (K[:, 2:Nm + 1] + K[:, :Nm - 1]) * Dg + Da * wc
        om = -Da * wc * u[:, 1:Nm] + grav * (K[:, 1:Nm] - K[:, :Nm - 1]) / dL
        if ts is not None:
            om = om + Da * ts
        diag = torch.where(live, torch.where(first, A * al1 - R, -R), unit)
        rhs = torch.where(live, om - torch.where(first, A * bt1, 0 * A) - torch.where(last, B * ur, 0 * B), 0 * om)
        xin = _pcr(torch.where(live & ~first, A, 0 * A), diag, torch.where(live & ~last, B, 0 * B), rhs)
        old = u
        u = torch.zeros_like(u)
        u[:, 1:Nm] = xin
        u[:, :1] = al1 * u[:, 1:2] + bt1
        for o in (0, 1):
            u.scatter_(1, Ns + o, ur)
        if os >= 1:
            hist[:, os - 1] = (u - old)[:, 1:Nm]
    out = u.cpu().numpy()
    return np.concatenate([out[i, :p["N"] + 2] for i, p in enumerate(params)])


class _FixedLines:
    """Line systems A u[i-1] - R u[i] + B u[i+1] = Om with fixed coefficients,
    u[0] = al1 u[1] + bt1 and u[N] = u[N-1], by cyclic reduction along axis 1."""

    def __init__(self, A, R, B, al1, bt1):
        self.al1, self.bt1, self.A1 = al1, bt1, A[:, 0].clone()
        a, b, c = A.clone(), -R.clone(), B.clone()
        b[:, 0] += A[:, 0] * al1
        a[:, 0] = 0
        b[:, -1] += B[:, -1]
        c[:, -1] = 0
        n, s = a.shape[1], 1
        self.lv = []
        while s < n:
            sh = lambda x, k: torch.roll(x, k, 1)  # noqa: E731
            k1, k2 = a / sh(b, s), c / sh(b, -s)  # zero where the neighbour is outside
            k1[:, :s] = 0
            k2[:, n - s:] = 0
            b, a, c = b - sh(c, s) * k1 - sh(a, -s) * k2, -sh(a, s) * k1, -sh(c, -s) * k2
            self.lv.append((s, k1, k2))
            s *= 2
        self.b = b

    def solve(self, om):
        d = om.clone()
        d[:, 0] -= self.A1 * self.bt1
        for s, k1, k2 in self.lv:
            up, dn = torch.roll(d, s, 1), torch.roll(d, -s, 1)
            d = torch.addcmul(torch.addcmul(d, up, k1, value=-1), dn, k2, value=-1)
        return d / self.b


def _exact_tg(p, V2, C0, steps, dev):
    f8 = torch.float64
    sN, M, tau, a = p["sN"], p["M"], p["tau"], p["alpha"]
    V = torch.from_numpy(V2).to(dev).reshape(M + 2, sN + 2)
    C = torch.from_numpy(C0).to(dev).reshape(M + 2, sN + 2).clone()
    b, st, Da = 1 - a, p["sigma"] / tau, 1.0 / math.gamma(1 - a)
    S2, d = 0.5 * p["S"], p["d"]
    wt = Da * tau ** b / b  # int over [x0, x1] tau of (X tau - s)^-alpha = tau^b / b (lag0^b - lag1^b)
    kx = wt * 0.5 ** b
    ky = kx
    kyh = wt * (1.0 - 0.5 ** b)
    v = V[1:M, 1:sN]
    Ax, Bx = v / p["dL"] * (d / p["dL"] + 0.5), v / p["dL"] * (d / p["dL"] - 0.5)
    Ay = v / p["dLx"] ** 2 * d
    xl = _FixedLines(Ax, st * kx + Ax + Bx, Bx, 0.0, p["C1"])
    yl = _FixedLines(Ay.T.contiguous(), (st * ky + 2 * Ay).T.contiguous(), Ay.T.contiguous(), 1.0, 0.0)
    hist = torch.zeros(steps, (M - 1) * (sN - 1), dtype=f8, device=dev)
    ks = torch.arange(steps, dtype=f8, device=dev)
    for j in range(steps):
        old = C.clone()
        om = S2 - st * kx * C[1:M, 1:sN]
        if j >= 1:
            k = ks[:j]
            w = wt * torch.stack([_t_weights(j + h - k, j + h - k - 1, b) for h in (0.5, 1.0)])
            hs = (w @ hist[:j]).reshape(2, M - 1, sN - 1)
            om = om + st * hs[0]
        u = xl.solve(om)
        C[1:M, 1:sN] = u
        C[1:M, 0] = p["C1"]
        C[1:M, sN] = C[1:M, sN + 1] = u[:, -1]
        c = C[1:M, 1:sN]
        om = S2 - st * ky * c + st * kyh * (old[1:M, 1:sN] - c)
        if j >= 1:
            om = om + st * hs[1]
        u = yl.solve(om.T.contiguous()).T
        C[1:M, 1:sN] = u
        C[0, 1:sN] = u[0]
        C[M, 1:sN] = C[M + 1, 1:sN] = u[-1]
        hist[j] = (C - old)[1:M, 1:sN].reshape(-1)
    return C.reshape(-1).cpu().numpy()


def _exact_ab(p, src, bl, br, C0, steps, dev):
    f8 = torch.float64
    m, tau, a = p["m"], p["tau"], p["alpha"]
    lam = a / (1 - a)
    # I(lag): the Mittag-Leffler series integrated over the lag's interval
    lag = torch.arange(1, steps + 2, dtype=f8, device=dev)
    lx = torch.log(lag * tau)
    lr = torch.where(lag >= 2, torch.log1p(-1 / lag), torch.full_like(lag, -math.inf))
    w = torch.zeros(steps + 2, dtype=f8, device=dev)
    for k in range(400):
        q = a * k + 1
        t = torch.exp(k * math.log(lam) + q * lx - math.lgamma(q + 1)) * -torch.expm1(q * lr)
        w[1:] += -t if k & 1 else t
        if k > 8 and float((t.abs() / w[1:].abs()).max()) < 1e-18:
            break
    Ii = float(w[1])
    h = 1.0 / m
    A, Cc, Bd = -1 / h ** 2 - 0.5 / h, -1 / h ** 2 + 0.5 / h, Ii / (1 - a) + 2 / h ** 2
    # the inverse of the interior matrix, column by column (Thomas on the unit matrix)
    n = m - 1
    al = np.zeros(n)
    G = np.eye(n)
    den = Bd
    G[0] /= den
    al[0] = Cc / den
    for i in range(1, n):
        den = Bd - A * al[i - 1]
        al[i] = Cc / den
        G[i, :i + 1] = (G[i, :i + 1] - A * G[i - 1, :i + 1]) / den
    for i in range(n - 2, -1, -1):
        G[i] -= al[i] * G[i + 1]
    G = torch.from_numpy(G).to(dev)
    src = torch.from_numpy(src).to(dev)
    C = torch.from_numpy(np.array(C0)).to(dev)
    dts = torch.zeros(steps + 1, m + 1, dtype=f8, device=dev)
    for i in range(1, steps + 1):
        r = min(i - 1, src.shape[0] - 1)
        rp = Ii / (1 - a) * C + src[r]
        if i >= 2:
            rp = rp - (w[2:i + 1].flip(0) @ dts[:i - 1]) / (1 - a)
        rhs = rp[1:m].clone()
        rhs[0] -= A * float(bl[r])
        rhs[-1] -= Cc * float(br[r])
        new = torch.empty_like(C)
        new[1:m] = G @ rhs
        new[0], new[m] = float(bl[r]), float(br[r])
        dts[i - 1] = (new - C) / tau
        C = new
    return C.cpu().numpy()
