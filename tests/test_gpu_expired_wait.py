"""After a device wait that ran out, reading the result reports it, and a new
initial state starts a solve that is as good as any.  The flags are set by the
library's test entries, as the kernels set them; no wait runs out here."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _expire(ctx, name, handle):
    fn = getattr(ctx.L, name)
    fn.argtypes, fn.restype = [C.c_void_p], C.c_int
    assert fn(handle) == 0


def _solves(ctx, make, start, step, read, name):
    """The result of a solve, its repetition after an expired wait, and that of the device entry."""
    from theses_code_gb300._lib import FH_ETIMEOUT, FhError
    s = make()
    out = []
    for k in range(3):
        start(s, k)
        step(s)
        out.append(np.copy(read(s)))
        _expire(ctx, name, s.h)
        with pytest.raises(FhError) as e:
            read(s)
        assert e.value.code == FH_ETIMEOUT
    s.close()
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])


@pytest.mark.parametrize("mode", ["FH_AB_FP64", "FH_AB_BLOCKED"])
def test_ab(mode):
    import torch
    from theses_code_gb300 import _lib, workloads
    from theses_code_gb300.solvers import ABSolver
    from conftest import torch_ordered_context
    ctx = torch_ordered_context()
    cfg, src, bl, br, C0 = workloads.ab_1d(m=40, alpha=0.7, tau=1e-3, seed=1)
    dev = torch.from_numpy(C0).cuda()
    torch.cuda.synchronize()

    def make():
        s = ABSolver(ctx, 40, 70, cfg["tau"], cfg["alpha"], getattr(_lib, mode))
        s.set_source(src, bl, br)
        return s
    _solves(ctx, make, lambda s, k: s.set_c_device(dev.data_ptr()) if k == 1 else s.set_c(C0),
            lambda s: s.calc_step(70), lambda s: s.get_c(), "fh_ab_test_expire")
    ctx.close()


@pytest.mark.parametrize("mode", ["FH_TG_FP64", "FH_TG_DF64", "FH_TG_BLOCKED"])
def test_tg(mode):
    import torch
    from theses_code_gb300 import _lib, workloads
    from theses_code_gb300.solvers import TGSolver
    from conftest import torch_ordered_context
    ctx = torch_ordered_context()
    p, V2, C0 = workloads.convection_2d(20, 18, alpha=0.7, tau=5e-4, d=0.1, seed=1)
    dv, dc = torch.from_numpy(V2).cuda(), torch.from_numpy(C0).cuda()
    torch.cuda.synchronize()
    _solves(ctx, lambda: TGSolver(ctx, p, 70, getattr(_lib, mode)),
            lambda s, k: s.set_state_device(dv.data_ptr(), dc.data_ptr()) if k == 1 else s.set_state(V2, C0),
            lambda s: s.calc_step(70), lambda s: s.get_c(), "fh_tg_test_expire")
    ctx.close()


def test_h_persistent():
    import torch
    from theses_code_gb300 import workloads
    from theses_code_gb300.solvers import HSolverBatch
    from conftest import torch_ordered_context
    ctx = torch_ordered_context()
    params, U0 = zip(*(workloads.caputo_1d(40 + k, 0.7, 0.5, 1e-3) for k in range(5)))
    dev = torch.from_numpy(np.concatenate(U0)).cuda()
    torch.cuda.synchronize()
    _solves(ctx, lambda: HSolverBatch(ctx, list(params), 41),
            lambda s, k: s.set_u_device(dev.data_ptr()) if k == 1 else s.set_u(list(U0)),
            lambda s: s.calc_step(40), lambda s: np.concatenate(s.get_u()), "fh_h_batch_test_expire")
    ctx.close()
