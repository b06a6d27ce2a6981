"""fh_ab_set_mode where the blocked mode finds no memory: the call says so, and the
solver goes on in its previous mode.  Device memory is held by torch meanwhile."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_mode_without_memory_keeps_the_solver():
    import torch
    from theses_code_gb300 import _lib, workloads
    from theses_code_gb300._lib import Context, FhError
    from theses_code_gb300.solvers import ABSolver
    m, steps = 1500, 40000  # planes of 0.5 GB
    cfg, src, bl, br, C0 = workloads.ab_1d(m=m, alpha=0.7, tau=1e-5, seed=1)
    ctx = Context(0)
    got = []
    for fail in (False, True):
        s = ABSolver(ctx, m, steps, cfg["tau"], cfg["alpha"], _lib.FH_AB_FP64)
        if fail:
            free = torch.cuda.mem_get_info()[0]
            hold = torch.empty(free - (200 << 20), dtype=torch.uint8, device="cuda")
            with pytest.raises(FhError) as e:
                _lib.check(ctx.L.fh_ab_set_mode(s.h, _lib.FH_AB_BLOCKED), ctx.h)
            assert e.value.code == _lib.FH_ENOMEM
            del hold
            torch.cuda.empty_cache()
        s.set_source(src, bl, br)
        s.set_c(C0)
        s.calc_step(150)
        got.append(s.get_c())
        s.close()
    ctx.close()
    assert np.array_equal(got[0], got[1])
