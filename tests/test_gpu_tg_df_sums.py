"""The DF64 mode's sums over every stored layer (restricted summing with a cut
below every weight): grids so large that the points alone fill the GPU, and more
layers than one CTA's shared memory holds weights for, against the FP64 mode.

Tolerance: the mode's 1e-12 of the largest value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sN,M,steps", [(64, 48, 150), (592, 596, 3085)])
def test_every_layer_in_pairs(sN, M, steps):
    from theses_code_gb300 import _lib, workloads
    from theses_code_gb300._lib import Context
    from theses_code_gb300.solvers import TGSolver
    p, V2, C0 = workloads.convection_2d(sN, M, alpha=0.8, tau=5e-4, d=0.1, seed=2)
    ctx = Context(0)
    got = []
    for mode, cut in ((_lib.FH_TG_DF64, 1e-300), (_lib.FH_TG_FP64, 0.0)):
        s = TGSolver(ctx, p, steps, mode)
        s.set_restricted(cut)
        s.set_state(V2, C0)
        s.calc_step(steps)
        got.append(s.get_c())
        s.close()
    ctx.close()
    assert float(np.max(np.abs(got[0] - got[1]))) <= 1e-12 * float(np.max(np.abs(got[1])))
