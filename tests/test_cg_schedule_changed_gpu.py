"""A solver refuses a matrix whose schedule was changed after its creation, also
where its solves run on the chip."""
from __future__ import annotations

import pytest

import gooseberry_b200 as gb
from gooseberry_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,f32", [(gb.CG_F64, False), (gb.CG_MIXED, False),
                                      (gb.CG_MIXED, True)])
@pytest.mark.parametrize("shape", [(40, 40), (150, 150), (1100, 1100)])
def test_refused(mode, f32, shape):
    import torch
    A = W.diffusion(shape, 1, 0.5, 2.0)
    M = gb.CsrMatrix.from_host(A, f64=True, f32=True)
    M.set_schedule(gb.SCHED_ROW)
    M.set_schedule(gb.SCHED_ROW, f32=True)
    S = gb.CgSolver(M, mode)
    b = torch.from_numpy(W.rhs(A.nrows, 1)).cuda()
    S.solve(b, tol=1e-6, niter=5)
    M.set_schedule(gb.SCHED_MERGE, f32=f32)
    with pytest.raises(gb.GooseberryError):
        S.solve(b, tol=1e-6, niter=5)
    M.set_schedule(gb.SCHED_ROW, f32=f32)
    _, r = S.solve(b, tol=1e-6, niter=5)
    assert r.iterations == 5
