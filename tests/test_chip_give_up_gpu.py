"""Waits inside a solve on the chip that run out: one CTA is missing or late, the
others give up and leave, and the graph-replayed kernels run the solve."""
from __future__ import annotations

import pytest

import gooseberry_b200 as gb
from gooseberry_b200 import workloads as W

pytestmark = pytest.mark.gpu

MATRICES = {
    # the neighbours' r fetched ahead, by warps that wait beside the sum
    "fetched_ahead": lambda: W.diffusion((200, 190), 5, 0.5, 2.0),
    # a band so wide that every warp fetches them at the iteration's start
    "wide_band": lambda: W.diffusion((200, 5000), 6, 0.5, 2.0),
}


@pytest.mark.parametrize("mode", [gb.CG_F64, gb.CG_MIXED])
@pytest.mark.parametrize("name", sorted(MATRICES))
def test_waits_run_out(name, mode):
    import torch
    A = MATRICES[name]()
    M = gb.CsrMatrix.from_host(A, f64=True, f32=True)
    M.set_schedule(gb.SCHED_ROW)
    M.set_schedule(gb.SCHED_ROW, f32=True)
    S = gb.CgSolver(M, mode)
    b = torch.from_numpy(W.rhs(A.nrows, 3)).cuda()
    x, r = S.solve(b, tol=1e-30, niter=70)
    on_chip = r.kernel_launches
    assert on_chip <= 2, r
    for fault in (gb.CHIP_FAULT_MISSING, gb.CHIP_FAULT_LATE, gb.CHIP_FAULT_MISSING):
        S.set_chip_fault(fault, 20)
        y, q = S.solve(b, tol=1e-30, niter=70)
        assert q.status == r.status == "maxiter" and q.iterations == 70
        assert q.kernel_launches > on_chip, (fault, q)
        # (mixed: FP32 iterations against FP64 ones, not converged)
        assert float((y - x).norm() / x.norm()) <= (1e-9 if mode == gb.CG_F64 else 1e-2)
    S.set_chip_fault(gb.CHIP_FAULT_NONE)
    y, q = S.solve(b, tol=1e-30, niter=70)
    assert q.kernel_launches == on_chip and torch.equal(x, y)


def test_refused():
    M = gb.CsrMatrix.from_host(W.laplacian_2d(20), f64=True, f32=True)
    with pytest.raises(gb.GooseberryError):  # one CTA waits for nobody
        gb.CgSolver(M).set_chip_fault(gb.CHIP_FAULT_MISSING, 20)
    M.set_schedule(gb.SCHED_MERGE)
    with pytest.raises(gb.GooseberryError):
        gb.CgSolver(M).set_chip_fault(gb.CHIP_FAULT_LATE, 20)
