"""Launches on the chip that the driver turns down (a fake of its error code): the
graph path, or the server's batch, solves the system."""
from __future__ import annotations

import numpy as np
import pytest

import gooseberry_b200 as gb
from gooseberry_b200 import workloads as W

pytestmark = pytest.mark.gpu

MODES = [gb.CG_F64, gb.CG_MIXED]


def check(A, b, x):
    assert np.linalg.norm(b - A.to_scipy() @ x) <= 2e-9 * np.linalg.norm(b)


@pytest.mark.parametrize("mode", MODES)
def test_solver(mode):
    import torch
    A = W.diffusion_2d(150, 4)
    b = W.rhs(A.nrows, 4)
    M = gb.CsrMatrix.from_host(A, f64=True, f32=True)
    M.set_schedule(gb.SCHED_ROW)
    M.set_schedule(gb.SCHED_ROW, f32=True)
    S = gb.CgSolver(M, mode)
    bd = torch.from_numpy(b).cuda()
    x, r = S.solve(bd, tol=1e-9)
    S.set_chip_fault(gb.CHIP_FAULT_REFUSED)
    y, q = S.solve(bd, tol=1e-9)
    assert q.status == "converged" and q.kernel_launches > r.kernel_launches
    check(A, b, y.cpu().numpy())
    S.set_chip_fault(gb.CHIP_FAULT_NONE)
    z, _ = S.solve(bd, tol=1e-9)
    assert torch.equal(x, z)


@pytest.mark.parametrize("mode", MODES)
def test_server(mode):
    srv = gb.Server(pool_bytes=1 << 28, max_slots=2, mode=mode)
    srv.set_chip_fault(gb.CHIP_FAULT_REFUSED)
    reqs = [(k, W.diffusion_2d(s, k), W.rhs(s * s, k)) for k, s in enumerate((20, 90, 120))]
    for k, A, b in reqs:
        srv.submit(k, A, b, tol=1e-9, niter=20_000)
    res = {r.id: r for r in srv.drain(timeout_s=60)}
    for k, A, b in reqs:
        assert res[k].status == "converged"
        check(A, b, res[k].x)
    srv.close()
