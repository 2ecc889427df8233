"""A solve cancelled while it waits for SMs that a server's solve holds: the norm
it reports is that of b - A x for the x it returns."""
from __future__ import annotations

import threading
import time

import numpy as np
import pytest

import gooseberry_b200 as gb
from gooseberry_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [gb.CG_F64, gb.CG_MIXED])
def test_norm_of_a_cancelled_solve(mode):
    import torch
    A = W.diffusion_2d(400, 12)
    bh = W.rhs(A.nrows, 2)
    b = torch.from_numpy(bh).cuda()
    M = gb.CsrMatrix.from_host(A, f64=True, f32=True)
    M.set_schedule(gb.SCHED_ROW)
    S = gb.CgSolver(M, mode)
    S.solve(b, tol=1e-3)
    srv = gb.Server(pool_bytes=1 << 29, max_slots=2, mode=gb.CG_F64)
    srv.submit(0, A, bh, tol=1e-300, niter=300_000)
    srv.step()
    got = []
    t = threading.Thread(target=lambda: got.append(S.solve(b, tol=1e-300, niter=10 ** 7)))
    t.start()
    time.sleep(0.3)
    S.cancel()
    # (the server's solve ends by itself, and a step gives its SMs back)
    t0 = time.time()
    while t.is_alive() and time.time() - t0 < 60:
        srv.step()
    t.join(1)
    x, r = got[0]
    assert r.status == "cancelled"
    true = np.linalg.norm(bh - A.to_scipy() @ x.cpu().numpy())
    # (past the attainable accuracy the recurrence's norm goes on falling)
    assert r.bnorm == pytest.approx(np.linalg.norm(bh), rel=1e-12)
    assert r.rnorm == pytest.approx(true, rel=1e-6) or true <= 1e-9 * r.bnorm
    assert r.rnorm > 0.0
    srv.close()
