"""A solve on the chip of several launches: the same bits as one launch gives, in
every form of the matrix; other streams' kernels run between the launches."""
from __future__ import annotations

import threading
import time

import numpy as np
import pytest

import gooseberry_b200 as gb
from gooseberry_b200 import workloads as W
from test_cg_resident_gpu import CASES

pytestmark = pytest.mark.gpu

NAMES = ["line33", "line513", "line4097", "line75777", "class2d", "class3d", "codes2d", "smem2d",
         "smem3d_f32", "global2d", "global3d"]


def solver(A, mode=gb.CG_F64):
    M = gb.CsrMatrix.from_host(A, f64=True, f32=True)
    M.set_schedule(gb.SCHED_ROW)
    M.set_schedule(gb.SCHED_ROW, f32=True)
    return gb.CgSolver(M, mode)


@pytest.mark.parametrize("name", NAMES)
def test_same_bits(name):
    import torch
    A = CASES[name][0]()
    b = torch.from_numpy(W.rhs(A.nrows, 21)).cuda()
    S = solver(A)
    for niter in (64, 65, 300):
        x, r, h = S.solve(b, tol=1e-300, niter=niter, history=True)
        if A.nrows > 2048:  # (fewer rows are one CTA's)
            S.set_chip_fault(gb.CHIP_FAULT_SHORT)
        y, q, g = S.solve(b, tol=1e-300, niter=niter, history=True)
        if A.nrows > 2048:
            S.set_chip_fault(gb.CHIP_FAULT_NONE)
            assert q.kernel_launches >= 1 + (r.iterations - 2) // 64, q
        assert torch.equal(x, y) and np.array_equal(h, g)
        assert (q.iterations, q.status, q.rnorm, q.bnorm) == \
            (r.iterations, r.status, r.rnorm, r.bnorm)


def test_wide_band_and_refinement():
    """x and the neighbours' values not in shared memory; mixed mode."""
    import torch
    for A, mode in ((W.diffusion((200, 5000), 6, 0.5, 2.0), gb.CG_F64),
                    (W.diffusion_2d(150, 3), gb.CG_MIXED)):
        b = torch.from_numpy(W.rhs(A.nrows, 4)).cuda()
        S = solver(A, mode)
        x, r = S.solve(b, tol=1e-13, niter=1500)
        S.set_chip_fault(gb.CHIP_FAULT_SHORT)
        y, q = S.solve(b, tol=1e-13, niter=1500)
        assert torch.equal(x, y) and q.kernel_launches > r.kernel_launches
        assert (q.iterations, q.refinements, q.status) == (r.iterations, r.refinements, r.status)


@pytest.mark.parametrize("mode", [gb.CG_F64, gb.CG_MIXED])
def test_server(mode):
    mats = [W.diffusion_2d(s, s) for s in (20, 50, 130, 300)] + [W.diffusion((3000,), 1, 0.5, 2.0)]
    got = []
    for fault in (gb.CHIP_FAULT_NONE, gb.CHIP_FAULT_SHORT):
        srv = gb.Server(pool_bytes=1 << 28, max_slots=4, mode=mode)
        srv.set_chip_fault(fault)
        for k, A in enumerate(mats):
            srv.submit(k, A, W.rhs(A.nrows, k), tol=1e-13, niter=2000)
        got.append({r.id: r for r in srv.drain()})
        srv.close()
    for k in range(len(mats)):
        p, q = got[0][k], got[1][k]
        assert (p.iterations, p.refinements, p.status, p.rnorm, p.bnorm) == \
            (q.iterations, q.refinements, q.status, q.rnorm, q.bnorm)
        assert np.array_equal(p.x, q.x)


def test_cancelled_between_launches():
    import torch
    A = W.laplacian_2d(700)
    bh = W.rhs(A.nrows, 5)
    b = torch.from_numpy(bh).cuda()
    S = solver(A)
    got = []
    t = threading.Thread(target=lambda: got.append(S.solve(b, tol=1e-300, niter=10 ** 7)))
    t.start()
    time.sleep(0.05)
    S.cancel()
    t.join(20)
    x, r = got[0]
    assert r.status == "cancelled" and 0 < r.iterations < 10 ** 6
    y, q = S.solve(b, tol=1e-300, niter=r.iterations)
    assert torch.equal(x, y) and q.rnorm == r.rnorm


def test_other_streams_get_their_turn():
    """Kernels of another stream do not wait for the end of a solve that holds
    every SM."""
    import torch
    A = W.diffusion((1_000_000,), 3, 0.5, 2.0)  # converges in about as many iterations
    b = torch.from_numpy(W.rhs(A.nrows, 6)).cuda()
    S = solver(A)
    v = torch.ones(512, 512, dtype=torch.float64, device="cuda")
    v @ v  # (a kernel too large for what the solve leaves of an SM)
    S.solve(b, tol=1e-300, niter=100)
    torch.cuda.synchronize()
    st, mine = torch.cuda.Stream(), torch.cuda.Stream()
    got = []
    t0 = time.time()
    t = threading.Thread(target=lambda: got.append(
        S.solve(b, torch.empty_like(b), tol=1e-300, niter=200_000, stream=st)))
    t.start()
    time.sleep(0.2)
    waits = []
    for _ in range(5):
        t1 = time.time()
        with torch.cuda.stream(mine):
            v @ v
        mine.synchronize()
        waits.append(time.time() - t1)
        assert t.is_alive()
        time.sleep(0.01)
    t.join(60)
    assert got[0][1].iterations == 200_000 and time.time() - t0 > 1.0
    assert max(waits) < 0.2, waits
