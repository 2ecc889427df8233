"""Stencil systems that fit the chip, solved off it: the graph-replayed kernels over
every layout of the entries, the FP32 iterations of mixed mode and the server's
batch, which larger systems and solves that are given up take."""
from __future__ import annotations

import numpy as np
import pytest

import gooseberry_b200 as gb
from gooseberry_b200 import workloads as W
from test_cg_codec_gpu import CASES, banded

pytestmark = pytest.mark.gpu

PATTERN_CASES = [n for n in sorted(CASES) if CASES[n][1] == 0]


def row_matrix(A):
    M = gb.CsrMatrix.from_host(A, f64=True, f32=True)
    M.set_schedule(gb.SCHED_ROW)
    M.set_schedule(gb.SCHED_ROW, f32=True)
    return M


@pytest.mark.parametrize("name", PATTERN_CASES)
def test_layouts_are_bit_identical(name):
    import torch
    build, entry, row = CASES[name]
    A = build()
    M = row_matrix(A)
    S = gb.CgSolver(M, on_chip=False)
    P = gb.CgSolver(M, plain_entries=True, on_chip=False)
    chip = gb.CgSolver(M)
    assert (S.entry_bytes(), S.row_bytes()) == (entry, row)
    b = torch.from_numpy(W.rhs(A.nrows, 9)).cuda()
    for tol, niter in ((1e-10, 0), (1e-30, 25)):
        x1, r1 = S.solve(b, tol=tol, niter=niter)
        x2, r2 = P.solve(b, tol=tol, niter=niter)
        x3, r3 = chip.solve(b, tol=tol, niter=niter)
        assert r1.kernel_launches > r1.iterations and r2.kernel_launches > r2.iterations
        assert r3.kernel_launches < r3.iterations  # which path each took
        assert (r1.iterations, r1.status, r1.rnorm) == (r2.iterations, r2.status, r2.rnorm)
        assert torch.equal(x1, x2)
        assert abs(r1.iterations - r3.iterations) <= 1 + r1.iterations // 50
        assert float((x1 - x3).norm() / x1.norm()) <= 1e-7  # both to tol, or 25 iterations


@pytest.mark.parametrize("name", ["diffusion3d", "diffusion2d", "band"])
def test_mixed_columns_are_bit_identical(name):
    import torch
    A = {"diffusion3d": lambda: W.diffusion_3d(24, seed=11),
         "diffusion2d": lambda: W.diffusion_2d(70, seed=12),
         "band": lambda: banded(5000, [-200, -3, -1, 0, 1, 3, 200], 8)}[name]()
    M = row_matrix(A)
    S = gb.CgSolver(M, gb.CG_MIXED, on_chip=False)
    P = gb.CgSolver(M, gb.CG_MIXED, plain_entries=True, on_chip=False)
    assert (S.entry_bytes(), S.row_bytes()) == (0, 33) and P.entry_bytes() == 8
    b = torch.from_numpy(W.rhs(A.nrows, 12)).cuda()
    x1, r1 = S.solve(b, tol=1e-10)
    x2, r2 = P.solve(b, tol=1e-10)
    assert r1.status == r2.status == "converged" and r1.kernel_launches > r1.iterations
    assert (r1.iterations, r1.refinements) == (r2.iterations, r2.refinements)
    assert torch.equal(x1, x2)


@pytest.mark.parametrize("make", [lambda: W.diffusion_3d(24, seed=31),
                                  lambda: W.diffusion_2d(96, seed=32),
                                  lambda: W.laplacian_2d(128)])
def test_mixed_reaches_fp64_accuracy(make):
    import torch
    A = make()
    b = W.rhs(A.nrows, 33)
    bd = torch.from_numpy(b).cuda()
    M = row_matrix(A)
    x64, r64 = gb.CgSolver(M, on_chip=False).solve(bd, tol=1e-10, niter=20000)
    xm, rm = gb.CgSolver(M, gb.CG_MIXED, on_chip=False).solve(bd, tol=1e-10, niter=20000)
    assert r64.status == rm.status == "converged" and rm.refinements >= 1
    assert rm.kernel_launches > rm.iterations and r64.kernel_launches > r64.iterations
    res = np.linalg.norm(b - A.to_scipy() @ xm.cpu().numpy()) / np.linalg.norm(b)
    assert res <= 1.05e-10 and rm.rnorm == pytest.approx(res * np.linalg.norm(b), rel=1e-3)
    assert rm.iterations <= 1.25 * r64.iterations + 10
    assert float((xm - x64).norm() / x64.norm()) <= 1e-6


@pytest.mark.parametrize("mode", [gb.CG_F64, gb.CG_MIXED])
def test_batch_takes_stencils(mode):
    """Uneven stencil requests through fewer slots, each with the bits it has alone."""
    mats = [W.laplacian_2d(45), W.diffusion_2d(46, 2), W.diffusion_2d(120, 3),
            W.diffusion((22, 21, 20), 5, 0.1, 10.0), W.diffusion_2d(150, 9), W.laplacian_2d(7)]
    reqs = [(k, A, W.rhs(A.nrows, 60 + k)) for k, A in enumerate(mats)]
    srv = gb.Server(pool_bytes=1 << 28, max_slots=4, mode=mode, on_chip=False)
    for k, A, b in reqs:
        srv.submit(k, A, b, tol=1e-10, niter=50_000)
    res = {r.id: r for r in srv.drain()}
    steps = srv.stats()["steps"]
    assert steps >= max(r.iterations for r in res.values()) // 16  # replays of 16 iterations
    srv.close()
    for k, A, b in reqs:
        r = res[k]
        assert r.status == "converged"
        assert np.linalg.norm(b - A.to_scipy() @ r.x) <= 2e-10 * np.linalg.norm(b)
        alone = gb.Server(pool_bytes=1 << 27, max_slots=1, mode=mode, on_chip=False)
        alone.submit(k, A, b, tol=1e-10, niter=50_000)
        r1 = alone.drain()[0]
        assert r1.iterations == r.iterations and np.array_equal(r1.x, r.x)
        alone.close()
