"""The CG solve that keeps its vectors on the chip (pattern matrices whose
vectors fit the SMs), at the sizes where its partition changes -- one CTA, a
last CTA of one row, each rows-per-thread form, the largest system, the first
one past it -- and on each form in which it holds the matrix: whole-row
classes, values in shared memory or in L2 (doubles, exact floats), value
codes, the plain CSR arrays."""
from __future__ import annotations

import numpy as np
import pytest

import gooseberry_b200 as gb
from gooseberry_b200 import workloads as W

pytestmark = pytest.mark.gpu


def line(n, seed=3):
    return W.diffusion((n,), seed, 0.5, 2.0)


def quantised(shape, seed):
    """A stencil with integer coefficients 1..6: few values, many distinct rows."""
    A = W.diffusion(shape, seed, 1.0, 6.9)
    v = np.where(A.rowval < 0, np.ceil(A.rowval), 0.0)  # -1 .. -6
    rows = np.repeat(np.arange(A.nrows), A.row_lengths())
    diag = np.full(A.nrows, 1.0)
    np.add.at(diag, rows, -v)
    v = np.where(A.rowval > 0, diag[rows], v)
    return W.Csr(A.nrows, A.ncols, A.rowptr, A.rowind, v)


def float_exact(A):
    return W.Csr(A.nrows, A.ncols, A.rowptr, A.rowind,
                 A.rowval.astype(np.float32).astype(np.float64))


CASES = {  # name: (matrix, solved in one launch)
    **{f"line{n}": (lambda n=n: line(n), True)
       for n in (1, 2, 33, 511, 513, 4096, 4097, 148 * 512, 148 * 512 + 1, 148 * 2048 + 1,
                 148 * 4096, 148 * 4096 + 1, 148 * 7296)},
    "line_past_the_chip": (lambda: line(148 * 7296 + 1), False),
    "class2d": (lambda: W.laplacian_2d(1024), True),
    "class3d": (lambda: W.diffusion((40, 40, 40), 1, 1.0, 1.0), True),
    "codes2d": (lambda: quantised((200, 190), 5), True),
    "codes3d": (lambda: quantised((30, 31, 32), 6), True),
    "smem2d": (lambda: W.diffusion((333, 517), 7, 0.1, 10.0), True),
    "smem3d": (lambda: W.diffusion((41, 37, 45), 8, 0.1, 10.0), True),
    "smem2d_f32": (lambda: float_exact(W.diffusion((211, 300), 9, 0.1, 10.0)), True),
    "smem3d_f32": (lambda: float_exact(W.diffusion((33, 35, 36), 9, 0.1, 10.0)), True),
    "global2d": (lambda: W.diffusion((1000, 1001), 10, 0.1, 10.0), True),
    "global2d_f32": (lambda: float_exact(W.diffusion((1000, 1000), 11, 0.1, 10.0)), True),
    "global3d": (lambda: W.diffusion((80, 80, 80), 12, 0.1, 10.0), True),
    "global3d_f32": (lambda: float_exact(W.diffusion((80, 81, 79), 13, 0.1, 10.0)), True),
    "halo_past_the_chip": (lambda: W.diffusion((100, 100, 100), 14, 1.0, 1.0), False),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_solve_on_the_chip(name):
    """The first 30 iterations against the oracle's (each recurrence step
    rounds differently by a few ulp, amplified at most by the iteration count
    and the vectors' spread: 1e-10 relative leaves three digits), against the
    solver over the plain CSR arrays bit for bit, and against itself."""
    import oracle
    import torch
    build, one_launch = CASES[name]
    A = build()
    b = W.rhs(A.nrows, 21)
    bd = torch.from_numpy(b).cuda()
    M = gb.CsrMatrix.from_host(A)
    M.set_schedule(gb.SCHED_ROW)
    S = gb.CgSolver(M)
    P = gb.CgSolver(M, plain_entries=True)
    x1, r1, h1 = S.solve(bd, tol=1e-12, niter=30, history=True)
    x2, r2 = P.solve(bd, tol=1e-12, niter=30)
    x3, r3 = S.solve(bd, tol=1e-12, niter=30)
    assert (r1.kernel_launches == 1) == one_launch, r1
    for x, r in ((x2, r2), (x3, r3)):
        assert torch.equal(x1, x) and r.rnorm == r1.rnorm
        assert (r.iterations, r.status) == (r1.iterations, r1.status)
    assert len(h1) == r1.iterations and h1[-1] == r1.rnorm
    xo, ito, hist = oracle.cgd(A.rowptr, A.rowind, A.rowval, b, 1e-12 * np.linalg.norm(b), 30)
    assert abs(r1.iterations - ito) <= 1, (r1.iterations, ito)
    xs = x1.cpu().numpy()
    if A.nrows > 60 and r1.iterations == ito == 30:
        assert np.linalg.norm(xs - xo) <= 1e-10 * np.linalg.norm(xo)
    else:  # the Krylov space is all but exhausted: iterates depend on the last bits
        res = np.linalg.norm(b - A.to_scipy() @ xs)
        assert abs(res - r1.rnorm) <= 1e-12 * np.linalg.norm(b)
    S.close()
    P.close()
    M.close()


def test_right_hand_side_as_solution_vector():
    """x may be the array of b."""
    import torch
    A = W.laplacian_2d(150)
    b = torch.from_numpy(W.rhs(A.nrows, 22)).cuda()
    S = gb.CgSolver(gb.CsrMatrix.from_host(A))
    x, r = S.solve(b, tol=1e-9)
    y = b.clone()
    S.solve(y, y, tol=1e-9)
    assert r.status == "converged" and torch.equal(x, y)


def test_threads_share_the_chip():
    """Solves of several threads and sizes at once: each waits for the SMs it
    needs, and gives the bits it gives alone."""
    import threading

    import torch
    jobs = []
    for k, side in enumerate((60, 150, 400, 700, 1000, 90)):
        A = W.laplacian_2d(side)
        b = torch.from_numpy(W.rhs(A.nrows, 30 + k)).cuda()
        S = gb.CgSolver(gb.CsrMatrix.from_host(A))
        jobs.append((S, b, S.solve(b, tol=1e-6)[0].clone()))
    torch.cuda.synchronize()
    got = [None] * len(jobs)

    def work(i):
        S, b, _ = jobs[i]
        st = torch.cuda.Stream()
        for _ in range(5):
            got[i] = S.solve(b, torch.empty_like(b), tol=1e-6, stream=st)[0]

    ts = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    for (_, _, want), x in zip(jobs, got):
        assert torch.equal(want, x)


def test_scale_changes_between_iterations():
    """Residual norms that fall by many orders in one iteration, and tiny or
    huge right-hand sides, keep the accuracy of the sums: the solution scales
    with b by an exact power of two."""
    import torch
    A = line(9000, 5)
    A.rowval[:] = np.where(A.rowval > 0, 4.0, -1e-9)  # nearly 4 I: rr falls by 1e19 a step
    M = gb.CsrMatrix.from_host(A)
    S = gb.CgSolver(M)
    b = torch.from_numpy(W.rhs(A.nrows, 40)).cuda()
    x, r = S.solve(b, tol=1e-14)
    assert r.status == "converged" and r.iterations <= 4
    y = M.spmv(x)
    assert float((b - y).norm() / b.norm()) <= 1e-14
    for e in (-400, 400):  # every r.r stays normal
        xe, re = S.solve(b * 2.0 ** e, tol=1e-14)
        assert re.iterations == r.iterations
        assert torch.equal(xe, x * 2.0 ** e)
