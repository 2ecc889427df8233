"""The mixed solver over symmetric diagonals (stencils past the chip and L2):
the same iterates as over the plain columns, for two and three distances above
the diagonal, and on a matrix whose values are not symmetric, which keeps the
rows of 8."""
from __future__ import annotations

import numpy as np
import pytest

import gooseberry_b200 as gb
from gooseberry_b200 import workloads as W

pytestmark = pytest.mark.gpu


def unsymmetric(A):
    v = A.rowval.copy()
    v[1] *= 1.0 + 1e-3  # one entry above the diagonal
    return W.Csr(A.nrows, A.ncols, A.rowptr, A.rowind, v)


CASES = {
    "3d": (lambda: W.diffusion((137, 133, 131), 3, 0.1, 10.0), 16),
    "2d": (lambda: W.diffusion((1601, 1499), 4, 0.1, 10.0), 12),
    "unsymmetric": (lambda: unsymmetric(W.diffusion((1601, 1499), 4, 0.1, 10.0)), 33),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_diagonals_give_the_plain_iterates(name):
    import torch
    build, want = CASES[name]
    A = build()
    M = gb.CsrMatrix.from_host(A, f64=True, f32=True)
    S = gb.CgSolver(M, gb.CG_MIXED)
    P = gb.CgSolver(M, gb.CG_MIXED, plain_entries=True)
    assert (S.entry_bytes(), S.row_bytes()) == (0, want)
    b = torch.from_numpy(W.rhs(A.nrows, 12)).cuda()
    x1, r1, h1 = S.solve(b, tol=1e-12, niter=90, history=True)
    x2, r2, h2 = P.solve(b, tol=1e-12, niter=90, history=True)
    assert (r1.iterations, r1.refinements, r1.status) == (r2.iterations, r2.refinements, r2.status)
    assert torch.equal(x1, x2) and np.array_equal(h1, h2)
    res = float((b - M.spmv(x1)).norm())
    assert r1.rnorm == pytest.approx(res, rel=1e-6)
    S.close()
    P.close()
    M.close()
