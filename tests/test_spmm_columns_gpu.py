"""Fused SpMM over the column groups of its kernels: every k around a group of
four, rows of at most 5, 7 and more entries, and a result that is not 32-byte
aligned, each bit for bit one SpMV of the row schedule per column."""
from __future__ import annotations

import pytest

import gooseberry_b200 as gb
from gooseberry_b200 import workloads as W

pytestmark = pytest.mark.gpu

MATRICES = {
    "rows5": lambda: W.diffusion_2d(61, 3),
    "rows7": lambda: W.diffusion((13, 12, 11), 4, 0.1, 10.0),
    "rows10": lambda: W.uniform_rows(700, 10, 5),
}


@pytest.mark.parametrize("k", [2, 3, 4, 5, 7, 8, 9, 12, 16])
@pytest.mark.parametrize("name", sorted(MATRICES))
def test_columns_equal_spmv(name, k):
    import torch
    A = MATRICES[name]()
    M = gb.CsrMatrix.from_host(A)
    M.set_schedule(gb.SCHED_ROW)
    B = torch.from_numpy(W.dense_x(A.ncols * k, 7)).cuda()
    want = torch.stack([M.spmv(B[j * A.ncols:(j + 1) * A.ncols].contiguous())
                        for j in range(k)], 1).reshape(-1)
    assert torch.equal(M.spmm(B, k), want)
    room = torch.zeros(A.nrows * k + 1, dtype=torch.float64, device="cuda")
    M.spmm(B, k, out=room[1:])  # 8-byte aligned only
    assert torch.equal(room[1:], want) and room[0].item() == 0.0
