"""SpMV over row classes and row patterns (the autotuner's compressed forms of
the row schedule): the same bits as the row schedule over the CSR arrays."""
from __future__ import annotations

import numpy as np
import pytest

import gooseberry_b200 as gb
from gooseberry_b200 import workloads as W

pytestmark = pytest.mark.gpu


def rectangular(n, m, seed):
    """n x m, rows of 0 to 7 entries at a few offsets from the diagonal."""
    rng = np.random.default_rng(seed)
    lists = [[], [0], [0, 1], [-2, 0, 3], [-7, -1, 0, 1, 7], [-9, -3, -1, 0, 1, 3, 9]]
    pick = rng.integers(0, len(lists), n)
    rows, cols = [], []
    for i in range(n):
        for d in lists[pick[i]]:
            if 0 <= i + d < m:
                rows.append(i)
                cols.append(i + d)
    rp = np.zeros(n + 1, np.int64)
    np.add.at(rp, np.asarray(rows, np.int64) + 1, 1)
    return W.Csr(n, m, np.cumsum(rp).astype(np.uint32), np.asarray(cols, np.uint32),
                 rng.uniform(-1, 1, len(cols)))


CASES = {
    "classes2d": lambda: W.laplacian_2d(1500),
    "classes3d": lambda: W.diffusion((110, 120, 100), 1, 1.0, 1.0),
    "patterns2d": lambda: W.diffusion((1300, 1100), 2, 0.1, 10.0),
    "patterns3d": lambda: W.diffusion((110, 100, 120), 3, 0.1, 10.0),
    "small": lambda: W.laplacian_2d(7),
    "one_row": lambda: W.diffusion((1,), 1, 1.0, 1.0),
    "tall": lambda: rectangular(50_001, 49_000, 4),
    "wide": lambda: rectangular(30_011, 60_000, 5),
}


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_autotuned_pattern_matrix_has_the_row_schedules_bits(name, f32):
    import torch
    A = CASES[name]()
    M = gb.CsrMatrix.from_host(A, f64=not f32, f32=f32)
    dt = torch.float32 if f32 else torch.float64
    x = torch.from_numpy(W.dense_x(A.ncols, 6)).cuda().to(dt)
    M.set_schedule(gb.SCHED_ROW, f32=f32)
    want = M.spmv(x)
    for _ in range(2):  # timed, then from the cache
        M.autotune(f32=f32)
        got = M.spmv(x)
        info = M.info()
        if (info.schedule_f32 if f32 else info.schedule) == gb.SCHED_ROW:
            assert torch.equal(got, want)
        else:  # another schedule won: its sums are reordered
            eps = 64 * 2.0 ** (-24 if f32 else -53)
            bound = A.to_scipy().__abs__() @ np.abs(x.cpu().numpy().astype(np.float64))
            assert np.all(np.abs((got - want).cpu().numpy()) <= eps * bound + 1e-300)
    M.set_schedule(gb.SCHED_ROW, f32=f32)  # drops the compressed form
    assert torch.equal(M.spmv(x), want)
