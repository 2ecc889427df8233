"""The autotuner's cached choice and the compressed forms: matrices of one shape
with whole rows, offset lists or nothing that repeats are each timed, whichever
is tuned first.  And the compressed forms themselves, taken without timing."""
from __future__ import annotations

import numpy as np
import pytest

import gooseberry_b200 as gb
from gooseberry_b200 import workloads as W
from test_spmv_pattern_gpu import CASES

pytestmark = pytest.mark.gpu


def columns_shuffled(A, seed):
    """The same row lengths; no list of offsets repeats."""
    p = np.random.default_rng(seed).permutation(A.nrows).astype(np.uint32)
    ind = p[A.rowind]
    for i in range(2, int(A.row_lengths().max()) + 1):  # columns ascending in every row
        rows = np.flatnonzero(A.row_lengths() == i)
        at = A.rowptr[rows][:, None] + np.arange(i)
        ind[at] = np.sort(ind[at], axis=1)
    return W.Csr(A.nrows, A.ncols, A.rowptr, ind, A.rowval)


# one shape for each order: the choice is cached for the process
@pytest.mark.parametrize("side,order", [(3001, "scrambled classes patterns"),
                                        (1601, "classes scrambled patterns"),
                                        (2203, "patterns scrambled classes")])
def test_order_of_tuning(side, order):
    import torch
    made = {}
    for kind in order.split():
        A = (W.laplacian_2d(side) if kind == "classes"
             else W.diffusion((side, side), 2, 0.5, 2.0) if kind == "patterns"
             else columns_shuffled(W.laplacian_2d(side), 3))
        M = gb.CsrMatrix.from_host(A)
        M.autotune()
        made[kind] = (A, M)
    # (2.7 and 1.3 times the row schedule's speed at these sizes)
    assert made["classes"][1].row_form() == gb.ROWS_CLASSES
    assert made["patterns"][1].row_form() == gb.ROWS_PATTERNS
    assert made["scrambled"][1].row_form() == gb.ROWS_PLAIN
    for A, M in made.values():
        x = torch.from_numpy(W.dense_x(A.ncols, 6)).cuda()
        y = M.spmv(x).cpu().numpy()
        want = A.to_scipy() @ x.cpu().numpy()
        bound = abs(A.to_scipy()) @ np.abs(x.cpu().numpy())
        assert np.all(np.abs(y - want) <= 16 * 2.0 ** -53 * bound)


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_compressed_forms_have_the_row_schedules_bits(name, f32):
    import torch
    A = CASES[name]()
    M = gb.CsrMatrix.from_host(A, f64=not f32, f32=f32)
    x = torch.from_numpy(W.dense_x(A.ncols, 6)).cuda().to(
        torch.float32 if f32 else torch.float64)
    M.set_schedule(gb.SCHED_ROW, f32=f32)
    assert M.row_form(f32) == gb.ROWS_PLAIN
    want = M.spmv(x)
    M.compress_rows(f32)
    classes = name in ("classes2d", "classes3d", "small", "one_row")
    assert M.row_form(f32) == (gb.ROWS_CLASSES if classes else gb.ROWS_PATTERNS)
    got = torch.full_like(want, 7.0)  # (empty rows are written too)
    M.spmv(x, got)
    assert torch.equal(got, want)


def test_no_form():
    A = columns_shuffled(W.laplacian_2d(50), 1)
    M = gb.CsrMatrix.from_host(A)
    M.set_schedule(gb.SCHED_MERGE)
    with pytest.raises(gb.GooseberryError):
        M.compress_rows()
    assert M.info().schedule == gb.SCHED_MERGE and M.row_form() == gb.ROWS_PLAIN
