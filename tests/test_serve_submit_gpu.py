"""What gb_server_submit costs for requests that may be solved on the chip: looking
for their rows' patterns does not dominate it, however the patterns mix."""
from __future__ import annotations

import time

import numpy as np
import pytest

import gooseberry_b200 as gb
from gooseberry_b200 import workloads as W

pytestmark = pytest.mark.gpu


def mixed_rows(n, lists, seed):
    """A symmetric tridiagonal matrix whose rows also hold explicit zeros at one of
    `lists` pairs of distances: as many lists of offsets, in no order."""
    rng = np.random.default_rng(seed)
    d = 2 + rng.integers(0, lists, n)
    i = np.arange(n)
    cols = np.stack([i - d, i - 1, i, i + 1, i + d], 1)
    vals = np.broadcast_to(np.array([0.0, -1.0, 3.0, -1.0, 0.0]), cols.shape)
    keep = (cols >= 0) & (cols < n)
    keep[:, 0] &= keep[:, 4]  # (both or none: no more lists at the ends)
    keep[:, 4] &= keep[:, 0]
    rp = np.concatenate([[0], np.cumsum(keep.sum(1))])
    return W.Csr(n, n, rp.astype(np.uint32), cols[keep].astype(np.uint32), vals[keep].copy())


def best_submit_ms(srv, A, b):
    ts = []
    for k in range(6):
        t = time.perf_counter()
        srv.submit(k, A, b, tol=1e-9)
        ts.append(time.perf_counter() - t)
    for k in range(6):
        srv.cancel(k)
    srv.poll()
    return 1e3 * min(ts)


@pytest.mark.parametrize("n", [400_000, 460_000])  # fits the chip; its rows do not
def test_submit(n):
    A = mixed_rows(n, 200, 1)
    b = W.rhs(n, 2)
    got = []
    for on_chip in (False, True):
        srv = gb.Server(pool_bytes=4 << 30, max_slots=2, mode=gb.CG_F64, on_chip=on_chip)
        got.append(best_submit_ms(srv, A, b))
        srv.close()
    assert got[1] <= (3.0 if n == 400_000 else 1.3) * got[0] + 1.0, got


def test_patterns_in_no_order():
    """Solved on the chip with its 240 lists told apart; 300 go to the batch."""
    for lists in (240, 300):
        A = mixed_rows(60_000, lists, 3)
        b = W.rhs(A.nrows, 4)
        srv = gb.Server(pool_bytes=1 << 28, max_slots=2, mode=gb.CG_F64)
        srv.submit(0, A, b, tol=1e-12)
        r = srv.drain()[0]
        assert r.status == "converged"
        assert np.linalg.norm(b - A.to_scipy() @ r.x) <= 2e-12 * np.linalg.norm(b)
        srv.close()
