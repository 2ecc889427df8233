"""The batch and the caller beside a solve on the chip that needs nearly every SM:
the batch's requests end long before it, and steps return."""
from __future__ import annotations

import time

import numpy as np
import pytest

import gooseberry_b200 as gb
from gooseberry_b200 import workloads as W
from test_serve_chip_gpu import nine_point

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [gb.CG_F64, gb.CG_MIXED])
@pytest.mark.parametrize("n", [454_000, 250_000])  # every SM; 82 of them
def test_batch_beside_a_long_solve(mode, n):
    srv = gb.Server(pool_bytes=1 << 30, max_slots=8, mode=mode)
    small = nine_point(40)
    b = W.rhs(small.nrows, 2)
    srv.submit(5, small, b, tol=1e-9, niter=20_000)  # tunes and loads the batch's kernels
    assert srv.drain()[0].status == "converged"
    A = W.diffusion((n,), 3, 0.5, 2.0)  # converges in about n iterations
    x = np.full(A.nrows, 3.0)
    srv.submit(0, A, W.rhs(A.nrows, 1), tol=1e-300, niter=400_000, x_out=x)
    srv.step()
    for k in (1, 2):
        srv.submit(k, small, b, tol=1e-9, niter=20_000)
    t0, longest, res = time.time(), 0.0, []
    while len(res) < 2 and time.time() - t0 < 20:
        t1 = time.time()
        srv.step()
        longest = max(longest, time.time() - t1)
        res += srv.poll()
    took = time.time() - t0
    srv.cancel(0)
    t1 = time.time()
    while len(res) < 3 and time.time() - t1 < 20:
        srv.step()
        res += srv.poll()
    assert time.time() - t1 < 0.5
    by = {r.id: r for r in res}
    assert by[0].status == "cancelled" and by[0].iterations > 0 and np.all(x == 3.0)
    for k in (1, 2):
        assert by[k].status == "converged"
        assert np.linalg.norm(b - small.to_scipy() @ by[k].x) <= 2e-9 * np.linalg.norm(b)
    assert took < 1.0 and longest < 0.25, (took, longest)
    srv.close()
