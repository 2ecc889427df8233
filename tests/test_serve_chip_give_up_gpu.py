"""Server requests whose solve on the chip is given up: the batch solves them, and
a slot is as new for its next request."""
from __future__ import annotations

import time

import numpy as np
import pytest

import gooseberry_b200 as gb
from gooseberry_b200 import workloads as W

pytestmark = pytest.mark.gpu

MODES = [gb.CG_F64, gb.CG_MIXED]


def check(A, b, r):
    assert r.status == "converged", r
    assert np.linalg.norm(b - A.to_scipy() @ r.x) <= 2e-9 * np.linalg.norm(b)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("fault", [gb.CHIP_FAULT_MISSING, gb.CHIP_FAULT_LATE])
def test_the_batch_takes_over(mode, fault):
    srv = gb.Server(pool_bytes=1 << 28, max_slots=3, mode=mode)
    reqs = [(k, W.diffusion_2d(s, k), W.rhs(s * s, k)) for k, s in enumerate((20, 80, 120, 90))]
    srv.set_chip_fault(fault, 20)
    for k, A, b in reqs:
        srv.submit(k, A, b, tol=1e-9, niter=20_000)
    res = {r.id: r for r in srv.drain()}
    for k, A, b in reqs:
        check(A, b, res[k])
    srv.close()


@pytest.mark.parametrize("mode", MODES)
def test_slot_of_a_cancelled_and_given_up_solve(mode):
    """The next request of the slot is not cancelled."""
    srv = gb.Server(pool_bytes=1 << 28, max_slots=1, mode=mode)
    A = W.diffusion_2d(100, 1)
    b = W.rhs(A.nrows, 1)
    srv.set_chip_fault(gb.CHIP_FAULT_MISSING, 100)
    x = np.full(A.nrows, 3.0)
    srv.submit(0, A, b, tol=1e-9, niter=20_000, x_out=x)
    srv.step()  # admitted and launched
    srv.cancel(0)
    srv.set_chip_fault(gb.CHIP_FAULT_NONE)
    t0 = time.time()
    res = []
    while not res and time.time() - t0 < 30:
        srv.step()
        res = srv.poll()
    assert res[0].status == "cancelled" and np.all(x == 3.0)
    srv.submit(1, A, b, tol=1e-9, niter=20_000)
    check(A, b, srv.drain()[0])
    srv.close()
