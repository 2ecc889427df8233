"""SMs that a server's solve on the chip held are free once its kernel has ended,
whether or not the server is stepped again; a wait for SMs has a limit."""
from __future__ import annotations

import os
import pathlib
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HEAD = """
import sys, time
import numpy as np, torch
import gooseberry_b200 as gb
from gooseberry_b200 import workloads as W
mode = int(sys.argv[1])
def system(side, seed):
    A = W.diffusion_2d(side, seed)
    return A, W.rhs(A.nrows, seed)
def solver(A):
    M = gb.CsrMatrix.from_host(A, f64=True, f32=True)
    M.set_schedule(gb.SCHED_ROW)
    M.set_schedule(gb.SCHED_ROW, f32=True)
    return gb.CgSolver(M, mode)
def server():
    return gb.Server(pool_bytes=1 << 29, max_slots=4, mode=mode)
def check(A, b, x, tol=2e-8):
    assert np.linalg.norm(b - A.to_scipy() @ x) <= tol * np.linalg.norm(b)
"""

THEN_SOLVE = HEAD + """
A, b = system(400, 1)
S, bd = solver(A), torch.from_numpy(b).cuda()
srv = server()
for k in range(3):
    srv.submit(k, A, b, tol=1e-8, niter=20_000)
srv.step()                      # launches what fits; nobody collects it
x, r = S.solve(bd, tol=1e-8)    # needs every SM
assert r.status == "converged" and r.kernel_launches <= 8, r
check(A, b, x.cpu().numpy())
xd, it, _ = gb.cgd(A.rowptr, A.rowind, A.rowval, b, 1e-8 * np.linalg.norm(b), 20_000)
check(A, b, xd)
for r in srv.drain():
    check(A, b, r.x)
srv.close()
"""

TWO_SERVERS = HEAD + """
A, b = system(500, 2)
first, second = server(), server()
first.submit(0, A, b, tol=1e-8, niter=20_000)
first.submit(1, A, b, tol=1e-8, niter=20_000)
first.step()
second.submit(2, A, b, tol=1e-8, niter=20_000)
second.submit(3, A, b, tol=1e-8, niter=20_000)
t = time.time()
got = second.drain(timeout_s=60)   # only this one is stepped
assert len(got) == 2 and time.time() - t < 30
got += first.drain(timeout_s=60)
assert sorted(r.id for r in got) == [0, 1, 2, 3]
for r in got:
    assert r.status == "converged"
    check(A, b, r.x)
first.close(); second.close()
"""

LIMIT = HEAD + """
# a server's solve that waits a second for a CTA that never starts holds its SMs
# for that long; others give up waiting for them after 50 ms
A, b = system(400, 3)
S, bd = solver(A), torch.from_numpy(b).cuda()
S.set_chip_fault(gb.CHIP_FAULT_MISSING, 20)  # loads the graph path's kernels
S.solve(bd, tol=1e-8)
S.set_chip_fault(gb.CHIP_FAULT_NONE, 50)
one, two = server(), server()
one.set_chip_fault(gb.CHIP_FAULT_MISSING, 1000)
one.submit(0, A, b, tol=1e-8, niter=20_000)
two.set_chip_fault(gb.CHIP_FAULT_NONE, 50)
two.submit(1, A, b, tol=1e-8, niter=20_000)
one.step()
t = time.time()
x, r = S.solve(bd, tol=1e-8)
assert r.status == "converged" and r.kernel_launches > 8, r
check(A, b, x.cpu().numpy())
assert time.time() - t < 0.9
got = two.drain(timeout_s=60)
one.set_chip_fault(gb.CHIP_FAULT_NONE)
got += one.drain(timeout_s=60)
assert len(got) == 2
for r in got:
    check(A, b, r.x)
one.close(); two.close()
x, r = S.solve(bd, tol=1e-8)
assert r.kernel_launches <= 8, r
"""


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("name", ["THEN_SOLVE", "TWO_SERVERS", "LIMIT"])
def test_in_one_thread(name, mode):
    subprocess.run([sys.executable, "-c", globals()[name], str(mode)], check=True, timeout=90,
                   cwd=pathlib.Path(__file__).parent.parent, env=os.environ)
