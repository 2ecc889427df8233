"""The solve server's solves on the chip: requests whose shapes they take and
refuse (more than 7 entries a row, more than 256 column patterns, bands too
wide) in one mix, both modes, the same bits alone and in the mix; a cancelled
running solve; more requests than slots and SMs at once."""
from __future__ import annotations

import pathlib
import subprocess
import sys

import numpy as np
import pytest

import gooseberry_b200 as gb
from gooseberry_b200 import workloads as W

pytestmark = pytest.mark.gpu


def shuffled(A, seed):
    """A symmetric renumbering: no patterns repeat, so the batch takes it."""
    p = np.random.default_rng(seed).permutation(A.nrows)
    S = A.to_scipy()[p][:, p].tocsr()
    S.sort_indices()
    return W.Csr(A.nrows, A.ncols, S.indptr.astype(np.uint32), S.indices.astype(np.uint32), S.data)


def nine_point(side):
    """A 9-entry row stencil: longer rows than the on-chip solve takes."""
    import scipy.sparse as sp
    L = W.laplacian_2d(side).to_scipy()
    S = (L @ L + sp.identity(L.shape[0])).tocsr()
    S.sort_indices()
    return W.Csr(S.shape[0], S.shape[0], S.indptr.astype(np.uint32), S.indices.astype(np.uint32),
                 S.data)


def mix():
    mats = [W.diffusion((1,), 1, 1.0, 1.0), W.diffusion((2,), 1, 0.5, 2.0), W.laplacian_2d(45),
            W.diffusion_2d(46, 2), W.diffusion_2d(255, 3), W.diffusion_2d(257, 4),
            W.diffusion((22, 21, 20), 5, 0.1, 10.0), shuffled(W.diffusion_2d(60, 6), 7),
            nine_point(40), W.diffusion((500, 130), 8, 0.1, 10.0), W.diffusion_2d(150, 9)]
    return [(k, A, W.rhs(A.nrows, 60 + k)) for k, A in enumerate(mats)]


@pytest.mark.parametrize("mode", [gb.CG_MIXED, gb.CG_F64])
def test_mix_of_chip_and_batch(mode):
    reqs = mix()
    srv = gb.Server(pool_bytes=1 << 30, max_slots=5, mode=mode, iters_per_step=16)
    for rid, A, b in reqs:
        srv.submit(rid, A, b, tol=1e-10, niter=50_000)
    res = {r.id: r for r in srv.drain()}
    assert sorted(res) == [r[0] for r in reqs]
    for rid, A, b in reqs:
        r = res[rid]
        assert r.status == "converged", (rid, r)
        true = np.linalg.norm(b - A.to_scipy() @ r.x)
        if mode == gb.CG_MIXED:
            assert true <= 1.05e-10 * np.linalg.norm(b), rid
            assert r.refinements >= 1 and r.rnorm == pytest.approx(true, rel=1e-3, abs=1e-300)
        else:
            assert true <= 2e-10 * np.linalg.norm(b), rid
    for rid, A, b in reqs:
        alone = gb.Server(pool_bytes=1 << 29, max_slots=1, mode=mode, iters_per_step=16)
        alone.submit(rid, A, b, tol=1e-10, niter=50_000)
        r1 = alone.drain()[0]
        assert r1.iterations == res[rid].iterations and np.array_equal(r1.x, res[rid].x), rid
        alone.close()
    srv.close()


def test_zero_right_hand_side_and_breakdown():
    srv = gb.Server(pool_bytes=1 << 28, max_slots=2, mode=gb.CG_MIXED)
    A = W.laplacian_2d(70)
    srv.submit(0, A, np.zeros(A.nrows))
    neg = W.Csr(A.nrows, A.ncols, A.rowptr, A.rowind, -A.rowval)
    srv.submit(1, neg, np.ones(A.nrows))
    res = {r.id: r for r in srv.drain()}
    assert res[0].status == "converged" and res[0].iterations == 0 and not res[0].x.any()
    assert res[1].status == "breakdown"
    srv.close()


def test_many_requests_and_a_running_one_cancelled():
    """40 requests through 16 slots; one of them could not converge and is
    cancelled while it runs, its x_out untouched."""
    srv = gb.Server(pool_bytes=1 << 30, max_slots=16, mode=gb.CG_F64)
    A = W.diffusion_2d(300, 11)
    x = np.full(A.nrows, 3.0)
    reqs = [(k, W.diffusion_2d(20 + 7 * k, 20 + k)) for k in range(40)]
    for k, B in reqs[:10]:
        srv.submit(k, B, W.rhs(B.nrows, k), tol=1e-8, niter=20_000)
    srv.step()
    # (r.r underflows to zero, which may end a solve early)
    srv.submit(1000, A, W.rhs(A.nrows, 1), tol=1e-300, niter=10 ** 7, x_out=x)
    srv.step()
    srv.cancel(1000)
    for k, B in reqs[10:]:
        srv.submit(k, B, W.rhs(B.nrows, k), tol=1e-8, niter=20_000)
    res = {r.id: r for r in srv.drain()}
    assert res[1000].status == "cancelled" and np.all(x == 3.0)
    for k, B in reqs:
        assert res[k].status == "converged"
        assert np.linalg.norm(W.rhs(B.nrows, k) - B.to_scipy() @ res[k].x) <= \
            2e-8 * np.linalg.norm(W.rhs(B.nrows, k))
    srv.close()


BEHIND = """
import sys
import gooseberry_b200 as gb
from gooseberry_b200 import workloads as W
mode = int(sys.argv[1])
srv = gb.Server(pool_bytes=1 << 29, max_slots=8, mode=mode)
A = W.diffusion_2d(300, 11)
reqs = [(k, W.diffusion_2d(w, k)) for k, w in enumerate((20, 40, 60, 100, 200))]
srv.submit(1000, A, W.rhs(A.nrows, 1), tol=1e-300, niter=400_000)
srv.step()
for k, B in reqs:
    srv.submit(k, B, W.rhs(B.nrows, k), tol=1e-8, niter=20_000)
order = [r.id for r in srv.drain()]
assert order[-1] == 1000 and sorted(order[:-1]) == [0, 1, 2, 3, 4], order
srv.close()
"""


@pytest.mark.parametrize("mode", [gb.CG_F64, gb.CG_MIXED])
def test_requests_behind_a_long_one(mode):
    """In a new process, where no kernel is loaded yet: small requests (which
    tune their tiles and take other kernels) end before a long one does."""
    subprocess.run([sys.executable, "-c", BEHIND, str(mode)], check=True, timeout=300,
                   cwd=pathlib.Path(__file__).parent.parent)


def test_close_while_solves_run():
    """Destroying a server stops its running solves; the SMs are free again."""
    import torch
    A = W.diffusion_2d(400, 12)
    for _ in range(3):
        srv = gb.Server(pool_bytes=1 << 29, max_slots=2, mode=gb.CG_F64)
        srv.submit(0, A, W.rhs(A.nrows, 1), tol=1e-300, niter=10 ** 7)
        srv.step()
        srv.close()
    M = gb.CsrMatrix.from_host(A)
    b = torch.from_numpy(W.rhs(A.nrows, 1)).cuda()
    _, r = gb.CgSolver(M).solve(b, tol=1e-8)
    assert r.status == "converged"


@pytest.mark.parametrize("mode", [gb.CG_F64, gb.CG_MIXED])
def test_more_solves_at_once_than_hardware_queues(mode):
    """60 requests of one or two CTAs each, all on the chip together: each ends
    with the bits that it has alone, and the statistics count their time."""
    reqs = [(k, W.diffusion_2d(24 + k, k)) for k in range(60)]
    many = gb.Server(pool_bytes=1 << 29, max_slots=64, mode=mode)
    for k, B in reqs:
        many.submit(k, B, W.rhs(B.nrows, k), tol=1e-9, niter=20_000)
    got = {r.id: r for r in many.drain()}
    assert 0.0 < many.stats()["gpu_ms"] < 1e4
    many.close()
    one = gb.Server(pool_bytes=1 << 29, max_slots=1, mode=mode)
    for k, B in reqs[::7]:
        one.submit(k, B, W.rhs(B.nrows, k), tol=1e-9, niter=20_000)
        r = one.drain()[0]
        assert got[k].status == r.status == "converged" and got[k].iterations == r.iterations
        assert np.array_equal(got[k].x, r.x)
    one.close()
