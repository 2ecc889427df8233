"""Large uploads of pageable host arrays on cudaStreamPerThread."""
from __future__ import annotations

import numpy as np
import pytest

import gooseberry_b200 as gb
from gooseberry_b200 import workloads as W

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_callers_per_thread_stream():
    """cudaStreamPerThread (handle 2) is another stream in every thread: the
    matrix's pieces are all there before the caller's own stream reads them."""
    import torch
    n = 3 << 20
    A = W.Csr(n, n, np.arange(n + 1, dtype=np.uint32),
              np.random.default_rng(5).permutation(n).astype(np.uint32),
              np.random.default_rng(6).uniform(1, 2, n))
    assert A.rowval.nbytes >= 24 * MB
    x = torch.arange(n, dtype=torch.float64, device="cuda")
    want = A.rowval * A.rowind
    torch.cuda.synchronize()
    for _ in range(5):
        M = gb.CsrMatrix.from_host(A, stream=2)
        y = M.spmv(x, stream=2)
        torch.cuda.synchronize()
        assert np.array_equal(y.cpu().numpy(), want)
        M.close()
