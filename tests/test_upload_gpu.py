"""Uploads of pageable host arrays: those large enough for the threaded path,
at its piece edges, alone and from several threads at once."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import gooseberry_b200 as gb

pytestmark = pytest.mark.gpu

MB = 1 << 20


def scaled(n, seed):
    v = np.random.default_rng(seed).uniform(-1, 1, n)
    return v, v * 2.0


@pytest.mark.parametrize("nbytes", [8, 24 * MB - 8, 24 * MB, 24 * MB + 8, 31 * MB + 4096, 67 * MB - 8])
def test_round_trip(nbytes):
    v, want = scaled(nbytes // 8, 1)
    assert np.array_equal(gb.scale(v, 2.0), want)


def test_several_threads():
    jobs = [scaled((24 + k) * MB // 8 + k, 10 + k) for k in range(5)]

    def work(v):
        gb.scale(v, 2.0)

    ts = [threading.Thread(target=work, args=(v,)) for v, _ in jobs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for v, want in jobs:
        assert np.array_equal(v, want)
