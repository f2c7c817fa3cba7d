"""Masked products whose rows a warp's hash table serves, the table half full:
many rows of up to 256 random mask entries, so that lookups probe for long.
Small integers: equal to the oracle's.
"""
import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import to_device

pytestmark = pytest.mark.gpu


def _random(m, n, least, most, rng):
    length = rng.integers(least, most + 1, m)
    order = np.argsort(rng.random((m, n), dtype=np.float32), axis=1)
    order[np.arange(n)[None, :] >= length[:, None]] = n  # the first `length` columns of each order
    order.sort(axis=1)
    rst = np.concatenate([[0], np.cumsum(length)]).astype(np.int32)
    return oracle.Csr(m, n, rst, order[order < n].astype(np.int32), rng.integers(1, 4, rst[-1]).astype(np.int32))


@pytest.mark.parametrize("seed", [100, 102, 104])
@pytest.mark.parametrize("least,most", [(200, 256), (100, 128)])
def test_long_probes(ctx, seed, least, most):
    rng = np.random.default_rng(seed)
    M, A, B = _random(9000, 1500, least, most, rng), _random(9000, 400, 1, 45, rng), _random(400, 1500, 0, 60, rng)
    ref = oracle.mxm_masked(A, B, M)
    dM = to_device(ctx, M)
    for dtype in (np.float32, np.int32, np.uint8, np.int64, np.float64):
        dA, dB = (to_device(ctx, oracle.Csr(X.m, X.n, X.rst, X.col, X.val.astype(dtype))) for X in (A, B))
        for algo in ("msa", "mca", "hybrid"):
            v = ga.mxm_masked(algo, dA, dB, dM).download()[2]
            bad = np.flatnonzero(v != ref.astype(dtype))
            assert len(bad) == 0, (np.dtype(dtype).name, algo, np.searchsorted(M.rst, bad, side="right") - 1)


def test_long_probes_of_ones(ctx):
    rng = np.random.default_rng(100)
    M, A, B = _random(12000, 1500, 200, 256, rng), _random(12000, 400, 1, 45, rng), _random(400, 1500, 0, 60, rng)
    A, B = (oracle.Csr(X.m, X.n, X.rst, X.col, np.ones(X.nnz, np.int32)) for X in (A, B))
    v = ga.mxm_masked("msa", to_device(ctx, A), to_device(ctx, B), to_device(ctx, M)).download()[2]
    assert np.array_equal(v, oracle.mxm_masked(A, B, M))
