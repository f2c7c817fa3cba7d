"""Row binning of the masked product with several rows per warp: empty masks,
rows without products, rows summed by the whole CTA, rows of several windows.
Whole numbers: equal to the oracle's.
"""
import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import to_device

pytestmark = pytest.mark.gpu


def _csr(m, n, row, col, rng, dtype):
    key = np.unique(row.astype(np.int64) * n + col)
    rst = np.concatenate([[0], np.cumsum(np.bincount(key // n, minlength=m))]).astype(np.int32)
    return oracle.Csr(m, n, rst, (key % n).astype(np.int32), rng.integers(-3, 4, len(key)).astype(dtype))


def _sparse(m, n, count, hubs, rng, dtype, empty=()):
    row, col = rng.integers(0, m, count), rng.integers(0, n, count)
    for r, d in hubs:
        row = np.concatenate([row, np.full(d, r)])
        col = np.concatenate([col, rng.integers(0, n, d)])
    keep = ~np.isin(row, np.asarray(empty))
    return _csr(m, n, row[keep], col[keep], rng, dtype)


@pytest.mark.parametrize("m", [9727, 9728 * 2, 45001, 9728 * 33])
@pytest.mark.parametrize("algo", ["msa", "mca", "heap", "hybrid"])
def test_bins(ctx, m, algo):
    rng = np.random.default_rng(m)
    k, n = 3000, 300000
    empty = rng.integers(0, m, m // 5)
    A = _sparse(m, k, 2 * m, [(0, 1023), (1, 1500), (m // 2, 2900), (m - 1, 2900)], rng, np.int32, empty)
    B = _sparse(k, n, 4 * k, [(5, 20000), (7, 300)], rng, np.int32, np.arange(0, k, 3))
    M = _sparse(m, n, 2 * m, [(0, 9000), (1, 300), (m // 2, 200), (m - 1, 5000)], rng, np.int32,
                rng.integers(0, m, m // 5))
    C = ga.mxm_masked(algo, to_device(ctx, A), to_device(ctx, B), to_device(ctx, M))
    rst, col, val = C.download()
    assert np.array_equal(rst, M.rst) and np.array_equal(col, M.col)
    assert np.array_equal(val, oracle.mxm_masked(A, B, M))
