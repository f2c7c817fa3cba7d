"""Heavy rows of a masked product, split into windows: rows above and below the
split, masks of few and of many entries, and more windows asked for than the
queue holds. Whole numbers: equal to the oracle's.
"""
import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import to_device

pytestmark = pytest.mark.gpu


def _rows(lengths, n, rng, dtype):
    rst = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    col = np.concatenate([np.sort(rng.choice(n, d, replace=False)) for d in lengths]).astype(np.int32)
    return oracle.Csr(len(lengths), n, rst, col, rng.integers(-3, 4, len(col)).astype(dtype))


@pytest.mark.parametrize("dtype", [np.int32, np.float64])
@pytest.mark.parametrize("algo", ["msa", "mca", "heap", "hybrid"])
def test_split(ctx, algo, dtype):
    rng = np.random.default_rng(8)
    k, n = 1200, 200000
    hubs = [1, 31, 32, 33, 64, 300, 2048, 4097, 9000]   # mask entries of the heavy rows
    A = _rows([1100] * len(hubs) + [70] * len(hubs) + [3] * 400, k, rng, dtype)
    B = _rows(rng.integers(300, 900, k).tolist(), n, rng, dtype)
    M = _rows(hubs * 2 + [5] * 400, n, rng, dtype)
    C = ga.mxm_masked(algo, to_device(ctx, A), to_device(ctx, B), to_device(ctx, M))
    rst, col, val = C.download()
    assert np.array_equal(rst, M.rst) and np.array_equal(col, M.col)
    assert np.array_equal(val, oracle.mxm_masked(A, B, M))


def test_more_windows_than_the_queue_holds(ctx):
    """A's sampled entries (every 8,000th) meet empty rows of B, so every row
    asks for windows. All rows of A are alike: C's columns are B's sums."""
    rng = np.random.default_rng(9)
    m, k, n = 2000, 1024, 6000
    A = oracle.Csr(m, k, (np.arange(m + 1) * k).astype(np.int32), np.tile(np.arange(k), m).astype(np.int32),
                   np.ones(m * k, np.int32))
    B = _rows(np.where(np.arange(k) % 64 == 0, 0, 300).tolist(), n, rng, np.int32)
    M = _rows([200] * m, n, rng, np.int32)
    C = ga.mxm_masked("msa", to_device(ctx, A), to_device(ctx, B), to_device(ctx, M))
    sums = np.zeros(n, np.int64)
    np.add.at(sums, B.col, B.val)
    assert np.array_equal(C.download()[2], sums[M.col])
