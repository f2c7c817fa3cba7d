"""Complemented product with few columns (the narrow path) against the oracle.

The values are small integers, so every dtype's sums are exact whatever the
order and the results must be equal.
"""
import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import random_csr, to_device

pytestmark = pytest.mark.gpu


def _operands(n, dtype, seed):
    rng = np.random.default_rng(seed)
    m, k = 37, 4200
    D = rng.random((m, k)) < 0.01
    D[0] = True                    # nine pieces
    D[1] = np.arange(k) < 512      # one piece, full
    D[2] = np.arange(k) < 513      # one piece and one entry
    D[17] = np.arange(k) < 257     # the shortest row in pieces
    D[20] = np.arange(k) < 256     # the longest row of one warp
    D[5] = False
    from graphs import dense_to_csr
    A = dense_to_csr(D, rng.integers(-3, 4, (m, k)), dtype)
    B = random_csr(k, n, 0.03, rng, np.int32)
    B = oracle.Csr(B.m, B.n, B.rst, B.col, B.val.astype(dtype))
    K = rng.random((m, n)) < 0.3
    K[3] = True                    # nothing left
    K[4] = False
    return A, B, dense_to_csr(K, np.ones((m, n)), dtype)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 64, 65, 129, 256, 1023, 1024, 1025])
@pytest.mark.parametrize("dtype", [np.int32, np.int64, np.float32, np.float64])
def test_narrow_cmask(ctx, n, dtype):
    A, B, M = _operands(n, dtype, n)
    # the oracle has int32 and fp64; the values are small integers in every dtype
    od = np.int32 if np.dtype(dtype).kind == "i" else np.float64
    R = oracle.mxm_cmask(*(oracle.Csr(X.m, X.n, X.rst, X.col, X.val.astype(od)) for X in (A, B, M)))
    C = ga.mxm_cmask(to_device(ctx, A), to_device(ctx, B), to_device(ctx, M))
    rst, col, val = C.download()
    assert np.array_equal(rst, R.rst) and np.array_equal(col, R.col)
    assert val.dtype == dtype and np.array_equal(val, R.val.astype(dtype))
