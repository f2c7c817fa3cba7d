"""Complemented products with few columns: memory that fails inside the narrow
path, and what it holds. Against the oracle; the values are small integers, so
the results must be equal.
"""
import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import to_device

pytestmark = pytest.mark.gpu


def _csr(m, n, key, dtype, rng):
    key = np.unique(key)
    rst = np.concatenate([[0], np.cumsum(np.bincount(key // n, minlength=m))]).astype(np.int32)
    return oracle.Csr(m, n, rst, (key % n).astype(np.int32), rng.integers(-3, 4, len(key)).astype(dtype))


def _operands(m, k, n, dtype, long_rows):
    """A (m x k, 8 entries per row, rows of the given lengths first), B (k x n), M (m x n, a row full, one empty)."""
    rng = np.random.default_rng(m + n)
    rows = [rng.integers(0, m, 8 * m) * k + rng.integers(0, k, 8 * m)]
    rows[0] = rows[0][rows[0] // k >= len(long_rows)]
    rows += [i * k + np.arange(length) for i, length in enumerate(long_rows)]
    A = _csr(m, k, np.concatenate(rows), dtype, rng)
    B = _csr(k, n, rng.integers(0, k, 3 * k) * n + rng.integers(0, n, 3 * k), dtype, rng)
    key = rng.integers(0, m, 2 * m) * n + rng.integers(0, n, 2 * m)
    M = _csr(m, n, np.concatenate([key[key // n != 9], 8 * n + np.arange(n)]), dtype, rng)
    return A, B, M


def test_memory_fails_inside(ctx):
    """Whichever allocation of the narrow path fails, the product is made without it."""
    A, B, M = _operands(3000, 4200, 200, np.int32, [4200, 257])
    R = oracle.mxm_cmask(A, B, M)
    dA, dB, dM = to_device(ctx, A), to_device(ctx, B), to_device(ctx, M)
    for n in range(12):
        ctx.set_option(ga.OPT_FAIL_ALLOC_AFTER, n)
        try:
            C = ga.mxm_cmask(dA, dB, dM)
        finally:
            ctx.set_option(ga.OPT_FAIL_ALLOC_AFTER, -1)
        rst, col, val = C.download()
        assert np.array_equal(rst, R.rst) and np.array_equal(col, R.col) and np.array_equal(val, R.val), n


def test_partial_sums_only_for_pieces(ctx):
    """A without a row in pieces takes no memory for partial sums, however many entries it has."""
    m, n = 1 << 15, 1024
    rng = np.random.default_rng(5)
    A = _csr(m, m, rng.integers(0, m, 64 * m) * m + rng.integers(0, m, 64 * m), np.float64, rng)
    B = _csr(m, n, rng.integers(0, m, m) * n + rng.integers(0, n, m), np.float64, rng)
    M = _csr(m, n, rng.integers(0, m, m) * n + rng.integers(0, n, m), np.float64, rng)
    dA, dB, dM = to_device(ctx, A), to_device(ctx, B), to_device(ctx, M)
    ctx.sync()
    base, _ = ctx.mem_stats(reset_peak=True)
    C = ga.mxm_cmask(dA, dB, dM)
    held = 4 * (m + 1) + 12 * C.nnz
    # words of A and B, counts and starts, 20 bytes per 170 entries for the pieces' list
    assert ctx.mem_stats()[1] - base <= held + 16 * 20 * m + 8 * (m + 1) + 20 * (3 * A.nnz // 512 + 2) + 65536
