"""Complemented products with few columns: the narrow path over its tile edges
(operands of enough rows that it is chosen), the general path where A has few
rows, memory that fails inside the narrow path, and what it holds. Against the
oracle; the values are small integers, so the results must be equal.
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


def _check(ctx, A, B, M, dtype):
    od = np.int32 if np.dtype(dtype).kind == "i" else np.float64
    R = oracle.mxm_cmask(*(oracle.Csr(X.m, X.n, X.rst, X.col, X.val.astype(od)) for X in (A, B, M)))
    C = ga.mxm_cmask(to_device(ctx, A), to_device(ctx, B), to_device(ctx, M))
    rst, col, val = C.download()
    assert np.array_equal(rst, R.rst) and np.array_equal(col, R.col)
    assert val.dtype == dtype and np.array_equal(val, R.val.astype(dtype))


@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 64, 65, 129, 256, 1023, 1024, 1025])
@pytest.mark.parametrize("dtype", [np.int32, np.int64, np.float32, np.float64])
def test_narrow(ctx, n, dtype):
    _check(ctx, *_operands(3000, 4200, n, dtype, [4200, 255, 256, 257, 511, 512, 513, 1025, 1, 300]), dtype)


@pytest.mark.parametrize("m", [1, 2, 40, 500, 2048])
@pytest.mark.parametrize("k", [70, 60000])
@pytest.mark.parametrize("n", [64, 1000])
def test_few_rows(ctx, m, k, n):
    _check(ctx, *_operands(max(m, 10), k, n, np.float64, [min(k, 600), 1][:m]), np.float64)


def test_few_rows_make_no_words(ctx):
    """Few rows of A against a tall B: no words of B's rows (12 bytes each per 64 columns)."""
    m, k, n = 16, 1 << 20, 1024
    rng = np.random.default_rng(6)
    A, B, M = (_csr(r, c, rng.integers(0, r, z) * c + rng.integers(0, c, z), np.float64, rng)
               for r, c, z in ((m, k, 1000), (k, n, k), (m, n, 100)))
    dA, dB, dM = to_device(ctx, A), to_device(ctx, B), to_device(ctx, M)
    ctx.sync()
    base, _ = ctx.mem_stats(reset_peak=True)
    ga.mxm_cmask(dA, dB, dM)
    assert ctx.mem_stats()[1] - base <= 1 << 20


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
