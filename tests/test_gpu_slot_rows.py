"""Masked products with accumulators of 8 bytes under mask rows around 128 and
256 entries (tables of columns, of slots, CTA items): against the oracle, small
integers, so equal; and rows just above 128 entries take about the time of rows
just below.
"""
import ctypes

import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import to_device

pytestmark = pytest.mark.gpu

LENGTHS = [256, 255, 257, 254, 128, 129, 127, 130, 1, 0, 200, 64, 512]


def _rows(lengths, n, values, rng):
    """A CSR of rows of the given lengths, columns drawn over [0, n); some rows a run from 0 or up to n."""
    rst = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    col = []
    for i, k in enumerate(lengths):
        c = np.arange(k) if i % 7 == 1 else np.arange(n - k, n) if i % 7 == 2 else np.sort(rng.permutation(n)[:k])
        col.append(c)
    col = np.concatenate(col).astype(np.int32)
    return oracle.Csr(len(lengths), n, rst, col, values(len(col)))


@pytest.mark.parametrize("algo", ["msa", "mca", "heap", "hybrid"])
@pytest.mark.parametrize("dtype", [np.float64, np.int64, np.float32])
@pytest.mark.parametrize("values", ["any", "unit B", "ones"])
@pytest.mark.parametrize("rows,inner", [(39, 700), (2500, 300)])
def test_lengths(ctx, algo, dtype, values, rows, inner):
    rng = np.random.default_rng(rows)
    n = 1500
    any_ = lambda k: rng.integers(-3, 4, k).astype(dtype)
    ones = lambda k: np.ones(k, dtype)
    M = _rows([LENGTHS[i % len(LENGTHS)] for i in range(rows)], n, ones, rng)
    A = _rows(rng.integers(0, 40, rows), inner, ones if values == "ones" else any_, rng)
    B = _rows(rng.integers(0, 60, inner), n, any_ if values == "any" else ones, rng)
    assert M.nnz > 64 * rows  # the mean from which rows above 128 entries are by slots
    wide = np.int32 if np.dtype(dtype).kind == "i" else np.float64
    ref = oracle.mxm_masked(*(oracle.Csr(X.m, X.n, X.rst, X.col, X.val.astype(wide)) for X in (A, B, M)))
    v = ga.mxm_masked(algo, to_device(ctx, A), to_device(ctx, B), to_device(ctx, M)).download()[2]
    assert np.array_equal(v, ref.astype(dtype))


@pytest.mark.parametrize("algo", ["msa", "heap"])
def test_no_cliff_at_128(ctx, algo):
    """100,000 rows of 100 products: with 140 mask entries each at most five times as long as with 120."""
    m, n, k = 100000, 100000, 20000
    rng = np.random.default_rng(1)

    def even(rows, cols, per, dtype):
        col = (np.arange(per) * (cols // per))[None, :] + rng.integers(0, cols // per, (rows, per))
        return ga.Csr.upload(ctx, rows, cols, (np.arange(rows + 1) * per).astype(np.int32),
                             col.ravel().astype(np.int32), np.full(rows * per, 3, dtype))

    A, B = even(m, k, 10, np.float64), even(k, n, 10, np.float64)
    best = []
    for per in (120, 140):
        M, ms = even(m, n, per, np.int32), ctypes.c_double()
        took = []
        for _ in range(6):
            ctx.sync()
            ga.lib().ga_timer_start(ctx.handle)
            C = ga.mxm_masked(algo, A, B, M)
            ga.lib().ga_timer_stop(ctx.handle, ctypes.byref(ms))
            took.append(ms.value)
            C.free()
        best.append(min(took))
    assert best[1] < 5 * best[0]
