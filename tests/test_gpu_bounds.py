"""The byte bound of a request covers what the call allocates, for the graphs
that need most beside their size: with values and directed (a copy and a
transpose), nearly dense with many sources (long neighbour lists in pieces).
And the transpose itself: what it holds beside its result.
"""
import numpy as np
import pytest

import graphalgo_gb300 as ga

pytestmark = pytest.mark.gpu


def _random(m, degree, directed, hub=0):
    """m vertices of `degree` neighbours on average, the last `hub` of them next to all; values 1 to 3."""
    rng = np.random.default_rng(m + degree)
    if directed:
        row = np.repeat(np.arange(m), degree)
        key = row * m + rng.integers(0, m, m * degree)
    else:
        a, b = rng.integers(0, m, (2, m * degree // 2))
        key = np.concatenate([a * m + b, b * m + a])
    ends = np.arange(m - hub, m)
    key = np.concatenate([key] + [np.concatenate([h * m + np.arange(m), np.arange(m) * m + h]) for h in ends])
    key = np.unique(key[key // m != key % m])
    row, col = key // m, key % m
    rst = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=m))]).astype(np.int32)
    return m, rst, col.astype(np.int32), ((row + col) % 3 + 1).astype(np.int32)


def _peak(ctx, run):
    ctx.sync()
    base, _ = ctx.mem_stats(reset_peak=True)
    run()
    ctx.sync()
    return ctx.mem_stats()[1] - base


@pytest.mark.parametrize("graph,ns", [
    ((30000, 48, True), 1),            # directed, many entries per vertex, one source
    ((30000, 48, True), 40),
    ((2500, 254, False), 1024),        # pieces of the shorter kind, as many sources as there can be
    ((2500, 254, False, 3), 1000),
    ((2600, 280, False, 4), 1024),     # the longer kind
    ((2600, 280, True, 4), 65),
], ids=str)
def test_bc(ctx, graph, ns):
    m, rst, col, val = _random(*graph)
    A = ga.Csr.upload(ctx, m, m, rst, col, val)
    src = np.arange(ns, dtype=np.int32)
    bound = ga.request_bytes_bound(ga.REQ_BC, m, len(col), ns)
    assert _peak(ctx, lambda: ga.bc(A, src)) <= bound


@pytest.mark.parametrize("dtype", [np.uint8, np.int32, np.int64, np.float32, np.float64])
@pytest.mark.parametrize("n", [1, 700, 5000, 1 << 20, 1 << 21])  # none to three passes of the sort
def test_transpose(ctx, n, dtype):
    """Equal to the transpose by numpy, in at most 10 bytes per entry beside the result (uint8: 14)."""
    m = 3001
    rng = np.random.default_rng(n)
    key = np.unique(rng.integers(0, m, 200000) * n + rng.integers(0, n, 200000))
    row, col = key // n, key % n
    rst = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=m))]).astype(np.int32)
    val = (np.arange(len(key)) % 251).astype(dtype)
    A = ga.Csr.upload(ctx, m, n, rst, col.astype(np.int32), val)
    kept = []
    peak = _peak(ctx, lambda: kept.append(ga.transpose(A)))
    r, c, v = kept[0].download()
    order = np.argsort(col, kind="stable")
    assert np.array_equal(r, np.concatenate([[0], np.cumsum(np.bincount(col, minlength=n))]))
    assert np.array_equal(c, row[order]) and np.array_equal(v, val[order])
    size = np.dtype(dtype).itemsize
    assert peak <= 4 * (n + 1) + len(key) * (4 + size + (10 if size >= 4 else 14)) + 65536
