"""Edge lists and transposes through the radix sort: sizes at the edges of its
tiles (4,096 keys), digits of every width, duplicates whose
earliest edge gives the value, and every flag, against numpy.
"""
import numpy as np
import pytest

import graphalgo_gb300 as ga

pytestmark = pytest.mark.gpu

LINE = 1 << 16  # sixteen tiles


def _expected(m, n, src, dst, val, flags):
    """Entries in the reference's order, then one per (row, column): the earliest edge's value."""
    s, d, v = src.astype(np.int64), dst.astype(np.int64), val
    e = np.arange(len(s))
    if flags & ga.EDGES_MIRROR:
        s, d, e = np.stack([s, d], 1).reshape(-1), np.stack([d, s], 1).reshape(-1), np.repeat(e, 2)
    if flags & (ga.EDGES_DROP_LOOPS | ga.EDGES_LOWER_SYMM):
        k = s != d
        s, d, e = s[k], d[k], e[k]
    if flags & ga.EDGES_LOWER_SYMM:
        k = s > d
        s, d, e = s[k], d[k], e[k]
        s, d, e = np.concatenate([s, d]), np.concatenate([d, s]), np.concatenate([e, e])
    order = np.lexsort((e, d, s))
    s, d, e = s[order], d[order], e[order]
    first = np.ones(len(s), bool)
    first[1:] = (s[1:] != s[:-1]) | (d[1:] != d[:-1])
    s, d, e = s[first], d[first], e[first]
    rst = np.concatenate([[0], np.cumsum(np.bincount(s, minlength=m))]).astype(np.int32)
    return rst, d.astype(np.int32), v[e]


@pytest.mark.parametrize("ne", [0, 1, 2, 33, 4095, 4096, 4097, LINE, LINE + 1, 4096 * 17 - 1, 200003])
@pytest.mark.parametrize("shape", [(1, 1), (3, 100000), (1000, 1000), (1025, 1 << 20), (70001, 70001)])
@pytest.mark.parametrize("flags", [0, ga.EDGES_DROP_LOOPS])
def test_edges(ctx, ne, shape, flags):
    m, n = shape
    rng = np.random.default_rng(ne + m)
    src, dst = rng.integers(0, m, ne).astype(np.int32), rng.integers(0, n, ne).astype(np.int32)
    val = rng.standard_normal(ne)
    r, c, v = _expected(m, n, src, dst, val, flags)
    R, C, V = ga.csr_from_edges(ctx, m, n, src, dst, val, flags=flags).download()
    assert np.array_equal(R, r) and np.array_equal(C, c) and np.array_equal(V, v)


@pytest.mark.parametrize("flags", [ga.EDGES_MIRROR, ga.EDGES_MIRROR | ga.EDGES_DROP_LOOPS, ga.EDGES_LOWER_SYMM,
                                   ga.EDGES_MIRROR | ga.EDGES_LOWER_SYMM])
@pytest.mark.parametrize("dtype", [np.int32, np.uint8, np.float64])
def test_edge_flags(ctx, flags, dtype):
    n, ne = 5000, 90001
    rng = np.random.default_rng(flags)
    # hubs, loops and many repeats
    src = (n * rng.random(ne) ** 3).astype(np.int32)
    dst = np.where(rng.random(ne) < 0.05, src, (n * rng.random(ne) ** 3).astype(np.int32)).astype(np.int32)
    val = rng.integers(0, 200, ne).astype(dtype)
    r, c, v = _expected(n, n, src, dst, val, flags)
    A = ga.csr_from_edges(ctx, n, n, src, dst, val, flags=flags)
    R, C, V = A.download()
    assert np.array_equal(R, r) and np.array_equal(C, c) and np.array_equal(V, v)
    U = ga.csr_from_edges(ctx, n, n, src, dst, val, flags=flags | ga.EDGES_UNIT).download()
    assert np.array_equal(U[1], c) and U[2].dtype == np.int32 and np.all(U[2] == 1)


def test_edges_refused(ctx):
    src = np.zeros(LINE, np.int32)
    for bad in (-1, 10):
        dst = np.zeros(LINE, np.int32)
        dst[777] = bad
        with pytest.raises(ga.GaError):
            ga.csr_from_edges(ctx, 10, 10, src, dst)
    loops = ga.csr_from_edges(ctx, 10, 10, src, src, flags=ga.EDGES_DROP_LOOPS)
    assert loops.nnz == 0 and not loops.download()[0].any()


@pytest.mark.parametrize("shape", [(1, 70000), (70000, 1), (300, 300), (40000, 1025), (999, 200001)])
@pytest.mark.parametrize("dtype", [np.int32, np.int64, np.float32, np.float64, np.uint8])
def test_transpose(ctx, shape, dtype):
    m, n = shape
    rng = np.random.default_rng(m)
    key = np.sort(rng.permutation(m * n)[:66000]) if m * n < 10 ** 6 else np.unique(rng.integers(0, m * n, 120000))
    _check_transpose(ctx, m, n, key, dtype, rng)


@pytest.mark.parametrize("count", [0, 1, 2, 31, 4096, 4097])
def test_transpose_small(ctx, count):
    rng = np.random.default_rng(count)
    _check_transpose(ctx, 90, 70, np.sort(rng.permutation(90 * 70)[:count]), np.float64, rng)


def _check_transpose(ctx, m, n, key, dtype, rng):
    row, col = key // n, key % n
    val = rng.integers(0, 100, len(key)).astype(dtype)
    rst = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=m))]).astype(np.int32)
    T = ga.transpose(ga.Csr.upload(ctx, m, n, rst, col.astype(np.int32), val))
    order = np.lexsort((row, col))
    r, c, v = T.download()
    assert T.shape == (n, m)
    assert np.array_equal(r, np.concatenate([[0], np.cumsum(np.bincount(col, minlength=n))]))
    assert np.array_equal(c, row[order]) and np.array_equal(v, val[order])
