"""C<A> = A·A of a symmetric A by halves (from 2^18 entries on): every variant
and value type against the oracle, the work counters against an asymmetric
twin's rules, and operands that must not take the path.
"""
import numpy as np
import pytest

import graphalgo_gb300 as ga
import oracle
from graphs import to_device

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph():
    m, rst, col = ga.gen_rmat(14, 20, seed=8)
    # some diagonal entries and an empty stretch of rows
    row = np.repeat(np.arange(m), np.diff(rst))
    keep = ~(((row >= 300) & (row < 340)) | ((col >= 300) & (col < 340)))
    row, col = np.concatenate([row[keep], np.arange(0, 200)]), np.concatenate([col[keep], np.arange(0, 200)])
    key = np.unique(row.astype(np.int64) * m + col)
    rst = np.concatenate([[0], np.cumsum(np.bincount(key // m, minlength=m))]).astype(np.int32)
    assert len(key) >= 1 << 18
    return m, rst, (key % m).astype(np.int32), key


def _symmetric_values(graph, dtype):
    m, _, col, key = graph
    row = key // m
    v = (np.minimum(row, col) * 7 + np.maximum(row, col) * 3) % 5 - 2
    return (v if np.dtype(dtype) != np.uint8 else v + 2).astype(dtype)


@pytest.mark.parametrize("algo", ["msa", "mca", "heap", "dot", "hybrid"])
@pytest.mark.parametrize("dtype", ["ones", np.int32, np.int64, np.float32, np.float64, np.uint8])
def test_half(ctx, graph, algo, dtype):
    m, rst, col, _ = graph
    val = np.ones(len(col), np.int32) if dtype == "ones" else _symmetric_values(graph, dtype)
    wide = np.int32 if val.dtype.kind in "iu" else np.float64  # small integers: exact in every type
    W = oracle.Csr(m, m, rst, col, val.astype(wide))
    ref = oracle.mxm_masked(W, W, W)
    A = ga.Csr.upload(ctx, m, m, rst, col, val)
    ctx.work_counters(reset=True)
    C = ga.mxm_masked(algo, A, A, A)
    w = ctx.work_counters(reset=True)
    r, c, v = C.download()
    assert np.array_equal(r, rst) and np.array_equal(c, col)
    want = (ref & 0xFF).astype(np.uint8) if val.dtype == np.uint8 else ref.astype(val.dtype)
    assert np.array_equal(v, want)
    # the counters report the whole product
    deg = np.diff(rst).astype(np.int64)
    assert w["mask_entries"] == len(col) and w["a_entries"] == len(col) and w["products"] == int(deg[col].sum())


@pytest.mark.parametrize("algo", ["msa", "mca", "heap"])
def test_not_symmetric(ctx, graph, algo):
    """A value that differs from its mirror's: the product in full."""
    m, rst, col, key = graph
    val = np.ones(len(col), np.int32)
    q = int(np.flatnonzero(key // m != col)[1000])
    val[q] = 5
    G = oracle.Csr(m, m, rst, col, val)
    A = to_device(ctx, G)
    v = ga.mxm_masked(algo, A, A, A).download()[2]
    assert np.array_equal(v, oracle.mxm_masked(G, G, G))
    # a symmetric A with another mask
    ones = oracle.Csr(m, m, rst, col, np.ones(len(col), np.int32))
    S, M = to_device(ctx, ones), ga.extract_lower(to_device(ctx, ones))
    mr, mc, _ = M.download()
    v = ga.mxm_masked(algo, S, S, M).download()[2]
    assert np.array_equal(v, oracle.mxm_masked(ones, ones, oracle.Csr(m, m, mr, mc, np.ones(len(mc), np.int32))))
